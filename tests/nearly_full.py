"""A device with little memory left."""
import contextlib


@contextlib.contextmanager
def nearly_full(free_bytes):
    """Holds all but about `free_bytes` of the device's memory (in pieces of
    2 MB, the unit in which the device hands it out)."""
    import torch
    hog, unit = [], 2 << 20
    torch.cuda.synchronize()
    try:
        while True:
            n = (torch.cuda.mem_get_info()[0] - free_bytes) // unit
            if n < 2:
                break
            hog.append(torch.cuda.caching_allocator_alloc(n * unit))
        yield
    finally:
        torch.cuda.synchronize()
        for p in hog:
            torch.cuda.caching_allocator_delete(p)
        torch.cuda.empty_cache()
