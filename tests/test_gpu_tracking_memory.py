"""Offline delta tracking's FP64 sums: what the library keeps of them goes back
with the volume, and a device that is nearly full renders in parts."""
import ctypes as C

import pytest

from tests.nearly_full import nearly_full

pytestmark = pytest.mark.gpu


def _offline_render(side, out):
    """A volume, one delta-tracking render into `out`, and the volume's end."""
    import torch
    import internship_b200 as mr
    from internship_b200 import _lib, scenes
    v = mr.VolumeRender(16)
    v.SetDatas(scenes.sphere_density(16))
    v.Update()
    p = scenes.make_params(side, side, 1, bounces=4)
    _lib.check(_lib.load().mr_render(v.handle, None, C.byref(p), C.c_void_p(out.data_ptr()), None))
    torch.cuda.synchronize()
    v.close()


def test_offline_tracking_gives_its_memory_back():
    """A 2048 x 2048 render sums its samples in 96 MiB of FP64; the library keeps
    at most 32 MiB of that after the volume."""
    import torch
    import internship_b200 as mr
    out = torch.zeros(2048 * 2048 * 3, device="cuda")
    _offline_render(64, out)  # kernels loaded
    mr.Network(mr.xavier_weights(1)).close()  # nothing kept from earlier calls
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    _offline_render(2048, out)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] >= free - (32 << 20)
    mr.Network(mr.xavier_weights(1)).close()
    assert torch.cuda.mem_get_info()[0] >= free


def test_offline_tracking_on_a_nearly_full_device():
    """With some 32 MB free the 72 MB of FP64 sums of a 2000 x 1501 render are
    had for a part of the rows at a time. A pixel's few samples sum exactly in
    FP64, so the image is the same, and the counters cover all rows."""
    import torch
    import internship_b200 as mr
    from internship_b200 import _lib, scenes
    v = mr.VolumeRender(16)
    v.SetDatas(scenes.sphere_density(16))
    v.Update()
    p = scenes.make_params(2000, 1501, 2, bounces=8)
    ref, out = torch.zeros(2000 * 1501 * 3, device="cuda"), torch.zeros(2000 * 1501 * 3, device="cuda")

    def render(x):
        _lib.check(_lib.load().mr_render(v.handle, None, C.byref(p), C.c_void_p(x.data_ptr()), None))
        torch.cuda.synchronize()
        n = (C.c_uint64 * 4)()
        _lib.check(_lib.load().mr_volume_counters(v.handle, n))
        return list(n)

    whole = render(ref)
    mr.Network(mr.xavier_weights(1)).close()  # gives the library's unused memory back
    with nearly_full(32 << 20):
        parts = render(out)
    v.close()
    assert (ref > 0).any()
    assert torch.equal(out, ref)
    assert parts == whole and whole[1] == 2 * 2000 * 1501
