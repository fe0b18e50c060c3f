"""What the library keeps between calls goes back with the objects whose calls
used it."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _offline_render(side, out):
    """A volume, one delta-tracking render into `out`, and the volume's end."""
    import internship_b200 as mr
    from internship_b200 import _lib, scenes
    v = mr.VolumeRender(16)
    v.SetDatas(scenes.sphere_density(16))
    v.Update()
    p = scenes.make_params(side, side, 1, bounces=4)
    _lib.check(_lib.load().mr_render(v.handle, None, C.byref(p), C.c_void_p(out.data_ptr()), None))
    v.close()


def test_offline_tracking_leaves_no_memory_behind():
    """A 2048 x 2048 render sums its samples in 96 MiB of FP64."""
    import torch
    import internship_b200 as mr
    out = torch.zeros(2048 * 2048 * 3, device="cuda")
    _offline_render(64, out)  # kernels loaded
    mr.Network(mr.xavier_weights(1)).close()  # nothing kept from earlier calls
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    _offline_render(2048, out)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] >= free
