"""Offline delta tracking captured into a CUDA graph."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def test_offline_tracking_replays_from_a_graph():
    """The samples' FP64 sums are nodes of the graph. The sum of a pixel's 9
    samples is exact in FP64 whatever their order, so replays give the eager
    image to the last bit."""
    import torch
    import internship_b200 as mr
    from internship_b200 import _lib, scenes
    v = mr.VolumeRender(32)
    v.SetDatas(scenes.sphere_density(32))
    v.Update()
    p = scenes.make_params(65, 33, 9, bounces=64)
    ref, out = torch.zeros(65 * 33 * 3, device="cuda"), torch.zeros(65 * 33 * 3, device="cuda")
    render = _lib.load().mr_render
    _lib.check(render(v.handle, None, C.byref(p), C.c_void_p(ref.data_ptr()), None))
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib.check(render(v.handle, None, C.byref(p), C.c_void_p(out.data_ptr()), s))
    for _ in range(2):
        out.fill_(-1.0)
        g.replay()
        torch.cuda.synchronize()
        assert (ref > 0).any() and torch.equal(out, ref)
    v.close()
