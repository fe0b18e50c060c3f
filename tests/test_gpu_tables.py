"""Scene set-up and descriptor gather at sizes where they can go wrong: odd
grids, lights along axes and nearly so, record counts on both sides of each
split of the gather, and descriptor buffers off the 16-byte alignment."""
import ctypes as C

import numpy as np
import pytest

from oracle import orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res", [2, 3, 5, 16, 33])
def test_majorant_of_odd_grids(res):
    import internship_b200 as mr
    rng = np.random.default_rng(res)
    d = rng.uniform(0, 1, (res,) * 3).astype(np.float32)
    for at in (0, res ** 3 - 1, res ** 3 // 2):
        d2 = d.copy()
        d2.flat[at] = 1.5 + at
        v = mr.VolumeRender(res)
        v.SetDatas(d2)
        v.Update()
        assert v.max_density == np.float32(1.5 + at)
        v.close()


# The oracle runs the same samples in the same fp32 steps; expf and the fused
# steps differ by ulps of an optical depth of at most a few tens: rtol 2e-4 as
# in the pyramid's other test.
@pytest.mark.parametrize("light", [(0, 1, 0), (0, 0, -1), (1e-6, -1, 0), (1, 1, 1), (-0.3, 0.5, 0.8), (1, 1e-20, 0)])
def test_transmittance_levels_match_oracle(light):
    import internship_b200 as mr
    from internship_b200 import _lib, scenes
    dens = scenes.sphere_density(24) * 0.3
    v = mr.VolumeRender(24)
    v.SetDatas(dens)
    v.Update()
    v.Update_TR(light, 20.0)
    L = np.asarray(light, np.float32)
    ref = orc.build_tr(orc.build_mips(dens)[1], 20.0, L / np.float32(np.sqrt((L * L).sum(dtype=np.float32))))
    off = 0
    for k in range(8):
        n = (128 >> k) ** 3
        np.testing.assert_allclose(v.read(_lib.READ_TR, k), ref[off:off + n], rtol=2e-4, atol=1e-7)
        off += n
    v.close()


@pytest.fixture(scope="module")
def scene():
    import torch
    import internship_b200 as mr
    v = mr.VolumeRender(48)
    rng = np.random.default_rng(4)
    v.SetDatas(rng.uniform(0, 1, (48,) * 3).astype(np.float32) ** 4)
    v.Update()
    v.Update_TR((0.3, 0.7, -0.5), 30.0)
    v.UpdateHGLut(0.8)
    net = mr.Network(mr.xavier_weights(1))
    n = 70000
    pos = torch.from_numpy(rng.uniform(-0.49, 0.49, (n, 3)).astype(np.float32)).cuda()
    d = rng.normal(size=(n, 3))
    dirs = torch.from_numpy((d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)).cuda()
    from internship_b200 import _lib
    frames = torch.empty(n, 12, device="cuda")
    _lib.check(_lib.load().mr_train_frames(C.c_void_p(dirs.data_ptr()), n, _lib.f3((0.3, 0.7, -0.5)), 1,
                                           C.c_void_p(frames.data_ptr()), None))
    yield v, net, pos, frames
    v.close()
    net.close()


def _gather(scene, a, b, shift=0):
    import torch
    from internship_b200 import _lib
    v, net, pos, frames = scene
    n = b - a
    buf = torch.zeros(n * 576 + 4, device="cuda")
    aux = torch.zeros(n, 5, device="cuda")
    p, f = pos[a:b].contiguous(), frames[a:b].contiguous()
    _lib.check(_lib.load().mr_gather_descriptors(v.handle, net.handle, C.c_void_p(p.data_ptr()),
                                                 C.c_void_p(f.data_ptr()), n, 30.0, 0.8, _lib.f3((0.95, 0.95, 0.95)),
                                                 C.c_void_p(buf.data_ptr() + 4 * shift), C.c_void_p(aux.data_ptr()),
                                                 None))
    torch.cuda.synchronize()
    return buf[shift:shift + n * 576].view(n, 576).cpu(), aux.cpu()


# A point's descriptor does not depend on how many points are gathered with it
# or where the rows start: equal to the last bit.
@pytest.mark.parametrize("n,shift", [(1, 0), (3, 1), (127, 0), (129, 2), (5000, 0), (20000, 3), (70000, 0)])
def test_gather_is_independent_of_its_split(scene, n, shift):
    import torch
    whole, aux = _gather(scene, 0, n, shift)
    k = min(n, 64)
    first, faux = _gather(scene, 0, k)
    last, laux = _gather(scene, n - k, n)
    assert torch.equal(whole[:k], first) and torch.equal(aux[:k], faux)
    assert torch.equal(whole[n - k:], last) and torch.equal(aux[n - k:], laux)
    assert torch.isfinite(whole).all() and (whole.abs().sum(1) > 0).all()
