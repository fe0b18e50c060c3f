"""The trackers' path machine (one step per iteration in every lane) where it
can go wrong: fewer paths than lanes, one-bounce and zero-bounce paths,
extinctions from none to beyond the fast quotient's range, negative
(distance-valued) densities, and frames of odd width with the checkerboard;
against the oracle on the same random streams."""
import ctypes as C

import numpy as np
import pytest

from oracle import orc

pytestmark = pytest.mark.gpu


def _volume(kind, res=32):
    import internship_b200 as mr
    from internship_b200 import scenes
    dens = scenes.sphere_density(res) if kind == "sphere" else scenes.sdf_sphere_density(res)
    v = mr.VolumeRender(res)
    v.SetDatas(dens)
    v.Update()
    return v, dens


# A path's decisions compare fp32 values that the host's and the device's
# logf / sincosf round differently by an ulp: of the order of 1e-6 of a
# path's steps flip, so a label of a few hundred steps rarely differs. 5 % of
# the labels may.
@pytest.mark.parametrize("kind,n,spp,bounces,alpha", [
    ("sphere", 1, 1, 1, 16.0), ("sphere", 33, 65, 3, 64.0), ("sdf", 100, 7, 64, 40.0), ("sphere", 5, 3, 0, 16.0),
    ("sphere", 40, 2, 8, 1e-20), ("sdf", 700, 1, 512, 200.0)])
def test_labels_match_oracle(kind, n, spp, bounces, alpha):
    v, dens = _volume(kind)
    rng = np.random.default_rng(n)
    pos = rng.uniform(-0.25, 0.25, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    L = np.array([0.3, 0.8, -0.5], np.float32)
    L /= np.linalg.norm(L)
    gpu = v.GetSamples(pos, d, L, alpha, 0.8, 0.95, bounces, spp, 11)
    v.close()
    if bounces == 0 or alpha < 1e-10:  # no vertex, no light
        assert np.all(gpu == 0)
        return
    ref = orc.get_samples(dens, float(max(dens.max(), 1e-5)), pos, d, np.tile(L, (n, 1)),
                          np.full(n, alpha, np.float32), np.full(n, 0.8, np.float32), np.full(n, 0.95, np.float32),
                          bounces, spp, 11)
    close = np.abs(gpu - ref) <= 1e-3 * np.abs(ref) + 1e-6
    assert close.mean() >= 0.95


@pytest.mark.parametrize("W,H,checker,bounces", [(33, 7, 0, 4), (33, 7, 1, 64), (1, 1, 0, 8), (2, 3, 1, 1), (31, 9, 0, 0)])
def test_interactive_frame_matches_oracle(W, H, checker, bounces):
    import torch
    from internship_b200 import _lib, scenes
    v, dens = _volume("sphere")
    p = scenes.make_params(W, H, 1, bounces=bounces, distance=1.2)
    acc = torch.full((H, W, 3), 7.0, device="cuda")
    hist = torch.zeros(W * H * 33, device="cuda")
    out = torch.empty(W * H, dtype=torch.int32, device="cuda")
    it = _lib.Interactive()
    it.frame_index, it.tone, it.denoise, it.checkerboard, it.exposure = 0, 0, 0, checker, 1.0
    _lib.check(_lib.load().mr_render_interactive(v.handle, None, C.byref(p), C.byref(it), C.c_void_p(acc.data_ptr()),
                                                 C.c_void_p(hist.data_ptr()), C.c_void_p(out.data_ptr()), None))
    got = acc.cpu().numpy()
    s, _, _ = orc.render_pt(dens, v.max_density, p)
    ref = s.reshape(H, W, 3)
    v.close()
    row, col = np.mgrid[0:H, 0:W]
    drawn = (row + col) % 2 == 0 if checker else np.ones((H, W), bool)
    assert np.all(got[~drawn] == 7.0)  # the other half of the frame is left alone
    close = np.all(np.abs(got - ref) <= 1e-3 * np.abs(ref) + 1e-5, axis=-1)
    assert close[drawn].mean() >= 0.95
