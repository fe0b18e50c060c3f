"""The denoiser's form for grey histograms (equal bins in the three channels)
and its choice per warp: all-grey frames with the radiance confined to the
first four, eight or all ten bins, frames that are grey on one side only, and
one coloured pixel in a grey frame; against the oracle's Denoise."""
import ctypes as C

import numpy as np
import pytest

from oracle import orc

pytestmark = pytest.mark.gpu


def _unpack(x):
    x = np.asarray(x, np.uint32)
    return np.stack([(x >> 16) & 255, (x >> 8) & 255, x & 255], -1).astype(np.int32)


# As in the denoiser's other test: approximate reciprocals and roots move a
# packed channel by one 8-bit step at most, in under 1 % of the channels.
@pytest.mark.parametrize("W,H,top,coloured", [(45, 29, 0.6, "none"), (45, 29, 3.5, "none"), (33, 17, 50.0, "none"),
                                              (64, 40, 2.0, "half"), (50, 30, 2.0, "one"), (16, 16, 0.6, "none"),
                                              (7, 3, 5.0, "none")])
def test_grey_histograms_match_oracle(W, H, top, coloured):
    import torch
    from internship_b200 import _lib
    rng = np.random.default_rng(W + H)
    acc = np.zeros((W * H, 3), np.float32)
    hist = np.zeros((W * H, 33), np.float32)
    pick = np.zeros(W * H, bool)
    if coloured == "half":
        pick = np.arange(W * H) % W >= W // 2
    elif coloured == "one":
        pick[(H // 2) * W + W // 2] = True
    frames = 6
    for f in range(frames):
        x = rng.uniform(0, top, (W * H, 3)).astype(np.float32)
        x[~pick] = x[~pick][:, :1]
        orc.histogram_frame(x, f, acc, hist)
    ref = orc.denoise(acc, hist, W, H, frames, frames & 1, 2, 1, 1.1)
    da, dh = torch.from_numpy(acc).cuda(), torch.from_numpy(hist).cuda()
    out = torch.empty(W * H, dtype=torch.int32, device="cuda")
    it = _lib.Interactive()
    it.frame_index, it.tone, it.denoise, it.checkerboard, it.exposure = frames, 2, 1, 0, 1.1
    _lib.check(_lib.load().mr_denoise(C.c_void_p(da.data_ptr()), C.c_void_p(dh.data_ptr()), C.c_void_p(out.data_ptr()),
                                      W, H, C.byref(it), None))
    d = np.abs(_unpack(out.cpu().numpy().view(np.uint32)) - _unpack(ref))
    assert d.max() <= 1 and (d > 0).mean() < 0.01
