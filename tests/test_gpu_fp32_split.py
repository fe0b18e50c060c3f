"""The fp32 trunk's split operands (three BF16 parts) against a float64
evaluation of the same network, whose head passes trunk outputs through."""
import numpy as np
import pytest

from oracle import orc

pytestmark = pytest.mark.gpu

WIDTH, FROM = [8, 8, 16, 16, 16, 32, 32, 32], [0, 8, 16, 32, 48, 64, 96, 128]


def _net64(w, desc, aux, channel):
    """X (the output before exp - 1) of rows in float64 (core/radiancePredict.cu:370-485)."""
    from internship_b200.weights import layout
    W, at = {}, 0
    for name, k in layout():
        W[name] = w[at:at + k].astype(np.float64)
        at += k

    def lin(x, name, bias=True):
        m = W[name + "W"].reshape(-1, x.shape[1])
        y = x @ m.T
        return y + W[name + "B"] if bias else y

    def relu(x):
        return np.maximum(x, 0.0)

    def sig(x):
        return 1.0 / (1.0 + np.exp(-x))

    n = len(desc)
    d = desc.astype(np.float64).reshape(n, 3, 192)
    g, gamma, sc = (aux[:, c:c + 1].astype(np.float64) for c in (0, 1, 2 + channel))
    mean, peak, heads = [], [], []
    for trunk, se, widths, starts, double in (("L", "LSE", WIDTH, FROM, (1, 4)),
                                              ("LD", "LDSE", [8] * 4, [160, 168, 176, 184], ())):
        y = [0.0, 0.0, 0.0]
        for i, (s, f) in enumerate(zip(widths, starts)):
            x = d[:, :, f:f + s]
            mean.append(x.mean(2))
            peak.append(x.max(2))
            t = np.concatenate([mean[-1], peak[-1], g, gamma], 1)
            gate = sig(lin(relu(lin(t, "%s%d1" % (se, i), False)), "%s%d2" % (se, i), False))
            for b, br in enumerate(("", "_Tr", "_Hg")):
                h = relu(lin(x[:, b] * gate[:, b:b + 1] + y[b], "%s%s%d1" % (trunk, br, i)))
                y[b] = np.concatenate([h, x[:, b]], 1) if i in double else h + x[:, b]
        heads += [relu(lin(y[b], "%s%s%d1" % (trunk, br, len(widths)))) for b, br in enumerate(("", "_Tr", "_Hg"))]
    pool = np.concatenate(mean + peak + [g, gamma, sc], 1)
    gates = sig(lin(relu(lin(pool, "LSEFin1", False)), "LSEFin2", False))
    a = np.concatenate([h * gates[:, i:i + 1] for i, h in enumerate(heads)]
                       + [relu(lin(np.concatenate([g, gamma, sc], 1), "LGGS"))], 1)
    for name in ("LC0", "LC1", "LC2", "LX"):
        a = relu(lin(a, name))
    for i in range(0, 12, 2):
        a = a + relu(lin(relu(lin(a, "LX%d" % i)), "LX%d" % (i + 1)))
    return relu(lin(a, "LX12"))[:, 0]


def _pass_through(w):
    """The network's head made to average 16 of the 96 trunk outputs: LC0 picks
    every sixth, LC1 .. LX pass them on, the residual layers add nothing."""
    from internship_b200.weights import layout
    head = {"LC0": 128, "LC1": 128, "LC2": 64, "LX": 32}
    w, at = w.copy(), 0
    for name, k in layout():
        m = w[at:at + k]
        if name[:-1] in head and name[-1] == "W":
            m = m.reshape(-1, head[name[:-1]])
            m[:] = 0
            for o in range(16):
                m[o, 6 * o if name == "LC0W" else o] = 1
        elif name == "LX12W":
            m[:] = 1.0 / 16
        elif name.startswith(("LC", "LX")):
            m[:] = 0
        at += k
    return w


# Every product of the head but one per output is zero, so that the head adds
# its TF32 parts' 2^-22 three times, about as much as fp32 sums of 32 terms lose
# in the trunk's nine layers; with two parts in place of three the trunk's
# products would be 2^-17 off, more than ten times that.
@pytest.mark.parametrize("n", [1, 127, 128, 129, 700])
def test_trunk_as_exact_as_fp32(n):
    import internship_b200 as mr
    from internship_b200 import _lib
    from internship_b200.weights import active_random_weights
    from test_gpu_tensorcore import _descriptors, _predict
    w = _pass_through(active_random_weights(4))
    desc, aux = _descriptors(n, 21)
    exact = _net64(w, desc, aux, 0)
    assert (exact > 0).all()

    def err(y):
        x = np.log1p(y[:, 0].astype(np.float64) / aux[:, 2].astype(np.float64))
        return np.sqrt(np.mean((x / exact - 1) ** 2))

    fp32 = err(orc.predict(w, desc, aux))
    assert fp32 < 1e-5
    assert err(_predict(mr, w, desc, aux, _lib.PREC_FP32)) <= 5 * max(fp32, 2e-7)
