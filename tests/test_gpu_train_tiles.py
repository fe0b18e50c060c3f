"""The training step's tile kernels at sizes where they can go wrong: fewer
rows than a tile, one row more or less than a tile, several tiles with a
remainder, and batches of more than one piece."""
import numpy as np
import pytest

from oracle import orc

pytestmark = pytest.mark.gpu


def _rows(n, seed):
    rng = np.random.default_rng(seed)
    desc = np.concatenate([rng.uniform(0, 1.5, (n, 192)), rng.uniform(0, 1, (n, 192)), rng.uniform(0, 2, (n, 192))],
                          1).astype(np.float32)
    aux = np.stack([rng.uniform(0.7, 0.9, n), rng.uniform(0, np.pi, n)] + [rng.uniform(0.6, 1.0, n)] * 3,
                   1).astype(np.float32)
    return desc, aux, rng.uniform(0.01, 2.0, n).astype(np.float32)


# The mean-loss gradient of n rows is the row-weighted mean of the gradients
# of any split of them, which puts every row at another place of a tile. fp32:
# each entry is a sum over the rows whose rounding is a few ulp of the sum of
# its terms, so 2e-5 of the gradient's norm leaves a wide margin. BF16: the
# 1 / n in the rows' gradients shifts their BF16 roundings, 2^-9 each at
# most, so 1 % as in the BF16 gradient's own test.
@pytest.mark.parametrize("precision,tol", [("fp32", 2e-5), ("bf16", 1e-2)])
@pytest.mark.parametrize("n,cut", [(1, 1), (3, 1), (63, 20), (64, 33), (65, 1), (129, 64), (1000, 431)])
def test_gradient_adds_up_over_splits(precision, tol, n, cut):
    import torch
    from internship_b200.train import Trainer
    from internship_b200.weights import active_random_weights
    w = active_random_weights(2)
    rows = _rows(n, n)
    d = [torch.from_numpy(x).cuda() for x in rows]
    tr = Trainer(w, precision)
    g, loss = tr.gradient(*d)
    ref = np.zeros(g.size)
    for a, b in ((0, cut), (cut, n)):
        if b > a:
            p, _ = tr.gradient(*[x[a:b].contiguous() for x in d])
            ref += p.astype(np.float64) * ((b - a) / n)
    tr.close()
    assert np.linalg.norm(g - ref) <= tol * np.linalg.norm(ref)
    assert loss == pytest.approx(orc.train_loss(w, *rows), rel=1e-4 if precision == "fp32" else 2e-2)


def test_large_batch_runs_in_pieces():
    import torch
    from internship_b200.train import Trainer
    from internship_b200.weights import active_random_weights
    n, cut = 65536 + 37, 30001
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    d = [torch.rand(n, 576, device="cuda", generator=gen), 0.6 + 0.4 * torch.rand(n, 5, device="cuda", generator=gen),
         0.01 + torch.rand(n, device="cuda", generator=gen)]
    tr = Trainer(active_random_weights(2))
    g, loss = tr.gradient(*d)
    ref, rloss = np.zeros(g.size), 0.0
    for a, b in ((0, cut), (cut, n)):
        p, l = tr.gradient(*[x[a:b].contiguous() for x in d])
        ref += p.astype(np.float64) * ((b - a) / n)
        rloss += l * (b - a) / n
    tr.close()
    assert np.linalg.norm(g - ref) <= 2e-5 * np.linalg.norm(ref)
    assert loss == pytest.approx(rloss, rel=1e-5)


def test_step_is_capturable_before_any_call():
    """A training step captured into a graph on a new trainer: one replay
    updates the weights as one direct step does (up to the atomics' order,
    which Adam's first step can turn into a sign at a gradient near zero)."""
    import ctypes as C
    import torch
    from internship_b200 import _lib
    from internship_b200.train import Trainer
    from internship_b200.weights import active_random_weights
    w = active_random_weights(2)
    d = [torch.from_numpy(x).cuda() for x in _rows(200, 9)]
    ptr = [C.c_void_p(x.data_ptr()) for x in d]
    a, b = Trainer(w), Trainer(w)
    b.step(*d, 1e-3)
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib.check(_lib.load().mr_trainer_step(a.handle, *ptr, 200, 1e-3, None, s))
    g.replay()
    torch.cuda.synchronize()
    wa, wb = a.weights(), b.weights()
    a.close()
    b.close()
    assert np.abs(wa - w).max() > 5e-4
    assert (np.abs(wa - wb) > 1e-6).mean() < 0.01
