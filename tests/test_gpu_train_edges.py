"""Training calls at the edges of what they accept: descriptor tables at any
float address, one row, steps captured into a graph before the trainer grows,
and steps on a device that is nearly full."""
import ctypes as C

import numpy as np
import pytest

from tests.nearly_full import nearly_full

pytestmark = pytest.mark.gpu


def _rows(n, seed):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return [torch.rand(n, 576, device="cuda", generator=gen), 0.6 + 0.4 * torch.rand(n, 5, device="cuda", generator=gen),
            0.01 + torch.rand(n, device="cuda", generator=gen)]


# The same rows at another address: every value before the weight gradients is
# the same bit for bit, and these are sums by atomics over the tiles in any
# order, a few ulp of the sum of their terms; 2e-5 of the gradient's norm
# leaves a wide margin.
@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("shift", [1, 2, 3])
@pytest.mark.parametrize("n", [5, 130])
def test_descriptors_at_any_float_address(precision, shift, n):
    import torch
    from internship_b200.train import Trainer
    from internship_b200.weights import active_random_weights
    desc, aux, label = _rows(n, n)
    flat = torch.empty(n * 576 + 4, device="cuda")
    moved = flat[shift:shift + n * 576].view(n, 576)
    moved.copy_(desc)
    assert desc.data_ptr() % 16 == 0 and moved.data_ptr() % 16 == 4 * shift
    tr = Trainer(active_random_weights(2), precision)
    ref, ref_loss = tr.gradient(desc, aux, label)
    got, loss = tr.gradient(moved, aux, label)
    tr.close()
    assert np.linalg.norm(ref) > 0
    assert np.linalg.norm(got - ref) <= 2e-5 * np.linalg.norm(ref)
    assert loss == pytest.approx(ref_loss, rel=1e-5)


# A batch of one row, and the same row 65 times, at every place of a tile and as
# the only row of a second one: the same mean gradient. The copies' terms are
# equal, so the sums round at the size of the gradient's entries; in BF16 the
# 1 / 65 shifts the roundings of the rows' gradients, 2^-9 each at most.
@pytest.mark.parametrize("precision,tol", [("fp32", 2e-5), ("bf16", 1e-2)])
def test_one_row_equals_its_copies(precision, tol):
    from internship_b200.train import Trainer
    from internship_b200.weights import active_random_weights
    one = _rows(1, 3)
    tr = Trainer(active_random_weights(2), precision)
    g, loss = tr.gradient(*one)
    ref, ref_loss = tr.gradient(*[x.expand(65, *x.shape[1:]).contiguous() for x in one])
    tr.close()
    assert np.linalg.norm(ref) > 0
    assert np.linalg.norm(g - ref) <= tol * np.linalg.norm(ref)
    assert loss == pytest.approx(ref_loss, rel=1e-5)


def _alloc_nodes(graph):
    """Memory allocation nodes of a captured graph (a cudaGraph_t)."""
    cuda = C.CDLL("libcuda.so.1")
    n = C.c_size_t()
    assert cuda.cuGraphGetNodes(C.c_void_p(graph), None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert cuda.cuGraphGetNodes(C.c_void_p(graph), nodes, C.byref(n)) == 0
    kind, count = C.c_int(), 0
    for h in nodes:
        assert cuda.cuGraphNodeGetType(C.c_void_p(h), C.byref(kind)) == 0
        count += kind.value == 10  # CU_GRAPH_NODE_TYPE_MEM_ALLOC
    return count


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_captured_step_outlives_the_trainers_buffers(precision):
    """A step captured while the trainer's buffers are large enough for it must
    not depend on them: a later call with more rows frees them. The graph's own
    allocation is checked before anything is replayed. One replay then updates
    the weights as one direct step does (up to the atomics' order, which Adam's
    first step can turn into a sign at a gradient near zero)."""
    import torch
    from internship_b200 import _lib
    from internship_b200.train import Trainer
    from internship_b200.weights import active_random_weights
    w = active_random_weights(2)
    d, more = _rows(200, 9), _rows(1000, 10)
    ptr = [C.c_void_p(x.data_ptr()) for x in d]
    a, b = Trainer(w, precision), Trainer(w, precision)
    b.step(*d, 1e-3)
    a.gradient(*d)  # the trainer has buffers for 200 rows
    g = torch.cuda.CUDAGraph(keep_graph=True)
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        s = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        _lib.check(_lib.load().mr_trainer_step(a.handle, *ptr, 200, 1e-3, None, s))
    assert _alloc_nodes(g.raw_cuda_graph()) == 1
    a.gradient(*more)
    g.instantiate()
    g.replay()
    torch.cuda.synchronize()
    wa, wb = a.weights(), b.weights()
    a.close()
    b.close()
    assert np.abs(wa - w).max() > 5e-4
    assert (np.abs(wa - wb) > 1e-6).mean() < 0.01


def test_step_on_a_nearly_full_device():
    """20,011 rows, whose buffers would take 110 MB, with some 64 MB free: the
    step runs in pieces. The gradient of the whole batch, in whichever pieces,
    is a sum by atomics (tolerance as above)."""
    from internship_b200.train import Trainer
    from internship_b200.weights import active_random_weights
    w = active_random_weights(2)
    d = _rows(20011, 5)
    tr = Trainer(w)
    ref, ref_loss = tr.gradient(*d)
    tr.close()
    tr = Trainer(w)
    tr.gradient(*[x[:64] for x in d])
    with nearly_full(64 << 20):
        got, loss = tr.gradient(*d)
    tr.close()
    assert np.linalg.norm(got - ref) <= 2e-5 * np.linalg.norm(ref)
    assert loss == pytest.approx(ref_loss, rel=1e-5)
