"""Training calls at the edges of what they accept: descriptor tables at any
float address."""
import numpy as np
import pytest

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
