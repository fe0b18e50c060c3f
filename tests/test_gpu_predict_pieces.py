"""mr_radiance_predict over tables of any length: a row's prediction does not
depend on where its tile, block or piece starts."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def table():
    import torch
    import internship_b200 as mr
    from internship_b200.weights import active_random_weights
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    n = 120000
    desc = torch.rand(n, 576, device="cuda", generator=gen)
    aux = torch.cat([0.7 + 0.2 * torch.rand(n, 1, device="cuda", generator=gen),
                     3.1 * torch.rand(n, 1, device="cuda", generator=gen),
                     0.6 + 0.4 * torch.rand(n, 3, device="cuda", generator=gen)], 1).contiguous()
    net = mr.Network(active_random_weights(3))
    yield net, desc, aux
    net.close()


def _predict(table, precision, a, b):
    import torch
    from internship_b200 import _lib
    net, desc, aux = table
    d, x = desc[a:b].contiguous(), aux[a:b].contiguous()
    out = torch.full((b - a + 1, 3), -7.0, device="cuda")
    _lib.check(_lib.load().mr_radiance_predict(net.handle, precision, C.c_void_p(d.data_ptr()), C.c_void_p(x.data_ptr()),
                                               b - a, C.c_void_p(out.data_ptr()), None))
    torch.cuda.synchronize()
    assert (out[-1] == -7.0).all()
    return out[:-1].cpu()


# Rows are independent and every row's arithmetic is the same wherever it
# falls: equal to the last bit, three albedo channels included.
@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 1000, 75776, 75777, 113665, 120000])
def test_rows_are_independent(table, precision, n):
    import torch
    whole = _predict(table, precision, 0, n)
    assert torch.isfinite(whole).all() and (whole > 0).any()
    k = min(n, 50)
    assert torch.equal(whole[:k], _predict(table, precision, 0, k))
    assert torch.equal(whole[n - k:], _predict(table, precision, n - k, n))
