"""mr_radiance_predict on a device that is nearly full."""
import ctypes as C

import pytest

from tests.nearly_full import nearly_full

pytestmark = pytest.mark.gpu


# 40,000 rows want a temporary of 92 MB (fp32) or 111 MB (BF16, FP8); with some
# 48 MB free they run in pieces. Rows are independent: equal to the last bit.
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_predict_on_a_nearly_full_device(precision):
    import torch
    import internship_b200 as mr
    from internship_b200 import _lib
    from internship_b200.weights import active_random_weights
    n = 40000
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    desc = torch.rand(n, 576, device="cuda", generator=gen)
    aux = 0.6 + 0.4 * torch.rand(n, 5, device="cuda", generator=gen)
    net = mr.Network(active_random_weights(3))

    def predict(out):
        _lib.check(_lib.load().mr_radiance_predict(net.handle, precision, C.c_void_p(desc.data_ptr()),
                                                   C.c_void_p(aux.data_ptr()), n, C.c_void_p(out.data_ptr()), None))

    ref, out = torch.zeros(n, 3, device="cuda"), torch.zeros(n, 3, device="cuda")
    predict(ref)
    torch.cuda.synchronize()
    mr.Network(active_random_weights(3)).close()  # gives the library's unused memory back
    with nearly_full(48 << 20):
        predict(out)
    net.close()
    assert (ref > 0).any()
    assert torch.equal(out, ref)
