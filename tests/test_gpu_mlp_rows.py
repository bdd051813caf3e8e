"""Loss gradient of the learned switch at row counts around its chunks of 64
(one row, one short, one past, several chunks) and from a feature matrix at
any address: a row's contribution does not depend on the rows beside it, so
the gradient is the sum of the single rows' gradients up to the order of the
FP32 sums, at most n 2^-23 of the sum of the magnitudes."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300 import _lib, sensor  # noqa: E402


def _grad(L, X, y, w, P):
    g = torch.zeros_like(P)
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    v = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    _lib.check(L.enl_mlp_grad(v(X), v(y), v(w), X.shape[0], v(P), v(g), v(loss)), "enl_mlp_grad")
    torch.cuda.synchronize()
    return g.double().cpu().numpy(), loss.item()


@pytest.mark.parametrize("n", [1, 63, 64, 65, 200])
@pytest.mark.parametrize("shift", [0, 1, 8])
def test_gradient_is_the_sum_over_rows(n, shift):
    L = _lib.lib()
    L.enl_set_stream(C.c_void_p(torch.cuda.current_stream().cuda_stream))
    gen = torch.Generator().manual_seed(n)
    flat = torch.rand(n * 40 + shift, generator=gen).to(torch.bfloat16).cuda()
    X = flat[shift:].view(n, 40)  # shift 1: 2 bytes past a 16-byte boundary
    y = (torch.rand(n, generator=gen) < 0.4).float().cuda()
    w = (0.5 + torch.rand(n, generator=gen)).cuda()
    P = torch.from_numpy(sensor.init_params(2)).cuda()
    P += 0.01
    got, loss = _grad(L, X, y, w, P)
    one = [_grad(L, X[i:i + 1].clone(), y[i:i + 1].clone(), w[i:i + 1].clone(), P) for i in range(n)]
    ref, size = sum(g for g, _ in one), sum(np.abs(g) for g, _ in one)
    assert np.all(np.abs(got - ref) <= n * 2.0 ** -23 * size)
    assert abs(loss - sum(v for _, v in one)) <= 1e-12 * abs(loss)
