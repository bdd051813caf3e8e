"""Loss gradient of the learned switch over many chunks of 64 rows, into a
gradient array on 8 bytes (two weights an atomic) or 4: the sum of the single
rows' gradients up to the order of the FP32 sums, at most n 2^-23 of the sum of
the magnitudes."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300 import _lib, sensor  # noqa: E402


@pytest.mark.parametrize("chunks,rest,odd", [(1, 1, 0), (2, 1, 1), (3, 65, 0)])
def test_gradient_of_many_chunks(chunks, rest, odd):
    L = _lib.lib()
    L.enl_set_stream(C.c_void_p(torch.cuda.current_stream().cuda_stream))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 64 * sms * chunks + rest
    gen = torch.Generator().manual_seed(n)
    X = torch.rand((n, 40), generator=gen).to(torch.bfloat16).cuda()
    y, w = (torch.rand(n, generator=gen) < 0.4).float().cuda(), (0.5 + torch.rand(n, generator=gen)).cuda()
    P = torch.from_numpy(sensor.init_params(2)).cuda() + 0.01
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    whole = torch.zeros(P.numel() + 1, device="cuda")[odd:odd + P.numel()]
    v = lambda t, o=0: C.c_void_p(t.data_ptr() + o)  # noqa: E731
    _lib.check(L.enl_mlp_grad(v(X), v(y), v(w), n, v(P), v(whole), v(loss)), "enl_mlp_grad")
    rows = torch.zeros((n, P.numel()), device="cuda")
    for i in range(n):
        _lib.check(L.enl_mlp_grad(v(X, 80 * i), v(y, 4 * i), v(w, 4 * i), 1, v(P), v(rows, 4 * P.numel() * i), None))
    torch.cuda.synchronize()
    ref, size = rows.double().sum(0), rows.abs().double().sum(0)
    assert torch.all((whole.double() - ref).abs() <= n * 2.0 ** -23 * size)
    assert float(size.min()) > 0 and np.isfinite(loss.item())
