"""Tags where values repeat (the shortcut for three equal values) against the
oracle, bit for bit: plateaus with single odd cells, signed zeros, infinities
and NaN, with thresholds of every kind."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300 import _lib  # noqa: E402
from test_gpu_state_and_tags import _tags  # noqa: E402


@pytest.fixture(scope="module")
def L():
    lib = _lib.lib()
    lib.enl_set_stream(C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return lib


@pytest.mark.parametrize("tol", [1e-2, 1.5, 0.0, 1e-200])
@pytest.mark.parametrize("odd", [1.0 + 2.0 ** -52, -1.0, 0.0, -0.0, 1e300, float("inf"), float("nan")])
def test_plateaus(L, ora, tol, odd):
    rng = np.random.default_rng(5)
    rho = np.repeat(np.repeat(rng.integers(0, 3, (10, 12)).astype(float), 5, 0), 7, 1)
    src = np.where(rng.random(rho.shape) < 0.02, odd, 0.0)
    rho[rng.random(rho.shape) < 0.02] = odd
    with np.errstate(all="ignore"):
        got, ref = _tags(L, ora, rho, src, (tol, tol, 5e-3))
    assert np.array_equal(got, ref)
