"""The CFL maximum on small tables, whose tiles are taken by two rows, and on
the first that is too large for it: ragged patches, the fastest cell in every
row of a tile in turn.  FP64: the largest of the correctly rounded |v| / rho + c,
so the same dt to the rounding of its quotient and of cfl dx; FP32 storage: the
four roundings of its own arithmetic."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300.constants import REFLECT, default_params  # noqa: E402
from enlightning_gb300.engine import PREC_FP32_STATE, PREC_FP64, Engine  # noqa: E402


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_FP32_STATE])
@pytest.mark.parametrize("nx,ny", [(1, 1), (31, 9), (33, 7), (70, 41), (1216 * 32, 1), (38910, 8), (1217 * 32, 8)])
def test_fastest_cell_of_every_row(precision, nx, ny):
    prm = default_params()
    E = Engine(prm, nx + 8, ny + 12, (0.5, 0.5), bc=(REFLECT,) * 4, precision=precision)
    E.set_patches(0, [(4, 3 + nx, 2, 1 + ny)])
    E.set_adaptive_dt(True, 0.5)
    w = E.buffer(0, 0)
    rng = np.random.default_rng(nx)
    off = np.array([prm["rho0"], 0, 0, 0, prm["rho0"] * prm["T0"], prm["p0"], prm["T0"]])[:, None, None]
    start = np.zeros(tuple(w.shape)) + (off if precision == PREC_FP64 else 0.0)
    start[0] += 0.1 * rng.random(start.shape[1:])
    start[1:3] += rng.uniform(-3, 3, start[1:3].shape)
    for j in sorted({*range(min(ny, 9)), ny - 1}):
        s = start.copy()
        i = int(rng.integers(nx))
        s[1 + j % 2, 3 + 2 + j, 3 + 4 + i] = (-1) ** j * (20.0 + j)
        s[1:3, :5] = s[1:3, 5 + ny:] = s[1:3, :, :7] = s[1:3, :, 7 + nx:] = 1e3  # (outside the patch)
        w.copy_(torch.from_numpy(s))
        v = w.double().cpu().numpy()[:3, 5:5 + ny, 7:7 + nx]
        rho = v[0] + (prm["rho0"] if precision == PREC_FP32_STATE else 0.0)
        want = 0.5 * 0.5 / np.max(np.maximum(np.abs(v[1]), np.abs(v[2])) / rho + prm["c"])
        torch.cuda.synchronize()
        E.step(1.0)
        torch.cuda.synchronize()
        assert E.time()[0] == pytest.approx(want, rel=2.0 ** -52 if precision == PREC_FP64 else 4 * 2.0 ** -24, abs=0)
    E.close()
