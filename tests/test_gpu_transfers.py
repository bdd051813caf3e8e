"""Transfers between levels at ratio 2 in FP64: refined cells against the
bilinear formula in long double (four operations a field: an error of at most
4 x 2^-53 of the largest coarse value), equal coarse values kept exactly;
coarsened cells bit for bit (((f00 + f10) + f01) + f11) / 4, down to the
smallest doubles."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300.constants import REFLECT, default_params  # noqa: E402
from enlightning_gb300.engine import PREC_FP64, Engine  # noqa: E402


def _engine(nx, ny, box):
    E = Engine(default_params(), nx, ny, (0.1, 0.1), nlevels=2, ratio=2, bc=(REFLECT,) * 4, precision=PREC_FP64)
    E.set_patches(0, [(0, nx - 1, 0, ny - 1)])
    E.set_patches(1, [box])
    return E


@pytest.mark.parametrize("box", [(0, 1, 0, 1), (0, 95, 0, 63), (31, 62, 15, 40), (94, 95, 62, 63)])
@pytest.mark.parametrize("values", ["random", "equal"])
def test_refined_cells(box, values):
    nx, ny = 48, 32
    E = _engine(nx, ny, (0, 2 * nx - 1, 0, 2 * ny - 1))
    rng = np.random.default_rng(4)
    c = rng.standard_normal((7, ny + 6, nx + 6)) if values == "random" else np.broadcast_to(
        rng.standard_normal((7, 1, 1)) * 10.0 ** rng.integers(-9, 9, (7, 1, 1)), (7, ny + 6, nx + 6)).copy()
    E.buffer(0, 0).copy_(torch.from_numpy(c))
    E.buffer(1, 0).fill_(np.nan)
    torch.cuda.synchronize()
    E.refine_init(1, [box])
    torch.cuda.synchronize()
    got = E.buffer(1, 0).cpu().numpy()[:, 3:-3, 3:-3]
    I, J = np.arange(box[0], box[1] + 1), np.arange(box[2], box[3] + 1)
    part = got[:, box[2]:box[3] + 1, box[0]:box[1] + 1]
    assert np.isnan(got).sum() == got.size - part.size
    ld = np.longdouble
    x, y = (I + 0.5) / 2 - 0.5, (J + 0.5) / 2 - 0.5
    i, j = np.floor(x).astype(int), np.floor(y).astype(int)
    fx, fy = (x - i).astype(ld), (y - j).astype(ld)[:, None]
    at = lambda b, a: c[:, 3 + j + b][:, :, 3 + i + a].astype(ld)  # noqa: E731
    ref = (1 - fy) * ((1 - fx) * at(0, 0) + fx * at(0, 1)) + fy * ((1 - fx) * at(1, 0) + fx * at(1, 1))
    if values == "equal":
        assert np.array_equal(part, np.broadcast_to(c[:, :1, :1], part.shape))
    else:
        assert np.max(np.abs(part - ref)) <= 4 * 2.0 ** -53 * np.abs(c).max()
    E.close()


@pytest.mark.parametrize("scale", [1.0, 1e-300, 2.0 ** -1020, 2.0 ** -1070])
def test_coarsened_cells_bit_exact(scale):
    """The coarse cells under the fine patch after a step are the means of the
    fine cells after it; momenta down to subnormal numbers."""
    nx, ny = 64, 32
    E = _engine(nx, ny, (20, 91, 10, 53))
    prm = default_params()
    rng = np.random.default_rng(1)
    for l in range(2):
        w = E.buffer(l, 0)
        n = tuple(w.shape[1:])
        w.zero_()
        w[0] = prm["rho0"]
        w[4] = prm["rho0"] * prm["T0"]
        w[5], w[6] = prm["p0"], prm["T0"]
        w[1] = torch.from_numpy(rng.standard_normal(n) * scale)
    torch.cuda.synchronize()
    E.step(1e-9)
    torch.cuda.synchronize()
    f = E.buffer(1, 0).cpu().numpy()[:, 3 + 10:3 + 54, 3 + 20:3 + 92]
    c = E.buffer(0, 0).cpu().numpy()[:, 3 + 5:3 + 27, 3 + 10:3 + 46]
    want = (((f[:, ::2, ::2] + f[:, ::2, 1::2]) + f[:, 1::2, ::2]) + f[:, 1::2, 1::2]) * 0.25
    assert np.array_equal(c, want)
    E.close()
