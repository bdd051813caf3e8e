"""The engine's tags of single-precision storage (a warp takes 2 or 8 rows of a
tile, by the number of tiles) against the test restated on the host in the same
precision, exactly: 2 |t1 t2| + ep over t1^2 + t2^2 + ep with each sum of a
product and a number rounded once, as the device's fused operations do (the
host's long double holds the products of 24-bit numbers exactly)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300.constants import REFLECT, default_params  # noqa: E402
from enlightning_gb300.engine import PREC_FP32_STATE, Engine  # noqa: E402

F, LD = np.float32, np.longdouble


def below(m, c, p, ep):
    t1, t2 = c - m, p - c
    num = (2 * np.abs(t1 * t2).astype(LD) + ep).astype(F)
    den = (t1.astype(LD) ** 2 + (t2.astype(LD) ** 2 + ep).astype(F)).astype(F)
    return num / den < F(0.9999)


def tags(q, ep):
    """Of the interior of a field with a cell around it."""
    c = q[1:-1, 1:-1]
    return below(q[1:-1, :-2], c, q[1:-1, 2:], ep) | below(q[:-2, 1:-1], c, q[2:, 1:-1], ep)


@pytest.mark.parametrize("nx,ny", [(1, 1), (33, 9), (70, 41), (1300, 700)])  # 2,432 tiles and more: 8 rows
def test_tags_equal_the_restatement(nx, ny):
    assert np.finfo(LD).nmant >= 62
    prm = default_params()
    NX, NY, i0, j0 = nx + 31, ny + 23, 4, 6  # the patch lies inside a larger domain
    E = Engine(prm, NX, NY, (0.1, 0.1), bc=(REFLECT,) * 4, precision=PREC_FP32_STATE)
    E.set_patches(0, [(i0, i0 + nx - 1, j0, j0 + ny - 1)])
    rng = np.random.default_rng(nx)
    shape = (NY + 6, NX + 6)
    rho = np.where(rng.random(shape) < 0.8, 0.0, 0.2 * rng.standard_normal(shape)).astype(F)
    src = np.where(rng.random(shape) < 0.98, 0.0, 5e3).astype(F)
    w, H = E.buffer(0, 0), E.buffer(0, 3)
    w.zero_()
    w[0], H[0] = torch.from_numpy(rho), torch.from_numpy(src)
    torch.cuda.synchronize()
    got = E.tag(0)
    torch.cuda.synchronize()
    f = lambda x: float(F(x))  # noqa: E731
    ep = [F(f(0.9) * t / (1.0 - f(0.9) * (t * t))) for t in prm["tol"]]
    part = (slice(j0 + 2, j0 + ny + 4), slice(i0 + 2, i0 + nx + 4))  # the patch and a cell around it
    want = tags(src[part], ep[0]) | tags(rho[part], ep[1])
    assert np.array_equal(got[j0:j0 + ny, i0:i0 + nx].cpu().numpy() != 0, want)
    assert int(got.sum()) == int(want.sum())
    assert nx < 30 or 0 < int(want.sum()) < nx * ny
    E.close()
