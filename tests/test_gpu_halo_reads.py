"""The interpolation's algorithmic bytes in the kernel-class profile: 7 fields
of every halo cell written and of every distinct coarse cell under their 2 x 2
stencils read, counted here cell by cell; ratios 2 and 3, halos that touch the
domain's sides, the profile on before or after the tables."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300.constants import REFLECT, default_params  # noqa: E402
from enlightning_gb300.engine import PREC_FP64, Engine  # noqa: E402


def _bytes(boxes, nx, ny, r):
    cover = np.zeros((ny + 6, nx + 6), bool)
    near = np.zeros_like(cover)
    for a, b, c, d in boxes:
        cover[3 + c:4 + d, 3 + a:4 + b] = True
        near[c:d + 7, a:b + 7] = True
    j, i = np.nonzero((near & ~cover)[3:-3, 3:-3])
    ic, jc = np.floor((i + 0.5) / r - 0.5).astype(int), np.floor((j + 0.5) / r - 0.5).astype(int)
    reads = {(x + p, y + q) for x, y in zip(ic, jc) for p in (0, 1) for q in (0, 1)}
    return 7 * 8 * (len(i) + len(reads))


@pytest.mark.parametrize("ratio", [2, 3])
@pytest.mark.parametrize("first", [True, False])
def test_interpolation_bytes(ratio, first):
    prm = default_params()
    nx, ny = 120, 72
    boxes = [(0, 35 * ratio - 1, 0, 10 * ratio - 1), (36 * ratio, nx * ratio - 1, 6 * ratio, 40 * ratio - 1),
             (4 * ratio, 10 * ratio - 1, 50 * ratio, 72 * ratio - 1)]
    E = Engine(prm, nx, ny, (0.1, 0.1), nlevels=2, ratio=ratio, bc=(REFLECT,) * 4, precision=PREC_FP64)
    E.set_patches(0, [(0, nx - 1, 0, ny - 1)])
    if first:
        E.profile(2)
    E.set_patches(1, boxes)
    if not first:
        E.profile(2)
    for l in range(2):
        w = E.buffer(l, 0)
        w.zero_()
        w[0], w[4], w[5], w[6] = prm["rho0"], prm["rho0"] * prm["T0"], prm["p0"], prm["T0"]
    torch.cuda.synchronize()
    E.step(1e-5)
    torch.cuda.synchronize()
    assert E.profile_kernels()["interp"][1] == 3 * _bytes(boxes, nx * ratio, ny * ratio, ratio)
    E.close()
