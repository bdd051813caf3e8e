"""The engine's tags (a warp takes 2 or 8 rows of a tile, by the number of
tiles) against the same tests cell by cell on the drop-in entry point, exactly:
ragged patches on a small and a large table, FP64."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300 import _lib  # noqa: E402
from enlightning_gb300.constants import REFLECT, default_params  # noqa: E402
from enlightning_gb300.engine import PREC_FP64, Engine  # noqa: E402


@pytest.mark.parametrize("nx,ny", [(1, 1), (33, 9), (70, 41), (1300, 700)])  # 2,432 tiles and more: 8 rows
def test_tags_equal_the_patch_entry_point(nx, ny):
    prm = default_params()
    NX, NY, i0, j0 = nx + 31, ny + 23, 4, 6  # the patch lies inside a larger domain
    E = Engine(prm, NX, NY, (0.1, 0.1), bc=(REFLECT,) * 4, precision=PREC_FP64)
    E.set_patches(0, [(i0, i0 + nx - 1, j0, j0 + ny - 1)])
    rng = np.random.default_rng(nx)
    w, H = E.buffer(0, 0), E.buffer(0, 3)
    quiet = rng.random((NY + 6, NX + 6)) < 0.9
    w.zero_()
    w[0] = torch.from_numpy(prm["rho0"] * (1 + np.where(quiet, 0.0, 0.2 * rng.standard_normal(quiet.shape))))
    H[0] = torch.from_numpy(np.where(rng.random(quiet.shape) < 0.98, 0.0, 5e3))
    torch.cuda.synchronize()
    tags = E.tag(0)
    torch.cuda.synchronize()
    L, I, P = E.L, _lib.iref, lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    part = (slice(None), slice(j0, j0 + ny + 6), slice(i0, i0 + nx + 6))  # the patch and 3 cells around it
    full = w[:5][part].contiguous()
    src, ref = H[part].contiguous(), torch.full((ny, nx), -1, dtype=torch.int32, device="cuda")
    L.tag_cells_(I(0), I(nx - 1), I(0), I(ny - 1), I(3), I(3), P(ref), P(full), P(src), I(1), _lib.darr(prm["tol"]),
                 I(5))
    _lib.check_sticky("tag_cells")
    torch.cuda.synchronize()
    assert torch.equal(tags[j0:j0 + ny, i0:i0 + nx], ref)
    assert int(tags.sum()) == int(ref.sum())
    assert nx < 30 or 0 < int(ref.sum()) < nx * ny
    E.close()
