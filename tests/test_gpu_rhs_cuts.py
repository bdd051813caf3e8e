"""The right-hand side of a cell is a function of its stencil alone: one region
as a whole patch and cut into patches whose sizes select tiles of 8, 4, 2 and 1
rows (on a GPU of 152 SMs) gives the same doubles and flags.  The row heights
of the lapse rate are whole multiples of 1/16, exact in every patch."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300 import _lib  # noqa: E402
from enlightning_gb300.constants import VARIANTS, default_params  # noqa: E402
from test_gpu_patch import G, P, L, dev, random_patch  # noqa: E402,F401

NX, NY, D = 512, 640, 0.125


@pytest.fixture(scope="module")
def state():
    prm = default_params()
    rng = np.random.default_rng(11)
    w = random_patch(7, NX, NY, prm)
    pres = prm["p0"] * (1 + 0.1 * rng.standard_normal(w.shape[1:]))
    temp = prm["T0"] * (1 + 0.01 * rng.standard_normal(w.shape[1:]))
    return [dev(a) for a in (w, pres, temp, rng.uniform(0, 1e3, (NY, NX)))]


def rhs(L, prm, variant, state, width, height):  # noqa: F811
    """The region in patches of width x height cells (the last ones ragged)."""
    w, pres, temp, H0 = state
    K = torch.full((5, NY, NX), float("nan"), dtype=torch.float64, device="cuda")
    flags = torch.full((NY, NX), -1, dtype=torch.int32, device="cuda")
    pitch = NX + 2 * G
    for j in range(0, NY, height):
        for i in range(0, NX, width):
            nx, ny, g, o = min(width, NX - i), min(height, NY - j), j * pitch + i, j * NX + i
            at = [P(t.reshape(-1)[n:]) for t, n in ((w, g), (H0, o), (K, o), (pres, g), (temp, g), (flags, o))]
            _lib.check(L.enl_rhs(variant, i, i + nx - 1, j, j + ny - 1, G, G, _lib.darr((i * D, j * D)),
                                 _lib.darr((D, D)), at[0], pitch, pitch * (NY + 2 * G), at[1], at[2], NX, NX * NY,
                                 at[3], at[4], prm["weno_alpha"], prm["kappa"], prm["mu"], prm["muB"], prm["R"],
                                 prm["T_star_n"], prm["tau_n"], _lib.darr(prm["tol"]), 0, prm["c"], prm["c_lr"],
                                 at[5]), "enl_rhs")
    torch.cuda.synchronize()
    return K.cpu().numpy(), flags.cpu().numpy()


@pytest.mark.parametrize("c_lr", [0.0, -3.9e-3])
@pytest.mark.parametrize("variant", ["hybrid_high_llf", "hybrid_low", "weno_high", "drp"])
def test_cut_patches_give_the_same_bits(L, state, variant, c_lr):  # noqa: F811
    prm, v = default_params(c_lr=c_lr), VARIANTS.index(variant)
    K, flags = rhs(L, prm, v, state, NX, NY)  # 8 rows
    assert np.all(np.isfinite(K)) and (variant != "hybrid_high_llf" or 0 < flags.sum() < flags.size)
    for width, height in ((NX, 128), (NX, 32), (333, 77), (64, 16)):  # 4, 2, 4 and 2, 1 rows
        cut, fcut = rhs(L, prm, v, state, width, height)
        assert np.array_equal(flags, fcut)
        for k in range(5):
            bad = K[k].view(np.int64) != cut[k].view(np.int64)
            assert not bad.any(), (width, height, k, int(bad.sum()))
