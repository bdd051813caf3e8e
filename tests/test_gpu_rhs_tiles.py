"""The tiled right-hand side at the sizes and magnitudes where it can go wrong.

* Patches one short of, at and one past the tile sides, in each of the tile
  heights (1, 2, 4 and 8 rows, chosen by the patch's size), against the oracle
  with the parity contract's 1e-12 relative L2 per field and equal flags.
* The triple-single flux differences against extended precision, for a scalar
  of any magnitude.  Bound: a split flux is formed with at most 4 units of
  rounding (u = rho u / rho within 2, the product, the difference), a
  reconstruction adds at most 20/6 times its largest input, a cell has 8 of
  them, and the weights at most double the effect of an input's error:
  4 x 20/6 x 8 x 2 < 256 units of 2^-53 of the largest split flux the cell's
  stencils hold, over dx.
"""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300 import _lib  # noqa: E402
from enlightning_gb300.constants import VARIANTS, default_params  # noqa: E402
from test_gpu_patch import G, TOL, eos, gpu_rhs, random_patch, relL2  # noqa: E402


@pytest.fixture(scope="module")
def L():
    lib = _lib.lib()
    lib.enl_set_stream(C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return lib


# 1 row: (1, 1) to (65, 9); 2 rows: (129, 63); 4 rows: (330, 117); 8 rows: (1030, 297)
@pytest.mark.parametrize("nx,ny", [(1, 1), (31, 7), (32, 8), (33, 9), (65, 9), (129, 63), (330, 117), (1030, 297)])
@pytest.mark.parametrize("variant", ["hybrid_high_llf", "hybrid_low"])
def test_tile_edges_match_oracle(L, ora, nx, ny, variant):
    prm = default_params()
    v = VARIANTS.index(variant)
    w = random_patch(nx, nx, ny, prm)
    box, xlo, dx = (3, 2 + nx, -4, ny - 5), (0.5, 1.0), (0.1, 0.125)
    pres, temp = eos(ora, w, box, xlo, dx, prm)
    H0 = np.ascontiguousarray(np.random.default_rng(ny).uniform(0, 1e3, (ny, nx)))
    for level in (0, 1):
        KK, flags = gpu_rhs(L, v, box, xlo, dx, w, pres, temp, H0, prm, level)
        ref, rflags = ora.rhs(v, box, (G, G), xlo, dx, w, H0, pres, temp, prm, level, flags=True)
        assert np.array_equal(flags, rflags)
        for k in range(5):
            assert relL2(KK[k], ref[k]) <= TOL, (level, k, relL2(KK[k], ref[k]))


def _weno_ld(order, plus, f):
    """wenop / wenom in extended precision, f: arrays at offsets -2..2."""
    ld = lambda x: np.longdouble(np.float64(np.float32(x)))  # noqa: E731
    if order == 5:
        a, b, c, d, e = f
        k, ep = ld(13.0 / 12.0), ld(10.0e-6)
        q = (k * (c - 2 * d + e) ** 2 + (3 * c - 4 * d + e) ** 2 / 4 + ep, k * (b - 2 * c + d) ** 2 + (b - d) ** 2 / 4 + ep,
             k * (a - 2 * b + c) ** 2 + (a - 4 * b + 3 * c) ** 2 / 4 + ep)
        z = [x / y / y for x, y in zip((ld(.3), ld(.6), ld(.1)) if plus else (ld(.1), ld(.6), ld(.3)), q)]
        g = ((2 * c + 5 * d - e, -b + 5 * c + 2 * d, 2 * a - 7 * b + 11 * c) if plus else
             (11 * c - 7 * d + 2 * e, 2 * b + 5 * c - d, -a + 5 * b + 2 * c))
        return ld(1.0 / 6.0) * (z[0] * g[0] + z[1] * g[1] + z[2] * g[2]) / (z[0] + z[1] + z[2])
    _, b, c, d, _ = f
    ep = ld(10.0e-6)
    z0 = (ld(2 / 3) if plus else ld(1 / 3)) / ((d - c) ** 2 + ep) ** 2
    z1 = (ld(1 / 3) if plus else ld(2 / 3)) / ((c - b) ** 2 + ep) ** 2
    g0, g1 = (c + d, 3 * c - b) if plus else (3 * c - d, b + c)
    return (z0 * g0 + z1 * g1) / (z0 + z1) / 2


@pytest.mark.parametrize("scale", [1e-200, 1e-20, 1.0, 1e20, 1e100])
@pytest.mark.parametrize("shape", ["noise", "jump", "smooth", "spike"])
@pytest.mark.parametrize("variant", ["weno_high", "weno_low"])
def test_flux_differences_against_extended_precision(L, variant, shape, scale):
    """Advection of rho s (no viscosity, conduction or relaxation): its
    right-hand side is the two flux differences alone."""
    prm = default_params(kappa=0.0, mu=0.0, muB=0.0)
    prm["tau_n"] = 1e300
    nx, ny, dx = 40, 21, 0.125
    rng = np.random.default_rng(3)
    NX, NY = nx + 2 * G, ny + 2 * G
    X, Y = np.meshgrid(np.arange(NX, dtype=float), np.arange(NY, dtype=float))
    s = {"noise": rng.standard_normal((NY, NX)), "jump": np.where(X + 0.3 * Y < 23, 1.0, 1e-7) * (1 + 1e-3 * rng.random((NY, NX))),
         "smooth": np.sin(0.21 * X) * np.cos(0.17 * Y), "spike": np.where((X == 20) & (Y == 12), 1.0, 0.0)}[shape] * scale
    rho = np.full((NY, NX), prm["rho0"])
    u, v = 37.5, -12.25
    w = np.stack([rho, rho * u, rho * v, s, rho * prm["T0"]])
    pres, temp = np.full((NY, NX), prm["p0"]), np.full((NY, NX), prm["T0"])
    KK, _ = gpu_rhs(L, VARIANTS.index(variant), (0, nx - 1, 0, ny - 1), (0.0, 0.0), (dx, dx), w, pres, temp,
                    np.zeros((ny, nx)), prm, 0)
    sl, al = s.astype(np.longdouble), np.longdouble(prm["weno_alpha"])
    order = 5 if "high" in variant else 3
    ref, size = np.zeros((ny, nx), np.longdouble), np.zeros((ny, nx))
    for ax, vel in ((1, u), (0, v)):
        at = lambda q: sl[G:G + ny, G + q:G + q + nx] if ax == 1 else sl[G + q:G + q + ny, G:G + nx]  # noqa: E731,B023
        fp = {q: (vel + al) * at(q) / 2 for q in range(-3, 4)}
        fm = {q: (vel - al) * at(q) / 2 for q in range(-3, 4)}
        st = lambda f, o: [f.get(q + o) for q in range(-2, 3)]  # noqa: E731
        ref += (_weno_ld(order, True, st(fp, -1)) + _weno_ld(order, False, st(fm, 0)) - _weno_ld(order, True, st(fp, 0))
                - _weno_ld(order, False, st(fm, 1))) / np.longdouble(dx)
        size = np.maximum(size, np.max([np.abs(at(q)).astype(float) for q in range(-3, 4)], 0) * (abs(vel) + float(al)) / 2)
    bound = 256 * 2.0 ** -53 * size / dx
    err = np.abs((KK[3].astype(np.longdouble) - ref).astype(float))
    assert np.all(err <= bound + 1e-320), np.max(err / (bound + 1e-320))
