"""Fifth-order flux differences where a stencil holds values of very different
size, so that its differences fall on and between the words of their common
grid (2^-19, 2^-40 and the rest), against extended precision with the bound of
the tiled right-hand side's test: 256 units of 2^-53 of the stencils' largest
split flux, over dx."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300 import _lib  # noqa: E402
from enlightning_gb300.constants import VARIANTS, default_params  # noqa: E402
from test_gpu_patch import G, gpu_rhs  # noqa: E402
from test_gpu_rhs_tiles import _weno_ld  # noqa: E402


@pytest.mark.parametrize("bits", [8, 18, 19, 20, 24, 33, 39, 41, 50, 60])
@pytest.mark.parametrize("shape", ["one side", "spots"])
def test_small_values_beside_large_ones(bits, shape):
    L = _lib.lib()
    L.enl_set_stream(C.c_void_p(torch.cuda.current_stream().cuda_stream))
    prm = default_params(kappa=0.0, mu=0.0, muB=0.0)
    prm["tau_n"] = 1e300
    nx, ny, dx, u, v = 48, 24, 0.125, 37.5, -12.25
    rng = np.random.default_rng(bits)
    NX, NY = nx + 2 * G, ny + 2 * G
    X, Y = np.meshgrid(np.arange(NX), np.arange(NY))
    large = X + Y < 35 if shape == "one side" else rng.random((NY, NX)) < 0.1
    s = rng.standard_normal((NY, NX)) * np.where(large, 1.0, 2.0 ** -bits)
    rho = np.full((NY, NX), prm["rho0"])
    w = np.stack([rho, rho * u, rho * v, s, rho * prm["T0"]])
    KK, _ = gpu_rhs(L, VARIANTS.index("weno_high"), (0, nx - 1, 0, ny - 1), (0.0, 0.0), (dx, dx), w,
                    np.full((NY, NX), prm["p0"]), np.full((NY, NX), prm["T0"]), np.zeros((ny, nx)), prm, 0)
    sl, al = s.astype(np.longdouble), np.longdouble(prm["weno_alpha"])
    ref, size = np.zeros((ny, nx), np.longdouble), np.zeros((ny, nx))
    for ax, vel in ((1, u), (0, v)):
        at = {q: sl[G:G + ny, G + q:G + q + nx] if ax == 1 else sl[G + q:G + q + ny, G:G + nx] for q in range(-3, 4)}
        fp, fm = ({q: (vel + sg * al) * at[q] / 2 for q in at} for sg in (1, -1))
        st = lambda f, o: [f.get(q + o) for q in range(-2, 3)]  # noqa: E731
        ref += (_weno_ld(5, True, st(fp, -1)) + _weno_ld(5, False, st(fm, 0)) - _weno_ld(5, True, st(fp, 0))
                - _weno_ld(5, False, st(fm, 1))) / np.longdouble(dx)
        size = np.maximum(size, np.max([np.abs(a).astype(float) for a in at.values()], 0) * (abs(vel) + float(al)) / 2)
    bound = 256 * 2.0 ** -53 * size / dx
    err = np.abs((KK[3].astype(np.longdouble) - ref).astype(float))
    assert np.all(err <= bound), np.max(err / bound)
