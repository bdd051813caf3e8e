"""update_state and tag_cells over the ranges where their cheaper arithmetic
can go wrong.

* Temperature and pressure against extended precision for densities from a
  thousandth to a thousand times ambient, on both sides of every table step
  near ambient, and entropies that move the exponent far.  Bound on T in units
  of 2^-53: 3 for the exponential and the product with T0; of the argument's
  entropy part 3 (quotient, sum, quotient) and of its logarithm part 5 (2 for
  the logarithm, product, sum, quotient), and the logarithm's absolute error,
  max(1, |log2|) units times R / c_v.  On p: 5 roundings of terms no larger
  than the sum of their magnitudes.
* Densities without a logarithm (zero, negative, NaN) give what the general
  formula gives.
* Tags bit for bit as the oracle's division decides them, for tolerances and
  differences from 1e-200 to 1e60 and for ratios within 1e-14 and within 1e-6
  of the threshold on both sides.
"""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300 import _lib  # noqa: E402
from enlightning_gb300.constants import default_params  # noqa: E402
from test_gpu_patch import G, P, dev  # noqa: E402


@pytest.fixture(scope="module")
def L():
    lib = _lib.lib()
    lib.enl_set_stream(C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return lib


def update_state(L, w, prm, dx=0.1, ylo=0.0):
    ny, nx = w.shape[1] - 2 * G, w.shape[2] - 2 * G
    d, p, t = dev(w), dev(np.zeros(w.shape[1:])), dev(np.zeros(w.shape[1:]))
    I, D = _lib.iref, _lib.dref
    L.update_state_(_lib.darr((dx, dx)), _lib.darr((0.0, ylo)), I(0), I(nx - 1), I(0), I(ny - 1), I(G), I(G), P(d), P(p),
                    P(t), D(prm["rho0"]), D(prm["c"]), D(prm["gamma1"]), D(prm["c_p"]), D(prm["p0"]), D(prm["T0"]),
                    D(prm["c_lr"]), D(prm["c_v"]), D(prm["R_tilde"]), D(prm["M"]), D(prm["R"]), I(5))
    _lib.check_sticky("update_state")
    torch.cuda.synchronize()
    return p.cpu().numpy()[G:-G, G:-G], t.cpu().numpy()[G:-G, G:-G]


@pytest.mark.parametrize("c_lr", [0.0, -3.9e-3])
@pytest.mark.parametrize("kind", ["near", "far", "hot"])
def test_state_against_extended_precision(L, kind, c_lr):
    prm = default_params(c_lr=c_lr)
    nx, ny = 257, 33
    rng = np.random.default_rng(5)
    w = np.ones((5, ny + 2 * G, nx + 2 * G))
    n = w[0].size
    step = {"near": 1.0 + np.linspace(-0.02, 0.02, n) + rng.choice([0, 2.0 ** -52, -2.0 ** -53], n),
            "far": np.exp(rng.uniform(-6.9, 6.9, n)), "hot": 1.0 + 0.5 * rng.random(n)}[kind]
    w[0] = prm["rho0"] * step.reshape(w[0].shape)
    w[3] = w[0] * {"near": 1.0, "far": 100.0, "hot": 1e5}[kind] * rng.standard_normal(w[0].shape)
    p, t = update_state(L, w, prm)
    ld = np.longdouble
    rho, rs = w[0, G:-G, G:-G].astype(ld), w[3, G:-G, G:-G].astype(ld)
    q = {k: ld(prm[k]) for k in ("rho0", "c", "gamma1", "c_p", "p0", "T0", "c_lr", "c_v", "R")}
    lg = np.log(rho / q["rho0"])
    a = (rs / rho + q["R"] * lg) / q["c_v"]
    T = q["T0"] * np.exp(a)
    units = 3 + 3 * np.abs(rs / rho / q["c_v"]) + 5 * np.abs(q["R"] / q["c_v"] * lg) + q["R"] / q["c_v"] * np.maximum(1, np.abs(lg) / np.log(ld(2)))
    assert np.all(np.abs(t - T) <= units * ld(2.0) ** -53 * T)
    h = ld(0.1) * (np.arange(ny, dtype=ld)[:, None] + ld(0.5))
    cc = q["c"] + q["c_lr"] * h
    d = rho - q["rho0"]
    terms = (d, (q["gamma1"] - 1) / (2 * q["rho0"]) * d * d, rs / q["c_p"])
    pr = cc * cc * sum(terms) + q["p0"]
    bound = 8 * ld(2.0) ** -53 * (cc * cc * sum(np.abs(x) for x in terms) + q["p0"])
    assert np.all(np.abs(p - pr) <= bound)


def test_state_without_a_logarithm(L):
    prm = default_params()
    w = np.ones((5, 1 + 2 * G, 6 + 2 * G)) * prm["rho0"]
    w[3] = 0.0
    w[0, G, G:-G] = [0.0, -1.0, np.nan, np.inf, 5e-324, prm["rho0"]]
    _, t = update_state(L, w, prm)
    # log(rho0 / rho) of 0, negative and NaN densities; an infinite one cools to nothing or is hot without bound
    assert np.isnan(t[0, 0]) and np.isnan(t[0, 1]) and np.isnan(t[0, 2])
    assert t[0, 5] == prm["T0"]
    assert np.isfinite(t[0, 4]) or np.isnan(t[0, 4])


def _tags(L, ora, rho, src, tol, val=1):
    ny, nx = rho.shape[0] - 2 * G, rho.shape[1] - 2 * G
    w = np.stack([rho] + [np.zeros_like(rho)] * 4)
    dw, ds = dev(w), dev(src)
    tags = torch.full((ny, nx), -1, dtype=torch.int32, device="cuda")
    I = _lib.iref
    L.tag_cells_(I(0), I(nx - 1), I(0), I(ny - 1), I(G), I(G), P(tags), P(dw), P(ds), I(val), _lib.darr(tol), I(5))
    _lib.check_sticky("tag_cells")
    torch.cuda.synchronize()
    ref = ora.tag_cells((0, nx - 1, 0, ny - 1), (G, G), w, src, tol)
    return tags.cpu().numpy(), ref


@pytest.mark.parametrize("tol", [1e-2, 1e-12, 1e-200, 0.0])
@pytest.mark.parametrize("amp", [1e-200, 1e-30, 1e-9, 1.0, 1e20, 1e60])
def test_tags_of_any_magnitude_bit_exact(L, ora, tol, amp):
    rng = np.random.default_rng(2)
    rho = amp * rng.standard_normal((41, 70))
    src = amp * np.where(rng.random((41, 70)) < 0.7, 0.0, rng.standard_normal((41, 70)))
    got, ref = _tags(L, ora, rho, src, (tol, tol, 5e-3))
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("gap", [1e-16, 1e-14, 1e-7, 3e-6, 1e-5])
def test_tags_near_the_threshold_bit_exact(L, ora, gap):
    """Sawtooth densities with differences t, k t around the k at which the
    ratio passes the threshold."""
    f32 = lambda x: float(np.float32(x))  # noqa: E731
    tol = 1e-2
    ep = (f32(0.9) * tol) / (1.0 - f32(0.9) * (tol * tol))
    lo, hi = 0.5, 1.0
    for _ in range(200):
        k = 0.5 * (lo + hi)
        low = (2.0 * (0.5 * (k * 0.5)) + ep) / ((0.25 + (k * 0.5) ** 2) + ep) < f32(0.9999)
        lo, hi = (k, hi) if low else (lo, k)
    nx, ny = 120, 30
    rho = np.empty((ny + 2 * G, nx + 2 * G))
    for j in range(rho.shape[0]):
        kj = k * (1 + (j - rho.shape[0] // 2) * gap)
        d = np.where(np.arange(rho.shape[1]) % 2 == 0, 0.5, 0.5 * kj)
        rho[j] = np.cumsum(d) - d.sum() / 2
    got, ref = _tags(L, ora, rho, np.zeros_like(rho), (tol, tol, 5e-3))
    assert np.array_equal(got, ref)
    assert 0 < ref.sum() < ref.size
