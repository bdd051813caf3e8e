"""Densities that leave no state (zero, infinite, NaN, too small for the
entropy per mass): pressure and temperature follow the reference's formulas,
p = c^2 (d + (gamma - 1) / (2 rho0) d^2 + rho / c_p (rho s / rho)) + p0, and are
non-finite where those are."""
import numpy as np
import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300.constants import default_params  # noqa: E402
from test_gpu_patch import G  # noqa: E402
from test_gpu_state_and_tags import L, update_state  # noqa: E402,F401


@pytest.mark.parametrize("ws", [0.0, 3.0, -3.0, np.inf, np.nan])
@pytest.mark.parametrize("rho", [0.0, -0.0, np.inf, -np.inf, np.nan, 1e-310, 1e-320, -0.7, 1.2])
def test_pressure_of_a_broken_state(L, rho, ws):  # noqa: F811
    prm = default_params()
    w = np.ones((5, 1 + 2 * G, 1 + 2 * G)) * prm["rho0"]
    w[0, G, G], w[3, G, G] = rho, ws
    p, t = update_state(L, w, prm)
    with np.errstate(all="ignore"):
        r, s, d = np.float64(rho), np.float64(ws) / np.float64(rho), np.float64(rho) - prm["rho0"]
        want = prm["c"] ** 2 * (d + (prm["gamma1"] - 1) / (2 * prm["rho0"]) * d * d + r / prm["c_p"] * s) + prm["p0"]
        T = prm["T0"] * np.exp((s - prm["R"] * np.log(prm["rho0"] / r)) / prm["c_v"])
    for got, ref in ((p[0, 0], want), (t[0, 0], T)):
        assert np.isnan(got) == np.isnan(ref) and np.isinf(got) == np.isinf(ref), (rho, ws, got, ref)
        if np.isfinite(ref):  # (few roundings of terms of the ambient size; T: an argument below 2000)
            assert got == pytest.approx(ref, rel=1e-12, abs=1e-300)
