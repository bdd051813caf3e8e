"""Ghost fill and absorbing envelope of one patch at the shapes where their
one-launch kernels can go wrong, against the oracle: patches of one cell to
just past a block, any set of sides (fill bit-exact); envelopes that reach far
into the patch, stop inside it, or belong to a patch that lies partly outside
the domain, where the factors do not grow along the walk (the parity
contract's 1e-12 on the fields and on the deviations from the ambient state)."""
import ctypes as C
import itertools

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300 import _lib  # noqa: E402
from enlightning_gb300.constants import ABSORB, REFLECT, default_params  # noqa: E402
from test_gpu_patch import G, TOL, P, dev, eos, random_patch, relL2  # noqa: E402


@pytest.fixture(scope="module")
def L():
    lib = _lib.lib()
    lib.enl_set_stream(C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return lib


@pytest.mark.parametrize("nx,ny", [(1, 1), (1, 40), (43, 2), (129, 33)])
@pytest.mark.parametrize("bc", [(REFLECT,) * 4, (REFLECT, ABSORB, ABSORB, REFLECT)])
def test_ghost_fill_of_any_sides_bit_exact(L, ora, nx, ny, bc):
    rng = np.random.default_rng(nx + ny)
    box = (0, nx - 1, 0, ny - 1)
    base = rng.standard_normal((8, ny + 2 * G, nx + 2 * G))
    for touches in itertools.product((0, 1), repeat=4):
        f = base.copy()
        d = dev(f)
        st = L.enl_phys_bc(*box, G, G, _lib.iarr(touches), _lib.iarr(bc), G, G, P(d), P(d[5]), P(d[6]), P(d[7]))
        _lib.check(st)
        torch.cuda.synchronize()
        w, pr, te, so = (np.ascontiguousarray(f[s]) for s in (slice(0, 5), 5, 6, 7))
        ora.phys_bc(box, (G, G), touches, bc, w, pr, te, so)
        assert np.array_equal(d.cpu().numpy(), np.concatenate([w, pr[None], te[None], so[None]])), touches


@pytest.mark.parametrize("nx,ny", [(33, 9), (70, 41)])
@pytest.mark.parametrize("width", [0.05, 0.6, 30.0])
@pytest.mark.parametrize("xlo", [(0.0, 0.0), (1.3, 0.7), (-0.45, -1.05)])
def test_envelope_matches_oracle(L, ora, nx, ny, width, xlo):
    prm = default_params(bc_absorb_width=width)
    box, dx, hi = (0, nx - 1, 0, ny - 1), (0.1, 0.1), (8.4, 4.9)
    w = random_patch(nx, nx, ny, prm)
    pres, temp = eos(ora, w, box, xlo, dx, prm)
    bc = (ABSORB, ABSORB, ABSORB, ABSORB)
    dw, dpr, dte = dev(w), dev(pres), dev(temp)
    st = L.enl_absorb(*box, G, G, _lib.darr(xlo), _lib.darr(dx), _lib.darr((0.0, 0.0)), _lib.darr(hi), _lib.iarr(bc),
                      width, prm["p0"], prm["T0"], prm["rho0"], P(dw), P(dpr), P(dte))
    _lib.check(st)
    torch.cuda.synchronize()
    ora.absorb(box, (G, G), xlo, dx, (0.0, 0.0), hi, bc, width, prm, w, pres, temp)
    got = dw.cpu().numpy()
    for k in range(5):
        assert relL2(got[k], w[k]) <= TOL, k
    assert relL2(dpr.cpu().numpy() - prm["p0"], pres - prm["p0"]) <= TOL
    assert relL2(dte.cpu().numpy() - prm["T0"], temp - prm["T0"]) <= TOL
