"""What a strategy asks of its parameters and patches (no GPU): the envelope's
width only where a side absorbs, and of every vector the entries it uses,
whatever kind of number they are."""
import numpy as np
import pytest

pytest.importorskip("torch")

from enlightning_gb300.constants import ABSORB, REFLECT, default_params  # noqa: E402
from enlightning_gb300.strategy import Enlightning, Patch  # noqa: E402


def make(bc, **over):
    s = object.__new__(Enlightning)
    s.p = default_params(**over)
    s.domain_xlo, s.domain_xhi, s.bc = (0.0, 0.0), (1.0, 1.0), tuple(bc)
    return s, Patch((0, 7, 0, 4), (0.0, 0.25), (0.125, 0.125)).allocate(device="cpu")


def test_width_is_read_where_a_side_absorbs():
    s, Q = make((REFLECT,) * 4)
    del s.p["bc_absorb_width"]
    s._patch_args(Q, absorb=True, ghosts=True)
    s.bc = (REFLECT, ABSORB, REFLECT, REFLECT)
    with pytest.raises(KeyError):
        s._patch_args(Q, absorb=True, ghosts=True)
    s._patch_args(Q, absorb=False, ghosts=True)  # (an envelope of the caller's own)


def test_vectors_may_be_longer_and_of_any_number_type():
    s, Q = make((REFLECT, ABSORB) * 2 + (REFLECT,), tol=np.array([1.5, 1e-2, 5e-3, 7.0], np.float32),
                rho0=np.float32(1.25), c=343)
    s.domain_xlo, s.domain_xhi = (0, 0, 0), np.array([4, 5, 6])
    Q.box, Q.xlo, Q.dx, Q.touches = np.array([0, 7, 0, 4, 9]), (0, 0.25, 1.0), [0.125, 0.125, 0.125], (1, 0, 1, 0, 1)
    Q.level = 1.0
    a = s._patch_args(Q, absorb=True, ghosts=False)
    assert list(a.box) == [0, 7, 0, 4] and list(a.xlo) == [0.0, 0.25] and list(a.dx) == [0.125, 0.125]
    assert list(a.tol) == [float(np.float32(x)) for x in (1.5, 1e-2, 5e-3)]
    assert list(a.touches) == [1, 0, 1, 0] and list(a.bc) == [REFLECT, ABSORB, REFLECT, ABSORB]
    assert list(a.grid_xhi) == [4.0, 5.0] and a.level == 1 and a.rho0 == 1.25 and a.c == 343.0
    assert a.source_g is None
