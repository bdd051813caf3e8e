"""enl_patch_stage against the separate entry points it stands for, bit for
bit (it does the same operations on the same values): patches of one cell to
just past its 32 x 8 blocks, sides that reflect, absorb or touch no boundary,
coarse and fine levels, an envelope that covers the patch, and a patch partly
outside the domain; and a strategy whose own methods replace the ghost fill or
the envelope."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300 import _lib  # noqa: E402
from enlightning_gb300.constants import ABSORB, REFLECT, default_params  # noqa: E402
from enlightning_gb300.strategy import Enlightning, Patch  # noqa: E402
from test_gpu_patch import P as ptr, random_patch  # noqa: E402

FIELDS = ("w_scr", "pres", "temp", "src_g", "w_cur", "K")


def make(nx, ny, xlo, bc, touches, level, width, variant, cls=Enlightning):
    prm = default_params(bc_absorb_width=width)
    s = cls(prm, variant, (0.0, 0.0), (8.4, 4.9), bc)
    box = (4, 3 + nx, -2, ny - 3)
    Q = Patch(box, xlo, (0.1, 0.1), level, touches).allocate()
    w = random_patch(nx + ny, nx, ny, prm)
    s.initialize_ambient(Q)
    Q.w_scr.copy_(torch.from_numpy(w))
    Q.w_cur.copy_(Q.interior(Q.w_scr))
    Q.src.copy_(torch.from_numpy(np.random.default_rng(1).standard_normal((ny, nx))))
    Q.src_g.copy_(torch.from_numpy(np.random.default_rng(2).standard_normal(tuple(Q.src_g.shape))))
    return s, Q


def separate(s, Q, dt, a1, a2, beta, ghosts):
    L, p, b, I, D = s.L, s.p, Q.box, _lib.iref, _lib.dref
    if ghosts:
        Enlightning.set_physical_boundary_conditions(s, Q)
    e = [I(v) for v in (*b, 3, 3)]
    L.rhs_(*e, _lib.darr(Q.xlo), _lib.darr(Q.dx), ptr(Q.w_scr), ptr(Q.src), ptr(Q.K), ptr(Q.pres), ptr(Q.temp),
           *[D(p[k]) for k in ("weno_alpha", "kappa", "mu", "muB", "R", "T_star_n", "T_star_o", "tau_n", "tau_o")],
           _lib.darr(p["tol"]), I(Q.level), D(p["c"]), D(p["c_lr"]), I(5))
    L.runge_kutta_(*e, D(dt), D(a1), D(a2), D(beta), ptr(Q.w_scr), ptr(Q.w_cur), ptr(Q.K), I(5))
    L.update_state_(_lib.darr(Q.dx), _lib.darr(Q.xlo), *e, ptr(Q.w_scr), ptr(Q.pres), ptr(Q.temp),
                    *[D(p[k]) for k in ("rho0", "c", "gamma1", "c_p", "p0", "T0", "c_lr", "c_v", "R_tilde", "M", "R")],
                    I(5))
    Enlightning.set_absorbing_boundary_conditions(s, Q)
    _lib.check_sticky()


def same(A, B):
    torch.cuda.synchronize()
    for f in FIELDS:
        x, y = getattr(A, f).cpu().numpy(), getattr(B, f).cpu().numpy()
        assert np.array_equal(x.view(np.int64), y.view(np.int64)), f


@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 9), (33, 8), (70, 41)])
@pytest.mark.parametrize("bc,touches", [((REFLECT,) * 4, (1, 1, 1, 1)), ((ABSORB, ABSORB, REFLECT, ABSORB), (1, 1, 1, 1)),
                                        ((ABSORB,) * 4, (0, 1, 0, 0))])
@pytest.mark.parametrize("xlo,width,level,variant", [
    ((0.0, 0.0), 0.6, 0, "hybrid_high_llf"), ((0.0, 0.0), 30.0, 2, "hybrid_high"), ((1.3, 0.7), 0.05, 1, "hybrid_low_llf"),
    ((-0.45, -1.05), 0.6, 0, "hybrid_high_llf")])
def test_stage_equals_separate_calls(nx, ny, bc, touches, xlo, width, level, variant):
    args = (nx, ny, xlo, bc, touches, level, width, variant)
    s, A = make(*args)
    _, B = make(*args)
    for stage in range(3):
        a1, a2, b = (s.rk[k][stage] for k in range(3))
        separate(s, A, 1e-5, a1, a2, b, True)
        Q = s._patch_args(B, absorb=True, ghosts=True)
        _lib.check(s.L.enl_patch_stage(C.byref(Q), 1e-5, a1, a2, b, 1))
        same(A, B)
    separate(s, A, 1e-5, 0.25, 0.75, 0.25, False)
    s.single_step(B, 1e-5, 0.25, 0.75, 0.25)
    same(A, B)


def test_replaced_methods_are_called():
    calls = []

    class Own(Enlightning):
        def set_physical_boundary_conditions(self, Q, fill=None):
            calls.append("bc")
            super().set_physical_boundary_conditions(Q, fill)

        def set_absorbing_boundary_conditions(self, Q):
            calls.append("absorb")

    args = (40, 24, (0.0, 0.0), (ABSORB,) * 4, (1, 1, 1, 1), 0, 0.6, "hybrid_high_llf")
    s, A = make(*args, cls=Own)
    s.advance(A, 1e-5, 2)
    assert calls == ["bc", "absorb"] * 6
    # no envelope: the same as sides that touch the domain with no absorbing bc
    # in the update, and not the same as the class's own
    t, B = make(*args)
    t.advance(B, 1e-5, 2)
    torch.cuda.synchronize()
    assert not torch.equal(A.w_cur, B.w_cur)


def test_arguments_are_checked():
    s, A = make(8, 8, (0.0, 0.0), (REFLECT,) * 4, (1, 1, 1, 1), 0, 0.6, "hybrid_high_llf")
    L = s.L
    assert L.enl_patch_stage(None, 1e-5, 1.0, 0.0, 1.0, 1) != 0
    for field, value in (("w_n", None), ("rhs", None), ("pressure", None), ("gcw", (C.c_int * 2)(2, 3))):
        Q = s._patch_args(A, absorb=True, ghosts=True)
        setattr(Q, field, value)
        assert L.enl_patch_stage(C.byref(Q), 1e-5, 1.0, 0.0, 1.0, 0) != 0, field
    L.enl_get_last_error()
