"""The work that users of this framework have it do, as measurable cases.

A case is one pass through the framework's public entry points:

  patch    one RK3 step of one patch through the drop-in patch strategy
           (``strategy.Enlightning.advance``: ghost fill, rhs_, runge_kutta_,
           update_state_, absorbing envelope, three stages) and the patch's
           refinement tags, as a host hierarchy drives them
  rhs      one right-hand side with its switch flags (``enl_rhs``)
  pulses   independent pulse problems advanced together by the batched engine
  amr      a small two-level hierarchy with a host exchange every step, for
           callers that keep the state on the host side
  shock    the Mach 1.5 shock: upload, RK3 step(s), download
  line     the three-level line source: upload, RK3 step(s), download
  regrid   tagging, clustering and rebuilding of every finer level
  train    loss and gradient of the learned switch on one batch

Inputs come from the seed alone.  Single patches and pulses start some way
into a run: rings of acoustic waves that carry the velocity of an outgoing
wave, at random places and radii.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

G = 3
REFLECT, ABSORB = 10, 20
VARIANTS = ("hybrid_high_llf", "hybrid_high", "hybrid_low_llf", "hybrid_low", "weno_high_llf", "weno_high",
            "weno_low_llf", "weno_low", "drp")
# RK3 as the reference's input file writes its coefficients
RK = ((1.0, 0.0, 1.0), (0.75, 0.25, 0.25), (0.3333333333, 0.6666666667, 0.6666666667))
F64, F32_RHS, F32_STATE = 0, 1, 2


def listed():
    return [
        # the smallest patches a hierarchy makes (sides from 16): calls and launches count
        dict(name="patch_24x16", kind="patch", nx=24, ny=16, variant="hybrid_high_llf", level=0, c_lr=0.0,
             sides="LRBT", absorb="", rings=1),
        # a ragged fine-level patch at two absorbing sides of the domain, WENO in every cell
        dict(name="patch_131x93_fine", kind="patch", nx=131, ny=93, variant="hybrid_high_llf", level=1, c_lr=0.0,
             sides="LT", absorb="LRT", rings=2),
        # the single 512x512 pulse with reflecting walls through the drop-in path
        dict(name="patch_512", kind="patch", nx=512, ny=512, variant="hybrid_high_llf", level=0, c_lr=0.0,
             sides="LRBT", absorb="", rings=1),
        # the lower-order scheme with a lapse rate, one call with its switch flags
        dict(name="rhs_low_llf_300x217", kind="rhs", nx=300, ny=217, variant="hybrid_low_llf", level=0, c_lr=-3.9e-3,
             rings=3),
        # a small two-level run that exchanges its state with the host every step
        dict(name="amr_96x80", kind="amr", nx=96, ny=80, precision=F64, variant="hybrid_high_llf", steps=1),
        # the batch of 64 independent pulses (sides 128 to 1024), FP64, two steps
        dict(name="pulses_64", kind="pulses", n=64, lo=128, hi=1024, precision=F64, learned=False,
             variant="hybrid_high_llf", steps=2),
        # a smaller batch in single-precision perturbation storage
        dict(name="pulses_24_f32", kind="pulses", n=24, lo=128, hi=768, precision=F32_STATE, learned=False,
             variant="hybrid_high_llf", steps=4),
        # the Mach 1.5 shock on 1024x512, two levels, learned switch, FP64
        dict(name="shock_1024", kind="shock", nx=1024, ny=512, precision=F64, learned=True, steps=1),
        # the headline: the line source on 4096x2048, three levels, learned switch, FP64
        dict(name="line_4096", kind="line", nx=4096, ny=2048, precision=F64, learned=True, steps=1),
        # the same in single-precision storage, ten steps (one regrid interval) per exchange
        dict(name="line_4096_f32", kind="line", nx=4096, ny=2048, precision=F32_STATE, learned=True, steps=10),
        # the regrid that the line source does every ten steps
        dict(name="regrid_4096", kind="regrid", nx=4096, ny=2048, precision=F64),
        # one batch of the learned switch's training
        dict(name="train_65536", kind="train", rows=65536),
    ]


def _log_int(rng, lo, hi, mult=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    return max(lo, min(hi, int(v / mult) * mult))


def draw(rng):
    kind = rng.choice(["patch", "patch", "rhs", "pulses", "amr", "shock", "line", "regrid", "train"])
    if kind in ("patch", "rhs"):
        variant = rng.choice(["hybrid_high_llf"] * 4 + list(VARIANTS))
        case = dict(kind=kind, nx=_log_int(rng, 16, 700), ny=_log_int(rng, 16, 700), variant=variant,
                    level=rng.choice([0, 0, 1]), c_lr=rng.choice([0.0, 0.0, -3.9e-3]), rings=rng.randint(1, 4))
        if kind == "patch":
            case["sides"] = rng.choice(["LRBT", "LB", "RT", "B", ""])
            case["absorb"] = rng.choice(["", "LRT"])
        return case
    if kind == "pulses":
        prec = rng.choice([F64, F64, F32_STATE, F32_RHS])
        return dict(kind=kind, n=_log_int(rng, 1, 40), lo=128, hi=rng.choice([256, 512, 1024]), precision=prec,
                    learned=rng.random() < 0.3, variant=rng.choice(["hybrid_high_llf"] * 3 + ["weno_high_llf", "drp"]),
                    steps=rng.choice([1, 2]))
    if kind == "amr":
        return dict(kind=kind, nx=_log_int(rng, 48, 400, 4), ny=_log_int(rng, 48, 400, 4),
                    precision=rng.choice([F64, F64, F32_STATE]), variant="hybrid_high_llf", steps=rng.choice([1, 2]))
    if kind == "shock":
        s = rng.choice([2, 3, 4, 5, 6, 7, 8])
        return dict(kind=kind, nx=128 * s, ny=64 * s, precision=rng.choice([F64, F64, F32_STATE]),
                    learned=rng.random() < 0.5, steps=1)
    s = rng.choice([3, 4, 5, 6, 7, 8, 10, 12, 14, 15])
    if kind == "line":
        return dict(kind=kind, nx=256 * s, ny=128 * s, precision=rng.choice([F64, F64, F32_STATE]),
                    learned=rng.random() < 0.5, steps=rng.choice([1, 2]))
    if kind == "regrid":
        return dict(kind=kind, nx=256 * s, ny=128 * s, precision=rng.choice([F64, F32_STATE]))
    return dict(kind="train", rows=_log_int(rng, 1000, 200000))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _prm(**over):
    from enlightning_gb300.constants import default_params
    return default_params(**over)


def _const(case):
    """The physical constants of a case as plain numbers (the reference's input file)."""
    p = dict(weno_alpha=360.0, c=343.0, gamma1=1.4, p0=101325.0, RH=20.0, T0=293.16, c_lr=case.get("c_lr", 0.0),
             rho0=1.2, R=287.06, c_p=1010.0, T_star_n=3352.0, mu=1.846e-5, muB=1.1076e-5, kappa=0.02624, c_v=720.4,
             tol=(1.5, 1e-2, 5e-3), cfl=0.5, absorb_width=1.0)
    # relaxation time of the nitrogen mode at p_ref = p0, T_ref = T0
    T0 = p["T0"]
    zeta = (10.79586 * (1 - (273.16 / T0)) - 5.02808 * math.log10(T0 / 273.16)
            + 1.50474e-4 * (1 - math.pow(10, (-8.29692 * ((T0 / 273.16) - 1))))
            - 4.2873e-4 * (1 - math.pow(10, (-4.76955 * ((273.16 / T0) - 1)))) - 2.2195983)
    h = p["RH"] * (p["p0"] * math.pow(10, zeta)) / p["p0"]
    p["tau_n"] = 1 / (2 * math.pi * (9 + 280 * h))
    return p


def _eos(w, p, height):
    """Pressure and temperature of a state (update_state)."""
    rho, rs = w[0], w[3]
    d = rho - p["rho0"]
    c = p["c"] + p["c_lr"] * height
    pres = c * c * (d + (p["gamma1"] - 1) / (2 * p["rho0"]) * d * d + rho / p["c_p"] * (rs / rho)) + p["p0"]
    return pres, p["T0"] * torch.exp((rs / rho - p["R"] * torch.log(p["rho0"] / rho)) / p["c_v"])


def _waves(nx, ny, p, rng, rings, i0=0, j0=0, sigma=(4.0, 16.0), amp=(0.01, 0.5)):
    """State (5, ny, nx) of `rings` outgoing ring waves around random centres
    of the patch, at radii up to half its shorter side."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    X = torch.arange(i0, i0 + nx, dtype=torch.float64, device=dev)[None, :]
    Y = torch.arange(j0, j0 + ny, dtype=torch.float64, device=dev)[:, None]
    side = min(nx + 2 * i0, ny + 2 * j0)
    dp = torch.zeros((ny, nx), dtype=torch.float64, device=dev)
    mx, my = torch.zeros_like(dp), torch.zeros_like(dp)
    for _ in range(rings):
        cx, cy = rng.uniform(0.3, 0.7) * nx, rng.uniform(0.3, 0.7) * ny
        s = rng.uniform(*sigma)
        r0 = rng.uniform(0.0, 0.5) * side
        a = rng.uniform(*amp) * p["p0"] / (1.0 + r0 / (4.0 * s))  # weaker as it spreads
        dx, dy = X - cx, Y - cy
        r = torch.sqrt(dx * dx + dy * dy)
        d = a * torch.exp(-((r - r0) ** 2) / (2 * s * s))
        d = torch.where(d > 1e-14 * p["p0"], d, torch.zeros_like(d))
        dp += d
        f = d / p["c"] / (r + 1.0)  # momentum of an outgoing wave, d / c along the radius
        mx += f * dx
        my += f * dy
    k = (p["gamma1"] - 1) / (2 * p["rho0"])
    rho = p["rho0"] + (torch.sqrt(1 + 4 * k * dp / p["c"] ** 2) - 1) / (2 * k)
    T = p["T0"] * torch.exp(-p["R"] * torch.log(p["rho0"] / rho) / p["c_v"])
    return torch.stack([rho, mx, my, torch.zeros_like(rho), rho * T])


def _patch_inputs(case, seed):
    """Ghosted state, pressure, temperature and source of one patch; on sides
    that are not the domain's the ghosts hold the neighbours' cells."""
    p, rng = _const(case), np.random.default_rng([seed, 1])
    nx, ny = case["nx"], case["ny"]
    small = min(nx, ny)
    sig = (min(4.0, small / 6.0), min(16.0, small / 3.0))
    w = _waves(nx + 2 * G, ny + 2 * G, p, rng, case["rings"], -G, -G, sigma=sig)
    dx = 0.1 / 2 ** case["level"]
    if case["kind"] == "rhs":  # entropy and relaxation away from equilibrium, a source
        gen = torch.Generator(device=w.device)
        gen.manual_seed(seed)
        w[3] += w[0] * 10.0 * torch.randn(w[0].shape, generator=gen, dtype=torch.float64, device=w.device)
        w[4] *= 1.0 + 0.002 * torch.randn(w[0].shape, generator=gen, dtype=torch.float64, device=w.device)
        H = 1e3 * torch.rand((ny, nx), generator=gen, dtype=torch.float64, device=w.device)
    else:
        H = torch.zeros((ny, nx), dtype=torch.float64, device=w.device)
    height = (torch.arange(-G, ny + G, dtype=torch.float64, device=w.device)[:, None] + 0.5) * dx
    pres, temp = _eos(w, p, height)
    return p, dx, w.contiguous(), pres.contiguous(), temp.contiguous(), H


def _bc(case):
    return tuple(ABSORB if s in case["absorb"] else REFLECT for s in "LRBT")


def _touches(case):
    return tuple(int(s in case["sides"]) for s in "LRBT")


_stream = None


def _side_stream():
    """Graph capture needs a stream that is not the default one."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def _mlp(E):
    from enlightning_gb300 import sensor
    E.set_mlp(*sensor.load_weights())


def _pulse_sizes(case):
    rng = np.random.default_rng([case["n"], case["lo"], case["hi"]])
    # sides are multiples of 32, as the batch of pulses is stated
    return [int(32 * rng.integers(case["lo"] // 32, case["hi"] // 32 + 1)) for _ in range(case["n"])]


def _pulse_state(case, seed, q, side, p):
    return _waves(side, side, p, np.random.default_rng([seed, 3, q]), 1)


def _pulse_dt(p, dx):
    return p["cfl"] * (dx / p["c"])


def _amr_boxes(case):
    """A base level of two patches and a fine level of two patches over its middle."""
    nx, ny = case["nx"], case["ny"]
    h, q = nx // 8 * 4, ny // 8 * 4
    base = [(0, h - 1, 0, ny - 1), (h, nx - 1, 0, ny - 1)]
    fine = [(h - 16, h + 15, q - 16, q + 15), (h + 16, h + 31, q - 8, q + 7)]
    return [base, fine]


def _amr_state(case, seed):
    p = _const(case)
    w = _waves(case["nx"], case["ny"], p, np.random.default_rng([seed, 4]), 2, sigma=(3.0, 8.0))
    return p, w


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("patch", "rhs"):
        return _prepare_patch(case, seed)
    if kind == "train":
        return _prepare_train(case, seed)
    S = _side_stream()
    S.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(S):
        st = {"pulses": _prepare_pulses, "amr": _prepare_amr, "shock": _prepare_shock, "line": _prepare_line,
              "regrid": _prepare_regrid}[kind](case, seed)
    st["kind"] = kind
    S.synchronize()
    return st


def run(st):
    return {"patch": _run_patch, "rhs": _run_rhs, "pulses": _run_pulses, "amr": _run_exchange, "shock": _run_exchange,
            "line": _run_exchange, "regrid": _run_regrid, "train": _run_train}[st["kind"]](st)


def _prepare_patch(case, seed):
    from enlightning_gb300.strategy import Enlightning, Patch
    p, dx, w, pres, temp, H = _patch_inputs(case, seed)
    nx, ny = case["nx"], case["ny"]
    prm = _prm(c_lr=case["c_lr"], bc_absorb_width=p["absorb_width"])
    dom_hi = (nx * dx, ny * dx)
    bc = _bc(case) if case["kind"] == "patch" else (REFLECT,) * 4
    A = Enlightning(prm, variant=case["variant"], domain_xhi=dom_hi, bc=bc)
    P = Patch((0, nx - 1, 0, ny - 1), (0.0, 0.0), (dx, dx), level=case["level"],
              touches=_touches(case) if case["kind"] == "patch" else (0, 0, 0, 0)).allocate()
    P.w_scr.copy_(w)
    P.pres[0].copy_(pres)
    P.temp[0].copy_(temp)
    P.src.copy_(H)
    w_cur = P.interior(w).contiguous()
    return dict(kind=case["kind"], A=A, P=P, w=w_cur, pres=pres[None], temp=temp[None], dt=A.compute_stable_dt(P),
                tags=torch.zeros((ny, nx), dtype=torch.int32, device="cuda"), variant=VARIANTS.index(case["variant"]),
                flags=torch.zeros((ny, nx), dtype=torch.int32, device="cuda"))


def _run_patch(st):
    A, P = st["A"], st["P"]
    # the step's current data arrives as the hierarchy hands it over
    P.w_cur.copy_(st["w"])
    P.pres.copy_(st["pres"])
    P.temp.copy_(st["temp"])
    A.advance(P, st["dt"], 1)
    A.tag_gradient_detector_cells(P, st["tags"])
    return {"w": P.w_cur, "pres": P.interior(P.pres), "temp": P.interior(P.temp), "tags": st["tags"]}


def _run_rhs(st):
    from enlightning_gb300 import _lib
    A, P = st["A"], st["P"]
    p, b, g = A.p, P.box, P.g
    pitch = P.nx + 2 * g
    _lib.check(A.L.enl_rhs(
        st["variant"], b[0], b[1], b[2], b[3], g, g, _lib.darr(P.xlo), _lib.darr(P.dx), C.c_void_p(P.w_scr.data_ptr()),
        pitch, pitch * (P.ny + 2 * g), C.c_void_p(P.src.data_ptr()), C.c_void_p(P.K.data_ptr()), P.nx, P.nx * P.ny,
        C.c_void_p(P.pres.data_ptr()), C.c_void_p(P.temp.data_ptr()), p["weno_alpha"], p["kappa"], p["mu"], p["muB"],
        p["R"], p["T_star_n"], p["tau_n"], _lib.darr(p["tol"]), P.level, p["c"], p["c_lr"],
        C.c_void_p(st["flags"].data_ptr())), "enl_rhs")
    return {"K": P.K, "flags": st["flags"]}


def _prepare_pulses(case, seed):
    from enlightning_gb300.engine import Engine
    from enlightning_gb300.workloads import shelf_pack
    p, dx = _const(case), 0.1
    sides = _pulse_sizes(case)
    width = 8192 if case["n"] > 24 else 4096 if case["n"] > 4 else 2304
    pos, height = shelf_pack(sides, width)
    E = Engine(_prm(), width, int(-(-height // 8) * 8), (dx, dx), nlevels=1, bc=(REFLECT,) * 4,
               variant=case["variant"], precision=case["precision"], learned=case["learned"], independent=True)
    if case["learned"]:
        _mlp(E)
    E.set_patches(0, [(x, x + s - 1, y, y + s - 1) for (x, y), s in zip(pos, sides)])
    for q, ((x, y), s) in enumerate(zip(pos, sides)):
        w = _pulse_state(case, seed, q, s, p)
        pres, temp = _eos(w, p, 0.0)
        E.set_box_state(0, x, y, w, pres, temp)
    dt = _pulse_dt(p, dx)
    buf = E.buffer(0)
    views = [buf[:, G + y:G + y + s, G + x:G + x + s] for (x, y), s in zip(pos, sides)]
    for v in views:
        v.engine = E  # the views look into the engine's memory: it lives as long as they do
    E.capture(dt)
    return dict(E=E, steps=case["steps"], buf=buf, start=buf.clone(), views=views)


def _run_pulses(st):
    # every pass starts from the given state
    with torch.cuda.stream(_side_stream()):
        st["buf"].copy_(st["start"])
        st["E"].replay(st["steps"])
    return st["views"]


def _exchange_state(E, steps, dt, most=0):
    """`most`: cells that the host's result buffer holds (a run that regrids
    sizes it once); what the hierarchy does not fill of it stays zero."""
    host_in = E.packed_host()
    E.download(host_in)
    E.sync()
    E.capture(dt)
    host_out = torch.zeros(max(E.packed_size(), 7 * most), dtype=E.dtype).pin_memory()
    return dict(E=E, steps=steps, host_in=host_in, host_out=host_out)


def _run_exchange(st):
    E = st["E"]
    E.upload(st["host_in"])
    E.replay(st["steps"])
    E.download(st["host_out"])
    return st["host_out"]


def _prepare_amr(case, seed):
    from enlightning_gb300.engine import Engine
    p, w = _amr_state(case, seed)
    E = Engine(_prm(), case["nx"], case["ny"], (0.1, 0.1), nlevels=2, bc=(REFLECT,) * 4, variant=case["variant"],
               precision=case["precision"])
    pres, temp = _eos(w, p, 0.0)
    E.set_level_state(0, w, pres, temp)
    boxes = _amr_boxes(case)
    for l in (0, 1):
        E.set_patches(l, boxes[l])
    E.fill(0)
    E.refine_init(1, boxes[1])
    return _exchange_state(E, case["steps"], _pulse_dt(p, 0.05))


def _prepare_shock(case, seed):
    from enlightning_gb300 import workloads
    E, Hy = workloads.mach_shock(_prm(), seed=seed, nx0=case["nx"], ny0=case["ny"], precision=case["precision"],
                                 learned=case["learned"])
    if case["learned"]:
        _mlp(E)
    for _ in range(4):
        E.step(1.0)
    Hy.regrid()
    return _exchange_state(E, case["steps"], 1.0, 5 * case["nx"] * case["ny"])


def _line(case, seed, learned):
    from enlightning_gb300 import workloads
    # the channel has 200 segments on the full domain, fewer on a smaller one
    nseg = max(12, round(200 * case["nx"] / 4096))
    E, Hy, _ = workloads.line_source(_prm(), nx0=case["nx"], ny0=case["ny"], seed=seed, nseg=nseg,
                                     precision=case["precision"], learned=learned)
    if learned:
        _mlp(E)
    for s in range(20):
        if s and s % 10 == 0:
            Hy.regrid()
        E.step(1.0)
    return E, Hy


def _prepare_line(case, seed):
    E, Hy = _line(case, seed, case["learned"])
    Hy.regrid()
    # the base level and the fine patches along the channel, with room for them to grow
    return _exchange_state(E, case["steps"], 1.0, case["nx"] * case["ny"] + 250 * case["nx"] + 40000)


def _prepare_regrid(case, seed):
    E, Hy = _line(case, seed, False)
    return dict(E=E, Hy=Hy)


def _run_regrid(st):
    out = np.full((len(st["E"].patches) - 1, 2048, 4), -1, np.int32)
    for l, boxes in enumerate(st["Hy"].regrid()):
        out[l, :len(boxes)] = boxes
    return out


def _train_inputs(case, seed):
    """Features as the harvest gives them (ratios in [0, 1], many near 1, a
    log-scaled jump), labels of both classes and their class weights."""
    gen = torch.Generator()
    gen.manual_seed(seed)
    n = case["rows"]
    X = torch.rand((n, 40), generator=gen)
    near = torch.rand((n, 40), generator=gen) < 0.5
    X = torch.where(near, 1.0 - 0.05 * X, X)
    X[:, 3::4] *= 2.0
    y = (X[:, 2::4].mean(1) + 0.1 * torch.randn(n, generator=gen) > 0.75).float()
    w = torch.where(y > 0.5, 2.0, 0.7)
    P = torch.zeros(40 * 64 + 64 + 64 * 64 + 64 + 64 + 1)
    P[:2560] = torch.randn(2560, generator=gen) * math.sqrt(2.0 / 40)
    P[2624:6720] = torch.randn(4096, generator=gen) * math.sqrt(2.0 / 64)
    P[2560:2624] = 0.1 * torch.randn(64, generator=gen)
    P[6720:6784] = 0.1 * torch.randn(64, generator=gen)
    P[6784:6848] = torch.randn(64, generator=gen) * math.sqrt(1.0 / 64)
    return X.to(torch.bfloat16), y, w, P


def _prepare_train(case, seed):
    from enlightning_gb300 import _lib
    X, y, w, P = (t.cuda() for t in _train_inputs(case, seed))
    L = _lib.lib()
    L.enl_set_stream(C.c_void_p(torch.cuda.current_stream().cuda_stream))
    return dict(kind="train", L=L, X=X, y=y, w=w, P=P, g=torch.zeros_like(P),
                loss=torch.zeros(1, dtype=torch.float64, device="cuda"))


def _run_train(st):
    from enlightning_gb300 import _lib
    v = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    st["g"].zero_()
    st["loss"].zero_()
    _lib.check(st["L"].enl_mlp_grad(v(st["X"]), v(st["y"]), v(st["w"]), st["X"].shape[0], v(st["P"]), v(st["g"]),
                                    v(st["loss"])), "enl_mlp_grad")
    return {"grad": st["g"], "loss": st["loss"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    """Bytes: each input read once, each result written once.  Operations: the
    reference algorithm's count per cell and stage (606 for a DRP cell, 3944
    for a WENO5 cell with LLF splitting, about 1700 with WENO3); hybrid cells
    of level 0 count as DRP cells, which is what quiet air needs."""
    kind = case["kind"]
    if kind == "train":
        n, net = case["rows"], 40 * 64 + 64 * 64 + 64
        return {"bytes": n * (80 + 8) + 8 * 6849, "flops": n * 6 * net}
    if kind in ("patch", "rhs"):
        cells, high = case["nx"] * case["ny"], "low" not in case["variant"]
        weno = case["variant"].startswith("weno") or (case["variant"].startswith("hybrid") and case["level"] > 0)
        per = (3944 if high else 1700) if weno else 606
        ghost = (case["nx"] + 6) * (case["ny"] + 6)
        if kind == "rhs":
            return {"bytes": 8 * (7 * ghost + 6 * cells) + 4 * cells, "flops": per * cells}
        return {"bytes": 8 * (7 * ghost + 7 * cells) + 4 * cells, "flops": 3 * per * cells}
    if kind == "pulses":
        mean = (case["lo"] + case["hi"]) / 2
        cells = case["n"] * (mean * mean + (case["hi"] - case["lo"]) ** 2 / 12)
        eb = 4 if case["precision"] == F32_STATE else 8
        per = 3944 if case["variant"].startswith("weno") else 606
        return {"bytes": 14 * eb * cells * case["steps"], "flops": 3 * per * cells * case["steps"]}
    base = case["nx"] * case["ny"]
    if kind == "regrid":
        # the density and the source of the two levels that are tagged
        return {"bytes": 2 * (4 if case["precision"] == F32_STATE else 8) * 1.03 * base, "flops": 40 * 1.03 * base}
    eb = 4 if case["precision"] == F32_STATE else 8
    # fine cells: the two small patches, the whole refined shock, the channel's patches
    fine = 1280 if kind == "amr" else 4 * base if kind == "shock" else 0.045 * base
    return {"bytes": 14 * eb * (base + fine) * (1 if kind != "line" else case["steps"]),
            "flops": 3 * (606 * (0 if kind == "line" else base) + 3944 * fine) * case["steps"]}


# ---------------------------------------------------------------------------
# the same results in plain 64-bit torch
# ---------------------------------------------------------------------------

def _f(x):
    """A single-precision literal of the reference, widened."""
    return float(np.float32(x))


_A = (_f(0.79926643), _f(-0.18941314), _f(0.02651995))


def _weno(order, plus, f):
    """Reconstruction from f[-2..2] (a dict of arrays by offset)."""
    eps = _f(10.0e-6)
    if order == 5:
        a, b, c, d, e = (f[q] for q in (-2, -1, 0, 1, 2))
        k = _f(13.0 / 12.0)
        q0 = k * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2 + eps
        q1 = k * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2 + eps
        q2 = k * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2 + eps
        d0, d1, d2 = (_f(0.3), _f(0.6), _f(0.1)) if plus else (_f(0.1), _f(0.6), _f(0.3))
        z0, z1, z2 = d0 / q0 ** 2, d1 / q1 ** 2, d2 / q2 ** 2
        if plus:
            f0, f1, f2 = 2 * c + 5 * d - e, -b + 5 * c + 2 * d, 2 * a - 7 * b + 11 * c
        else:
            f0, f1, f2 = 11 * c - 7 * d + 2 * e, 2 * b + 5 * c - d, -a + 5 * b + 2 * c
        return _f(1.0 / 6.0) * ((z0 * f0 + z1 * f1 + z2 * f2) / (z0 + z1 + z2))
    b, c, d = f[-1], f[0], f[1]
    q0, q1 = eps + (d - c) ** 2, eps + (c - b) ** 2
    c0, c1 = (_f(2 / 3), _f(1 / 3)) if plus else (_f(1 / 3), _f(2 / 3))
    z0, z1 = c0 / q0 ** 2, c1 / q1 ** 2
    f0 = c + d if plus else 3 * c - d
    f1 = 3 * c - b if plus else b + c
    return 0.5 * ((z0 * f0 + z1 * f1) / (z0 + z1))


def _ratio_low(m, c, p, eps):
    t1, t2 = c - m, p - c
    return (2 * (t1 * t2).abs() + eps) / ((t1 * t1 + t2 * t2) + eps) < _f(0.9999)


def _eps_of(t):
    return (_f(0.9) * t) / (1.0 - _f(0.9) * (t * t))


def _exact_rhs(w, pres, temp, H0, p, dx, ylo, level, variant):
    """(KK, flags) of the interior of ghosted arrays (.., ny + 6, nx + 6)."""
    ny, nx = w.shape[1] - 2 * G, w.shape[2] - 2 * G

    def at(q, di, dj):
        return q[G + dj:G + dj + ny, G + di:G + di + nx]

    order = 3 if "low" in variant else 5
    u, v = w[1] / w[0], w[2] / w[0]
    if variant.startswith("weno") or (variant.startswith("hybrid") and level != 0):
        flag = torch.ones((ny, nx), dtype=torch.bool, device=w.device)
    elif variant == "drp":
        flag = torch.zeros((ny, nx), dtype=torch.bool, device=w.device)
    else:
        e = _eps_of(p["tol"][2])
        flag = torch.zeros((ny, nx), dtype=torch.bool, device=w.device)
        for q in (-1, 0, 1):
            flag |= _ratio_low(at(w[0], q - 1, 0), at(w[0], q, 0), at(w[0], q + 1, 0), e)
            flag |= _ratio_low(at(w[0], 0, q - 1), at(w[0], 0, q), at(w[0], 0, q + 1), e)
    H = _exact_sources(w, u, v, temp, H0, p, dx, at)
    K = []
    if "llf" in variant:
        qr = 3 if order == 5 else 2
        rows = torch.arange(ny, dtype=torch.float64, device=w.device)[:, None]
        ht = lambda q: ylo + dx * (rows + q + 0.5)  # noqa: E731
        ax = torch.stack([at(u, q, 0).abs() for q in range(-qr, qr + 1)]).amax(0) + p["c"] + p["c_lr"] * ht(0)
        ay = torch.stack([at(v, 0, q).abs() + p["c"] + p["c_lr"] * ht(q) for q in range(-qr, qr + 1)]).amax(0)
    else:
        ax = ay = torch.full((ny, nx), p["weno_alpha"], dtype=torch.float64, device=w.device)
    for k in range(5):
        Fx = u * w[k] + (pres if k == 1 else 0)
        Gy = v * w[k] + (pres if k == 2 else 0)
        drp = H[k] - sum(a * (at(Fx, m, 0) - at(Fx, -m, 0)) for m, a in zip((1, 2, 3), _A)) / dx \
            - sum(a * (at(Gy, 0, m) - at(Gy, 0, -m)) for m, a in zip((1, 2, 3), _A)) / dx
        out = drp
        if bool(flag.any()):
            tot = H[k]
            for F, a, off in ((Fx, ax, lambda q: (q, 0)), (Gy, ay, lambda q: (0, q))):
                fp = {q: 0.5 * (at(F, *off(q)) + a * at(w[k], *off(q))) for q in range(-3, 4)}
                fm = {q: 0.5 * (at(F, *off(q)) - a * at(w[k], *off(q))) for q in range(-3, 4)}
                sh = lambda f, s: {q: f.get(q + s) for q in range(-2, 3)}  # noqa: E731
                tot = tot + (_weno(order, True, sh(fp, -1)) + _weno(order, False, sh(fm, 0))
                             - _weno(order, True, sh(fp, 0)) - _weno(order, False, sh(fm, 1))) / dx
            out = torch.where(flag, tot, drp)
        K.append(out)
    return torch.stack(K), flag


def _exact_sources(w, u, v, temp, H0, p, dx, at):
    c43, c23 = _f(4 / 3), _f(2 / 3)
    dxx = lambda q: (at(q, -1, 0) - 2 * at(q, 0, 0) + at(q, 1, 0)) / dx ** 2  # noqa: E731
    dyy = lambda q: (at(q, 0, -1) - 2 * at(q, 0, 0) + at(q, 0, 1)) / dx ** 2  # noqa: E731
    dxy = lambda q: (at(q, 1, 1) - at(q, 1, -1) - at(q, -1, 1) + at(q, -1, -1)) / (4 * dx * dx)  # noqa: E731
    d1x = lambda q: (at(q, 1, 0) - at(q, -1, 0)) / (2 * dx)  # noqa: E731
    d1y = lambda q: (at(q, 0, 1) - at(q, 0, -1)) / (2 * dx)  # noqa: E731
    mu, muB, kap = p["mu"], p["muB"], p["kappa"]
    uxx, uyy, vxy, vyy, vxx, uxy = dxx(u), dyy(u), dxy(v), dyy(v), dxx(v), dxy(u)
    H1 = muB * (uxx + vxy) + mu * (c43 * uxx - c23 * vxy + uyy + vxy)
    H2 = muB * (vyy + uxy) + mu * (uxy + vxx + c43 * vyy - c23 * uxy)
    ux, uy, vx, vy, tx, ty = d1x(u), d1y(u), d1x(v), d1y(v), d1x(temp), d1y(temp)
    T, rho = at(temp, 0, 0), at(w[0], 0, 0)
    Tn = at(w[4], 0, 0) / rho
    M = (T - Tn) / p["tau_n"]
    cvn = _f(0.78) * p["R"] * (p["T_star_n"] / Tn) ** 2 * torch.exp(-p["T_star_n"] / Tn)
    An = (T / Tn - 1) * cvn
    pxx, pxy, pyy = c43 * ux - c23 * vy, uy + vx, c43 * vy - c23 * ux
    sigma = (muB / T * (ux + vy) ** 2 + mu / (2 * T) * (pxx ** 2 + 2 * pxy ** 2 + pyy ** 2)
             + kap / T ** 2 * (tx ** 2 + ty ** 2) + rho / T * An * M)
    H3 = sigma - rho / Tn * cvn * M - kap * (tx ** 2 + ty ** 2) / T ** 2 + kap * (dxx(temp) + dyy(temp)) / T
    H4 = rho / p["tau_n"] * (T - Tn)
    return [H0, H1, H2, H3, H4]


def _exact_fill(q, touches, bc):
    """Physical ghosts of a ghosted patch (fields: w 0..4, p, T), in place."""
    ny, nx = q.shape[1] - 2 * G, q.shape[2] - 2 * G
    sx, sy = torch.ones(7, 1, 1, dtype=q.dtype, device=q.device), torch.ones(7, 1, 1, dtype=q.dtype, device=q.device)
    sx[1], sy[2] = -1, -1
    for d, (ghost, src) in enumerate(((slice(0, G), G), (slice(G + nx, None), G + nx - 1))):
        if touches[d]:
            q[:, G:G + ny, ghost] = q[:, G:G + ny, src:src + 1] * (sx if bc[d] == REFLECT else 1)
    for d, (ghost, src) in enumerate(((slice(0, G), G), (slice(G + ny, None), G + ny - 1)), 2):
        if touches[d]:
            q[:, ghost, G:G + nx] = q[:, src:src + 1, G:G + nx] * (sy if bc[d] == REFLECT else 1)
    for xs, (gx, src) in enumerate(((slice(0, G), G), (slice(G + nx, None), G + nx - 1))):
        for ys, gy in enumerate((slice(0, G), slice(G + ny, None))):
            if touches[xs] or touches[2 + ys]:
                q[:, gy, gx] = q[:, gy, src:src + 1] * (sx if bc[xs] == REFLECT else 1)


def _exact_absorb(q, p, bc, dx, nx, ny):
    """Absorbing envelope of a patch that is the whole domain, in place."""
    amb = torch.tensor([p["rho0"], 0, 0, 0, p["rho0"] * p["T0"], p["p0"], p["T0"]], dtype=q.dtype,
                       device=q.device)[:, None, None]
    inner = q[:, G:G + ny, G:G + nx]
    for d in range(4):
        if bc[d] != ABSORB:
            continue
        n = nx if d < 2 else ny
        x = (torch.arange(n, dtype=q.dtype, device=q.device) + 0.5) * dx
        dist = x if d in (0, 2) else (n * dx - x)
        env = 1 - torch.exp(-math.log(2.0) / p["absorb_width"] ** 2 * dist * dist)
        go = (1 - env).abs() > 1e-8
        if d in (1, 3):
            env, go = env.flip(0), go.flip(0)
        before = torch.cat([torch.ones(1, dtype=torch.bool, device=q.device), go[:-1]]).cumprod(0).bool()
        first = before & go[0]  # the first row (and the walks in y) test the edge cell too
        if d < 2:
            reach = before[None, :].repeat(ny, 1)
            reach[0] = first
            fac = env[None, :].expand(ny, n)
        else:
            reach = first[:, None].expand(n, nx)
            fac = env[:, None].expand(n, nx)
        if d in (1, 3):
            ax = 1 if d == 1 else 0
            reach, fac = reach.flip(ax), fac.flip(ax)
        inner.copy_(torch.where(reach, (inner - amb) * fac + amb, inner))


def _exact_stage(q, un, p, s, dt, dx, level, variant, H0):
    """Interior (7, ny, nx) after RK stage s from the filled ghosted state q."""
    ny, nx = q.shape[1] - 2 * G, q.shape[2] - 2 * G
    K, _ = _exact_rhs(q[:5], q[5], q[6], H0, p, dx, 0.0, level, variant)
    a1, a2, b = RK[s]
    w = a1 * un + a2 * q[:5, G:G + ny, G:G + nx] + b * dt * K
    height = (torch.arange(ny, dtype=q.dtype, device=q.device)[:, None] + 0.5) * dx
    pres, temp = _eos(w, p, height)
    return torch.cat([w, pres[None], temp[None]])


def _exact_patch(case, seed):
    p, dx, w, pres, temp, H = _patch_inputs(case, seed)
    nx, ny = case["nx"], case["ny"]
    inner = (slice(None), slice(G, G + ny), slice(G, G + nx))
    if case["kind"] == "rhs":
        K, flag = _exact_rhs(w, pres, temp, H, p, dx, 0.0, case["level"], case["variant"])
        return {"K": K, "flags": flag.to(torch.int32)}
    q = torch.cat([w, pres[None], temp[None]])
    un, bc, touches = q[:5][inner].clone(), _bc(case), _touches(case)
    for s in range(3):
        _exact_fill(q, touches, bc)
        q[inner] = _exact_stage(q, un, p, s, _pulse_dt(p, dx), dx, case["level"], case["variant"], H)
        _exact_absorb(q, p, bc, dx, nx, ny)
    r = q[0]
    e = _eps_of(p["tol"][1])
    at = lambda di, dj: r[G + dj:G + dj + ny, G + di:G + di + nx]  # noqa: E731
    # the source is zero, its ratios are 1: the density alone tags
    tags = _ratio_low(at(-1, 0), at(0, 0), at(1, 0), e) | _ratio_low(at(0, -1), at(0, 0), at(0, 1), e)
    return {"w": q[:5][inner], "pres": q[5:6][inner], "temp": q[6:7][inner], "tags": tags.to(torch.int32)}


def _exact_pulses(case, seed):
    p, dx, out = _const(case), 0.1, []
    off = torch.zeros(7, dtype=torch.float64, device="cuda")
    if case["precision"] == F32_STATE:
        off = torch.tensor([p["rho0"], 0, 0, 0, p["rho0"] * p["T0"], p["p0"], p["T0"]], dtype=torch.float64,
                           device="cuda")
    for n, s in enumerate(_pulse_sizes(case)):
        w = _pulse_state(case, seed, n, s, p)
        q = torch.zeros((7, s + 2 * G, s + 2 * G), dtype=torch.float64, device="cuda")
        inner = (slice(None), slice(G, G + s), slice(G, G + s))
        pres, temp = _eos(w, p, 0.0)
        q[inner] = torch.cat([w, pres[None], temp[None]])
        H = torch.zeros((s, s), dtype=torch.float64, device="cuda")
        for _ in range(case["steps"]):
            un = q[:5][inner].clone()
            for k in range(3):
                _exact_fill(q, (1,) * 4, (REFLECT,) * 4)
                q[inner] = _exact_stage(q, un, p, k, _pulse_dt(p, dx), dx, 0, case["variant"], H)
        out.append(q[inner] - off[:, None, None])
    return out


def _exact_amr(case, seed):
    p, w = _amr_state(case, seed)
    boxes, dt = _amr_boxes(case), _pulse_dt(p, 0.05)
    nx, ny = (case["nx"], 2 * case["nx"]), (case["ny"], 2 * case["ny"])
    lev = [torch.zeros((7, ny[l] + 2 * G, nx[l] + 2 * G), dtype=torch.float64, device=w.device) for l in (0, 1)]
    mask = [torch.zeros((ny[l], nx[l]), dtype=torch.bool, device=w.device) for l in (0, 1)]
    for l in (0, 1):
        for b in boxes[l]:
            mask[l][b[2]:b[3] + 1, b[0]:b[1] + 1] = True
    pres, temp = _eos(w, p, 0.0)
    lev[0][:, G:-G, G:-G] = torch.cat([w, pres[None], temp[None]])

    def interp(c):  # bilinear in cell centres at ratio 2, to every fine cell
        i = torch.arange(2 * (c.shape[2] - 2 * G), device=c.device)
        j = torch.arange(2 * (c.shape[1] - 2 * G), device=c.device)
        xi, xj = (i + 0.5) / 2 - 0.5, (j + 0.5) / 2 - 0.5
        fi, fj = xi - xi.floor(), (xj - xj.floor())[:, None]
        a, b = xi.floor().long() + G, xj.floor().long() + G
        lo = (1 - fi) * c[:, b][:, :, a] + fi * c[:, b][:, :, a + 1]
        hi = (1 - fi) * c[:, b + 1][:, :, a] + fi * c[:, b + 1][:, :, a + 1]
        return (1 - fj) * lo + fj * hi

    def fill(L):
        _exact_fill(L[0], (1,) * 4, (REFLECT,) * 4)
        f = L[1][:, G:-G, G:-G]
        f.copy_(torch.where(mask[1], f, interp(L[0])))
        _exact_fill(L[1], (1,) * 4, (REFLECT,) * 4)

    _exact_fill(lev[0], (1,) * 4, (REFLECT,) * 4)
    lev[1][:, G:-G, G:-G] = interp(lev[0])
    H = [torch.zeros((ny[l], nx[l]), dtype=torch.float64, device=w.device) for l in (0, 1)]
    for _ in range(case["steps"]):
        un = [q[:5, G:-G, G:-G].clone() for q in lev]
        for s in range(3):
            fill(lev)
            for l in (0, 1):
                new = _exact_stage(lev[l], un[l], p, s, dt, 0.1 / 2 ** l, l, case["variant"], H[l])
                v = lev[l][:, G:-G, G:-G]
                v.copy_(torch.where(mask[l], new, v))
        f, c = lev[1][:, G:-G, G:-G], lev[0][:, G:-G, G:-G]
        mean = 0.25 * (f[:, 0::2, 0::2] + f[:, 0::2, 1::2] + f[:, 1::2, 0::2] + f[:, 1::2, 1::2])
        c.copy_(torch.where(mask[1][0::2, 0::2], mean, c))
    # the packed order: field by field, level by level, patch by patch, in 32x8 tiles
    off = (p["rho0"], 0, 0, 0, p["rho0"] * p["T0"], p["p0"], p["T0"])
    parts = []
    for k in range(7):
        for l in (0, 1):
            q = lev[l][k, G:-G, G:-G] - (off[k] if case["precision"] == F32_STATE else 0.0)
            for b in boxes[l]:
                for j in range(b[2], b[3] + 1, 8):
                    for i in range(b[0], b[1] + 1, 32):
                        parts.append(q[j:min(j + 8, b[3] + 1), i:min(i + 32, b[1] + 1)].reshape(-1))
    return torch.cat(parts).cpu()


def _exact_train(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    X, y, w, P = (t.to(dev).double() for t in _train_inputs(case, seed))
    P.requires_grad_(True)
    W1, b1, W2, b2 = P[:2560].view(40, 64), P[2560:2624], P[2624:6720].view(64, 64), P[6720:6784]
    gelu = torch.nn.functional.gelu
    z = gelu(gelu(X @ W1 + b1) @ W2 + b2) @ P[6784:6848] + P[6848]
    loss = (w * (z.clamp(min=0) - y * z + torch.log1p(torch.exp(-z.abs())))).sum()
    loss.backward()
    return {"grad": P.grad, "loss": loss.detach().reshape(1)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("patch", "rhs"):
        return _exact_patch(case, seed)
    if kind == "pulses" and not case["learned"]:
        return _exact_pulses(case, seed)
    if kind == "amr":
        return _exact_amr(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    return None  # the learned decisions and the clustered hierarchy have no plain 64-bit value
