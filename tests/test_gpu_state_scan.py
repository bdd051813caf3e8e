"""The pass over the state at the start of an adaptive step, on a table large
enough (9,728 tiles or more) that stage 1 skips uniform tiles with its
records: the state must be bit for bit that of the cell-by-cell computation,
and dt the CFL rule's (one rounding each of the quotient, the sum and the
division by the maximum: 3 x 2^-53, the storage's roundings for FP32)."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300 import workloads  # noqa: E402
from enlightning_gb300.constants import default_params  # noqa: E402
from enlightning_gb300.engine import PREC_FP32_STATE, PREC_FP64  # noqa: E402
from test_gpu_uniform import _bits  # noqa: E402


def _engine(precision, dense, uv):
    """A ragged base (2,412 x 1,050 cells), ambient but for the source, a tile
    with one odd cell in each field in turn, and (uv) a uniform flow."""
    E, H, _ = workloads.line_source(default_params(), nx0=2412, ny0=1050, dx0=0.5, nlevels=2, nseg=20,
                                    precision=precision, base_patch=256, dense=dense)
    w = E.buffer(0, 0)
    if uv:
        w[1, 700:900, 1200:1700] += 3.0
        w[2, 700:900, 1200:1700] -= 5.0
    for k in range(7):  # cells in the middle of otherwise uniform tiles, and at a tile's corners
        w[k, 3 + 900 + 8 * k, 3 + 300 + 32 * k] *= 1.0 + 1e-6
        w[k, 3 + 903 + 8 * k, 3 + 310 + 32 * k] += 1e-3
    E.buffer(0, 3)[0, 3 + 980, 3 + 1500] = 7.0  # H0 alone
    torch.cuda.synchronize()
    return E


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_FP32_STATE])
@pytest.mark.parametrize("uv", [False, True])
def test_stage_one_skips_bit_identically(precision, uv):
    out, times, reused = {}, {}, {}
    for dense in (True, False):
        E = _engine(precision, dense, uv)
        E.stats()
        times[dense] = []
        for _ in range(3):
            E.step(1.0)
            times[dense].append(E.time())
        torch.cuda.synchronize()
        assert E.health() == 0
        reused[dense] = int(E.stats()[:, 3].sum())
        out[dense] = [_bits(E.buffer(l, 0)) for l in range(E.nlevels)]
        E.close()
    assert reused[True] == 0 and reused[False] > 3 * 256 * 4000
    assert times[True] == times[False]
    for a, b in zip(out[True], out[False]):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_FP32_STATE])
def test_dt_is_the_rule(precision):
    E = _engine(precision, False, True)
    prm = default_params()
    big = 0.0
    for l in range(E.nlevels):
        w = E.buffer(l, 0)[:, 3:-3, 3:-3].double().cpu().numpy()
        for b in E.patches[l]:
            s = w[:3, b[2]:b[3] + 1, b[0]:b[1] + 1]
            rho = s[0] + (prm["rho0"] if precision == PREC_FP32_STATE else 0.0)
            big = max(big, float(np.max(np.maximum(np.abs(s[1]), np.abs(s[2])) / np.abs(rho))))
    E.step(1.0)
    dt, _ = E.time()
    want = 0.5 * 0.25 / (big + prm["c"])
    assert dt == pytest.approx(want, rel=3 * 2.0 ** -53 if precision == PREC_FP64 else 4 * 2.0 ** -24, abs=0)
    # a cell without a speed forces the smallest step and is reported
    E.buffer(0, 0)[1, 3 + 980, 3 + 1500] = float("nan")
    E.buffer(0, 0)[2, 3 + 980, 3 + 1500] = float("nan")
    torch.cuda.synchronize()
    E.step(1.0)
    assert E.time()[0] < 1e-290
    E.close()


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_FP32_STATE])
@pytest.mark.parametrize("learned", [False, True])
def test_line_source_with_regrids_bit_identical(precision, learned):
    """Three levels and regrids, stage 1 skipping all the while (10,240 base
    tiles), with the captured step as users replay it."""
    from enlightning_gb300 import sensor
    out = {}
    for dense in (True, False):
        E, H, _ = workloads.line_source(default_params(), nx0=2048, ny0=1280, dx0=0.5, nlevels=3, nseg=60,
                                        precision=precision, learned=learned, dense=dense)
        if learned:
            E.set_mlp(*sensor.load_weights())
        E.stats()
        torch.cuda.synchronize()
        side = torch.cuda.Stream()  # (a capture needs a stream of its own)
        with torch.cuda.stream(side):
            E.L.enl_set_stream(C.c_void_p(side.cuda_stream))
            for s in range(12):
                if s and s % 5 == 0:
                    H.regrid()
                if s % 3 == 2:
                    E.capture(1.0)
                    E.replay(1)
                else:
                    E.step(1.0)
        torch.cuda.synchronize()
        E.L.enl_set_stream(C.c_void_p(torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert E.health() == 0
        assert (int(E.stats()[:, 3].sum()) == 0) == dense
        out[dense] = ([list(p) for p in E.patches], [_bits(E.buffer(l, 0)) for l in range(E.nlevels)], E.time())
        E.close()
    assert out[True][0] == out[False][0] and out[True][2] == out[False][2]
    for a, b in zip(out[True][1], out[False][1]):
        assert np.array_equal(a, b)
