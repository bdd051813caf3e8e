"""The stage kernel's deal: every block's first run of tiles, and its second
where runs are single tiles, come from the block's index, the rest from the
counter (in FP64, up to eight tiles a block, when the tile before is done).
Tables around one, two, eight and sixteen tiles a block, in each tile order and
run length, give the state of the schedule that counts every tile (order 3) bit
for bit; and a table of fewer tiles than blocks takes one tile's time."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from enlightning_gb300.constants import REFLECT, default_params  # noqa: E402
from enlightning_gb300.engine import PREC_FP32_STATE, PREC_FP64, Engine  # noqa: E402
from test_gpu_uniform import _bits  # noqa: E402


def row_of_tiles(n, precision, variant="hybrid_high_llf"):
    """One level of n tiles side by side, the last one ragged, in motion."""
    nx, prm = 32 * n - 4, default_params()
    E = Engine(prm, nx, 8, (0.1, 0.1), bc=(REFLECT,) * 4, precision=precision, variant=variant, dense=True)
    E.set_patches(0, [(0, nx - 1, 0, 7)])
    w = E.buffer(0, 0)
    rng = torch.Generator(device="cuda").manual_seed(n)
    off = [prm["rho0"], 0.0, 0.0, 0.0, prm["rho0"] * prm["T0"], prm["p0"], prm["T0"]]
    for k, (o, a) in enumerate(zip(off, (0.01, 3.0, 3.0, 1.0, 0.1, 50.0, 0.1))):
        w[k] = (o if precision == PREC_FP64 else 0.0) + a * torch.randn(w.shape[1:], generator=rng, device="cuda",
                                                                        dtype=w.dtype)
    torch.cuda.synchronize()
    return E


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_FP32_STATE])
@pytest.mark.parametrize("share", [0, 1, 2, 8, 16])
def test_every_tile_once(precision, share):
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    for n in sorted({max(1, share * nsm + d) for d in (-1, 0, 1)}):
        E = row_of_tiles(n, precision)
        start, ref = E.buffer(0, 0).clone(), None
        for order, run in ((3, 1), (0, 1), (1, 1), (2, 1), (0, 3), (1, 16)):
            E.set_schedule(blocks_per_sm=1, tile_order=order, reuse=0, run=run)
            E.buffer(0, 0).copy_(start)
            for q in (1, 2):
                E.buffer(0, q).fill_(float("nan"))
            torch.cuda.synchronize()
            E.step(1e-6)
            torch.cuda.synchronize()
            out = _bits(E.buffer(0, 0)[:, 3:-3, 3:-3])
            ref = out if ref is None else ref
            assert np.array_equal(out, ref), (n, order, run)
        assert not np.array_equal(ref, _bits(start[:, 3:-3, 3:-3]))
        E.close()


def test_fewer_tiles_than_blocks_take_one_tiles_time():
    """FP64 WENO tiles on half of the SMs take the time of one tile, but for
    their shared caches (2 tiles in a row in some block: twice that)."""
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    ms = []
    for n in (1, nsm // 2):
        E = row_of_tiles(n, PREC_FP64, "weno_high_llf")
        E.profile(1)
        t = []
        for _ in range(12):
            E.step(1e-7)
            torch.cuda.synchronize()
            t.append(E.profile(1)[0])
        ms.append(min(t[2:]))
        E.close()
    assert ms[1] < 1.5 * ms[0], ms
