"""The screening form for dense populations: candidates screened in the buffer that
holds them."""
import numpy as np
import pytest

from helpers import records_equal

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ladds_b200 import build, capi

    build.build_gpu()
    return capi


def test_buffer_form_is_faster_where_cells_are_crowded(capi):
    """500,000 objects in cells of 256 (some 1e9 pair tests by tiles, 3e7 candidates): the
    scan in the buffer form takes no longer than the listed form, whose candidates go
    through memory, and finds the same records."""
    n, edge = 500_000, 2000.0
    rng = np.random.default_rng(7)
    r, v = rng.uniform(7000.0, 7000.0 + edge, (n, 3)), rng.uniform(-7.0, 7.0, (n, 3))
    one = np.ones(n)
    pop = dict(x=r[:, 0].copy(), y=r[:, 1].copy(), z=r[:, 2].copy(), vx=v[:, 0].copy(), vy=v[:, 1].copy(),
               vz=v[:, 2].copy(), radius=0.1 * one, aom=1e-9 * one, bc_inv=0.01 * one,
               id=np.arange(n, dtype=np.uint64))
    cfg = dict(cellSize=160.0, boxMin=[7000.0] * 3, boxMax=[7000.0 + edge] * 3, conjunctionThreshold=0.2,
               nearThresholdRel=0.0)
    found, times = [], []
    for screen in (capi.SCREEN_LISTS, capi.SCREEN_BUFFER):
        with capi.Context(capi.default_config(scanScreen=screen, **cfg)) as ctx:
            ctx.upload(pop)
            found.append(ctx.conjunctions(10.0, cap=1 << 16))
            ctx.set_profiling(True)
            best = np.inf
            for _ in range(5):
                before = ctx.phase_times()
                ctx.conjunctions(10.0, cap=1 << 16)
                after = ctx.phase_times()
                best = min(best, sum(getattr(after, p) - getattr(before, p) for p in ("candidatesMs", "evaluateMs")))
            times.append(best)
    assert len(found[0]) > 100 and records_equal(found[0], found[1])
    assert times[1] < times[0]
