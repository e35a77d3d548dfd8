"""Few objects on a fine grid: the row tables, not the objects, are the work of a scan."""
import numpy as np
import pytest

from helpers import records_equal, to_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ladds_b200 import build, capi

    build.build_gpu()
    return capi


@pytest.mark.parametrize("n", [1, 255, 257, 5000])
@pytest.mark.parametrize("rows", [(1, 1), (31, 33), (32, 32), (640, 800), (1000, 1000)])
def test_counts_are_cleared_for_the_next_scan(capi, oracle, n, rows):
    """Row tables below and above what the objects' own blocks clear, to several
    values a thread: scan after scan, on both sets, finds the oracle's records."""
    ny, nz = rows
    lo, hi = np.zeros(3), np.array([12.0, ny, nz])
    rng = np.random.default_rng(n + ny)
    middle = (lo + hi) / 2
    r = np.clip(rng.normal(middle, np.minimum(6.0, hi / 4), (n, 3)), lo + 1e-3, hi - 1e-3)
    v, one = rng.uniform(-1.0, 1.0, (n, 3)), np.ones(n)
    pop = dict(x=r[:, 0].copy(), y=r[:, 1].copy(), z=r[:, 2].copy(), vx=v[:, 0].copy(), vy=v[:, 1].copy(),
               vz=v[:, 2].copy(), radius=1e-4 * one, aom=1e-9 * one, bc_inv=0.01 * one,
               id=np.arange(n, dtype=np.uint64))
    from ladds_b200.population import as_population

    p = oracle.scan_params(cutoff=0.9, dt=0.1, evasion_cutoff=0.01, conjunction_threshold=0.5)
    ref = oracle.scan_bruteforce(to_oracle(oracle, as_population(pop)), p, cap=max(1024, n * n // 2))
    assert n < 5000 or len(ref) > 50
    cfg = dict(cutoff=0.9, cellSize=1.0, boxMin=list(lo), boxMax=list(hi), conjunctionThreshold=0.5, evasionCutoff=0.01)
    with capi.Context(capi.default_config(**cfg)) as ctx:
        ctx.upload(pop)
        for _ in range(5):
            assert records_equal(ctx.conjunctions(0.1, cap=1 << 16), ref)
        assert ctx.grid()[0] == (12, ny, nz)


def test_few_objects_cost_no_more_than_many(capi):
    """2.56e6 rows (cells of 12.5 km): an iteration of ten objects takes no longer than one of 10,000
    (equal here; 2.2 times as long when one block cleared the counts)."""
    pop = capi.generate_population(0, 11, 10_000)
    best = []
    for n in (10, 10_000):
        with capi.Context(capi.default_config(cutoff=10.0, conjunctionThreshold=0.5)) as ctx:
            ctx.upload({k: v[:n] for k, v in pop.items()})
            best.append(min(ctx.step(20).stats.deviceMs for _ in range(8)))
            assert ctx.grid()[0][1] * ctx.grid()[0][2] == 2_560_000
    assert best[0] < 1.3 * best[1]
