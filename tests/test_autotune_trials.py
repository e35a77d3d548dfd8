"""The autotuner's trials run what the tuned context runs: the scan's breakup groups
and halo, and graphs where the context's calls run in graphs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ladds_b200 import build, capi

    build.build_gpu()
    return capi


def with_clouds(pop, clouds, fragments, seed=3):
    """The population with the first objects of each slice moved close around one of them,
    as fragments of one breakup."""
    rng = np.random.default_rng(seed)
    pop = {k: v.copy() for k, v in pop.items()}
    pop["parent"][:] = np.uint64(0xFFFFFFFFFFFFFFFF)
    for c in range(clouds):
        s = slice(c * fragments, (c + 1) * fragments)
        for k in ("x", "y", "z"):
            pop[k][s] = pop[k][c * fragments] + rng.normal(0.0, 15.0, fragments)
        for k in ("vx", "vy", "vz"):
            pop[k][s] = pop[k][c * fragments] + rng.normal(0.0, 0.01, fragments)
        pop["parent"][s] = c
    return pop


def test_trials_skip_breakup_groups(capi):
    """Two clouds of 20,000 fragments within 100 km: 4e8 pairs, none of which can yield a
    record.  A trial's iteration takes the time of the context's own (both on the device, the
    best of several); without the groups it is 15 times as long."""
    pop = with_clouds(capi.generate_population(0, 31, 150_000), 2, 20_000)
    cfg = dict(componentMask=capi.KEP, precision=capi.PRECISION_SPLIT)
    with capi.Context(capi.default_config(**cfg)) as tuned, capi.Context(capi.default_config(**cfg)) as plain:
        for ctx in (tuned, plain):
            ctx.upload(pop)
        own = min(plain.step(2).stats.deviceMs / 2 for _ in range(4))
        best, trials = tuned.autotune(2)
        edge = plain.grid()[2]
        same = min(t["msPerStep"] for t in trials if t["cellSize"] == edge)
        assert best["msPerStep"] <= same < 3.0 * own
        plain.upload(pop)
        plain.set_iteration(0)
        a, b = tuned.step(8), plain.step(8)
        assert a.records.tobytes() == b.records.tobytes()
        for p, q in zip(tuned.get_state(), plain.get_state()):
            assert np.array_equal(p, q)


@pytest.mark.parametrize("steps", [16, 128])
def test_trials_run_in_graphs(capi, steps):
    """Below 125,000 objects, where launches bound an iteration: trials at the context's
    edge take the time of its own calls in graphs (15.5 us an iteration here), whatever
    their chunk length; launched one by one they take 2.3 times as long."""
    pop = capi.generate_population(0, 31, 10_000)
    with capi.Context(capi.default_config(conjunctionThreshold=0.5)) as tuned, \
            capi.Context(capi.default_config(conjunctionThreshold=0.5)) as plain:
        tuned.upload(pop)
        plain.upload(pop)
        own = min(plain.step(128).stats.deviceMs / 128 for _ in range(6))
        edge = plain.grid()[2]
        trials = [t for _ in range(2) for t in tuned.autotune(steps)[1]]
        for screen in (0, 1):
            assert min(t["msPerStep"] for t in trials if t["cellSize"] == edge and t["scanScreen"] == screen) < 1.5 * own
        by_chunk = {t["chunkSteps"]: [] for t in trials}
        for t in trials:
            by_chunk[t["chunkSteps"]].append(t["msPerStep"])
        assert set(by_chunk) == {32, 64, 128}
        assert max(min(v) for v in by_chunk.values()) < 1.5 * own
