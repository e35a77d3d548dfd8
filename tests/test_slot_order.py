"""The population in slot order on the GPU: the order in which records leave
(pack_layers) through growth, removal and truncation, the cell order for row
tables of every scan form, overlapped iterations against single ones, and the
pair walk for every reach against the oracle."""
import numpy as np
import pytest

from helpers import describe_diff, records_equal, to_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ladds_b200 import build, capi

    build.build_gpu()
    return capi


def cloud(n, seed, lo, hi, first_id=0):
    rng = np.random.default_rng(seed)
    r = rng.uniform(lo, hi, (n, 3))
    v = rng.uniform(-2.0, 2.0, (n, 3))
    one = np.ones(n)
    return dict(x=r[:, 0], y=r[:, 1], z=r[:, 2], vx=v[:, 0], vy=v[:, 1], vz=v[:, 2], radius=0.1 * one,
                aom=1e-9 * one, bc_inv=0.01 * one, id=np.arange(first_id, first_id + n, dtype=np.uint64))


@pytest.mark.parametrize("scanned", [False, True])
def test_pack_order_through_growth_removal_truncation(capi, scanned):
    import torch

    lo, hi = [7000.0, -100.0, -100.0], [7200.0, 100.0, 100.0]
    a, b = cloud(3000, 1, lo, hi), cloud(6000, 2, lo, hi, 3000)  # the append outgrows the first capacity
    with capi.Context(capi.default_config(cutoff=10.0, boxMin=lo, boxMax=hi)) as ctx:
        ctx.upload(a)
        order = np.arange(3000)
        if scanned:
            ctx.conjunctions(1.0)
            order = ctx.cell_order()[1].astype(np.int64)
        ctx.append(b)
        ids = np.concatenate([order, np.arange(3000, 9000)])  # ids in the population's order
        buf = torch.empty(9000 * 96, dtype=torch.uint8, device="cuda")

        def packed():
            n = ctx.pack_layers(0, ctx.grid()[0][2], False, buf, 9000)
            return np.frombuffer(buf.cpu().numpy().tobytes(), dtype=capi.STATE_RECORD_DTYPE)["id"][:n]

        assert np.array_equal(packed(), ids)
        gone = np.random.default_rng(3).choice(9000, 2500, replace=False)
        ctx.remove_slots(gone)
        ids = ids[~np.isin(ids, gone)]
        assert np.array_equal(packed(), ids)
        left = np.sort(ids)  # slot order
        assert np.array_equal(ctx.download()["id"], left)
        ctx.truncate(4000)
        ids = ids[np.isin(ids, left[:4000])]
        assert np.array_equal(packed(), ids)
        assert np.array_equal(ctx.download()["id"], left[:4000])


@pytest.mark.parametrize("ny,nz", [(1, 1), (31, 33), (32, 32), (341, 384), (256, 512), (500, 300), (1100, 1000)])
def test_cell_order_for_row_tables(capi, ny, nz):
    """Row counts around one block of the row scan, the last size it takes in one
    launch (128 blocks), two passes, and three levels (above 2^20 rows)."""
    n, nx = 20_011, 7
    lo, hi = np.zeros(3), np.array([nx, ny, nz], dtype=float)
    pop = cloud(n, ny + nz, lo - 0.5, hi + 0.5)
    with capi.Context(capi.default_config(cutoff=0.5, cellSize=1.0, boxMin=list(lo), boxMax=list(hi))) as ctx:
        ctx.upload(pop)
        for _ in range(2):  # the second sort uses the other set of tables
            ctx.conjunctions(1.0)
            keys, slots = ctx.cell_order()
            assert ctx.grid()[0] == (nx, ny, nz)
            ix, iy, iz = (np.clip(np.floor(pop[k]), 0, m - 1).astype(np.int64)
                          for k, m in zip("xyz", (nx, ny, nz)))
            want = (iz * ny + iy) * nx + ix
            order = np.argsort(want, kind="stable")
            assert np.array_equal(slots, order)
            assert np.array_equal(keys, want[order])


@pytest.mark.parametrize("every", [1, 2, 3, 5])
@pytest.mark.parametrize("precision", [0, 1])
def test_overlapped_iterations_equal_single_ones(capi, every, precision):
    """A call of many iterations (ring of three states, two sets of sort tables,
    one propagation launch per scan; the repeated calls in graphs) against one
    call per iteration without graphs."""
    pop = capi.generate_population(0, 5, 3001)
    pop["activity"][::40] = capi.EVASIVE_PRESERVING
    kw = dict(componentMask=capi.PROP_ALL, precision=precision, timestepsPerCollisionDetection=every,
              conjunctionThreshold=70.0)
    with capi.Context(capi.default_config(**kw)) as a, capi.Context(capi.default_config(useGraphs=0, **kw)) as b:
        for ctx in (a, b):
            ctx.upload(pop)
            ctx.mark_deleted(np.arange(0, 3001, 37))
        for calls in (11, 4, 1) + (30,) * 6:
            many = a.step(calls).records
            ones = np.concatenate([b.step(1).records for _ in range(calls)])
            assert len(many) > 0 or calls < every
            assert many.tobytes() == ones.tobytes()
            for p, q in zip(a.get_state(), b.get_state()):
                assert np.array_equal(p, q)


@pytest.mark.parametrize("every", [1, 4, 100])
def test_graph_calls_from_every_buffer(capi, every):
    """Calls of the iterations that graphs are kept for, begun in each of the
    ring's buffers and sort sets (calls of 1 to 5 iterations in between), and
    calls without a scan after one with: records, states and the order in which
    records leave equal those of launches one by one."""
    import torch

    pop = capi.generate_population(0, 5, 3001)
    kw = dict(componentMask=capi.PROP_ALL, timestepsPerCollisionDetection=every, conjunctionThreshold=70.0)
    with capi.Context(capi.default_config(**kw)) as a, capi.Context(capi.default_config(useGraphs=0, **kw)) as b:
        bufs = [torch.zeros(3001 * capi.STATE_RECORD_DTYPE.itemsize, dtype=torch.uint8, device="cuda") for _ in range(2)]
        for ctx in (a, b):
            ctx.upload(pop)
        for steps in (40, 1, 40, 2, 40, 3, 40, 40, 5, 40, 33, 40):
            got, want = a.step(steps).records, b.step(steps).records
            assert got.tobytes() == want.tobytes()
            for p, q in zip(a.get_state(), b.get_state()):
                assert np.array_equal(p, q)
            for ctx, buf in zip((a, b), bufs):
                assert ctx.pack_layers(0, ctx.grid()[0][2], False, buf, 3001) == 3001
            assert torch.equal(*bufs)


@pytest.mark.parametrize("screen", [0, 1])
@pytest.mark.parametrize("cell", [20.0, 15.0, 14.0, 10.0, 7.0, 5.0, 2.5])
def test_pair_walk_for_every_reach(capi, oracle, cell, screen):
    """Reach 1; reach 2 without and with its corner rows at full width (cells
    above and below cutoff / sqrt(2) and cutoff / sqrt(3)); 3, 4 and 8 (rows
    beyond the table).  A third of the objects lie outside the grid box on every
    side; parents, deleted objects and a halo are among them."""
    lo, hi = np.array([7000.0, -60.0, -60.0]), np.array([7130.0, 60.0, 70.0])
    pop = cloud(3000, 17, lo - 35.0, hi + 35.0)
    pop["parent"] = np.full(3000, np.uint64(0xFFFFFFFFFFFFFFFF))
    pop["parent"][:300] = np.arange(300) % 3
    kw = dict(cutoff=20.0, cellSize=cell, boxMin=list(lo), boxMax=list(hi), scanScreen=screen,
              conjunctionThreshold=15.0, evasionCutoff=3.0)
    with capi.Context(capi.default_config(**kw)) as ctx:
        ctx.upload(pop)
        recs = ctx.conjunctions(1.0)
        p = oracle.scan_params(cutoff=20.0, dt=1.0, evasion_cutoff=3.0, conjunction_threshold=15.0)
        ref = oracle.scan_bruteforce(to_oracle(oracle, ctx.download()), p)
        assert len(ref) > 1000
        assert records_equal(recs, ref), describe_diff(recs, ref)
        gone = np.arange(5, 3000, 11)
        ctx.mark_deleted(gone)
        left = ctx.conjunctions(1.0)
        keep = ~np.isin(ref["slotA"], gone) & ~np.isin(ref["slotB"], gone)
        assert records_equal(left, ref[keep]), describe_diff(left, ref[keep])


@pytest.mark.parametrize("screen", [0, 1])
@pytest.mark.parametrize("cell", [20.0, 10.0])
def test_crowded_cells_beside_sparse_ones(capi, oracle, cell, screen):
    """Fragment clouds in a few cells: source batches of one group, of two, and
    of less than half of any; sparse cells beside them whose windows hold enough
    items for the walk to leave passes to the tiles; rows sorted by a CTA."""
    rng = np.random.default_rng(23)
    lo, hi = np.array([7000.0, -50.0, -50.0]), np.array([7100.0, 50.0, 50.0])
    parts = [(2600, [7030.0, 10.0, 10.0], 3.0, 1), (1500, [7045.0, 10.0, 10.0], 6.0, 2),
             (400, [7045.0, 12.0, 10.0], 6.0, 3), (30, [7030.0, 10.0, 10.0], 3.0, None)]
    r = np.concatenate([rng.normal(c, s, (m, 3)) for m, c, s, _ in parts] + [rng.uniform(lo, hi, (900, 3))])
    n = len(r)
    pop = cloud(n, 5, lo, hi)
    pop["x"], pop["y"], pop["z"] = r[:, 0].copy(), r[:, 1].copy(), r[:, 2].copy()
    none = np.uint64(0xFFFFFFFFFFFFFFFF)
    pop["parent"] = np.concatenate([np.full(m, none if g is None else np.uint64(g)) for m, _, _, g in parts]
                                   + [np.full(900, none)])
    pop["parent"][-60:] = 1  # fragments of the first cloud in sparse cells
    order = rng.permutation(n)
    pop = {k: (v if k == "id" else v[order]) for k, v in pop.items()}
    kw = dict(cutoff=20.0, cellSize=cell, boxMin=list(lo), boxMax=list(hi), scanScreen=screen,
              conjunctionThreshold=0.5, evasionCutoff=0.1)
    with capi.Context(capi.default_config(**kw)) as ctx:
        ctx.upload(pop)
        recs = ctx.conjunctions(0.2)
    p = oracle.scan_params(cutoff=20.0, dt=0.2, evasion_cutoff=0.1, conjunction_threshold=0.5)
    ref = oracle.scan_bruteforce(to_oracle(oracle, capi_pop(pop)), p)
    assert len(ref) > 200
    assert records_equal(recs, ref), describe_diff(recs, ref)


def capi_pop(pop):
    from ladds_b200.population import as_population

    return as_population(pop)


@pytest.mark.parametrize("n", [1, 31, 700, 9000])
def test_sparse_rows_in_batches(capi, oracle, n):
    """Fewer objects than rows: batches of rows sorted side by side, with rows of
    254 to 257 objects (byte counters to 255), crowded cells, one batch of more
    objects than it stages, and an empty last batch (rows not a multiple of 8)."""
    nx, ny, nz = 300, 101, 99
    lo, hi = np.zeros(3), np.array([nx, ny, nz], dtype=float)
    rng = np.random.default_rng(n)
    pop = cloud(n, 4, lo, hi)
    if n >= 9000:
        at = 0
        for count, (y, z) in ((254, (10, 5)), (255, (30, 5)), (256, (50, 6)), (257, (70, 7)), (250, (2, 50)),
                              (200, (3, 50)), (180, (4, 50))):
            s = slice(at, at + count)
            pop["x"][s] = rng.uniform(0, nx, count) if count != 255 else 40.0 + rng.uniform(0, 5, count)
            pop["y"][s], pop["z"][s] = y + 0.5, z + rng.uniform(0.0, 1.0, count)
            at += count
    order = rng.permutation(n)
    pop = {k: (v if k == "id" else v[order]) for k, v in pop.items()}
    kw = dict(cutoff=0.9, cellSize=1.0, boxMin=list(lo), boxMax=list(hi), conjunctionThreshold=0.6, evasionCutoff=0.1)
    with capi.Context(capi.default_config(**kw)) as ctx:
        ctx.upload(pop)
        recs = ctx.conjunctions(0.1)
        keys, slots = ctx.cell_order()
    ix, iy, iz = (np.clip(np.floor(pop[k]), 0, m - 1).astype(np.int64) for k, m in zip("xyz", (nx, ny, nz)))
    want = (iz * ny + iy) * nx + ix
    order = np.argsort(want, kind="stable")
    assert np.array_equal(slots, order) and np.array_equal(keys, want[order])
    p = oracle.scan_params(cutoff=0.9, dt=0.1, evasion_cutoff=0.1, conjunction_threshold=0.6)
    ref = oracle.scan_bruteforce(to_oracle(oracle, capi_pop(pop)), p)
    assert n < 9000 or len(ref) > 100
    assert records_equal(recs, ref), describe_diff(recs, ref)
