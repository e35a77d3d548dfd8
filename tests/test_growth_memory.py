"""Growth of a population on a device whose memory is nearly full: the new arrays do
not fit beside the old ones, or not at all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 2_000_000  # 429 bytes each: 0.86 GB, and 1.29 GB for the 3,000,000 that an append grows them to


@pytest.fixture(scope="module")
def capi():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ladds_b200 import build, capi

    build.build_gpu()
    return capi


def leave_free(nbytes):
    """Device memory taken so that about `nbytes` are left."""
    import torch

    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    taken = torch.empty(free - nbytes, dtype=torch.uint8, device="cuda")
    assert abs(torch.cuda.mem_get_info()[0] - nbytes) < 64 << 20
    return taken


@pytest.mark.parametrize("free_mb,grows", [(1000, True), (200, False)])
def test_growth_beside_full_memory(capi, free_mb, grows):
    """With 1.0 GB free the new block does not fit beside the old one, but in its place;
    with 0.2 GB not even so: an error, and the population, its cell order, its iteration
    and the order in which records leave are what they were.  Either way the next
    iterations are those of a context with all memory."""
    import torch

    pop = capi.generate_population(0, 9, N + 1000)
    first = {k: v[:N] for k, v in pop.items()}
    more = {k: v[N:] for k, v in pop.items()}
    buf = torch.zeros((N + 1000) * capi.STATE_RECORD_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    cfg = dict(componentMask=capi.KEP | capi.J2, conjunctionThreshold=1.0)

    def packed(ctx):
        n = ctx.pack_layers(0, ctx.grid()[0][2], False, buf, N + 1000)
        return np.frombuffer(buf.cpu().numpy().tobytes(), dtype=capi.STATE_RECORD_DTYPE)[:n]

    with capi.Context(capi.default_config(**cfg)) as ctx, capi.Context(capi.default_config(**cfg)) as roomy:
        for c in (ctx, roomy):
            c.upload(first)
            c.step(2)
            c.get_state()  # the pinned staging of both is in place
        order, records = ctx.cell_order(), packed(ctx)
        roomy.reserve(N + 1000)
        taken = leave_free(free_mb << 20)
        try:
            if grows:
                ctx.append(more)
            else:
                with pytest.raises(capi.LaddsError) as e:
                    ctx.append(more)
                assert e.value.code == capi.ERR_ALLOC
                for a, b in zip(ctx.cell_order(), order):
                    assert np.array_equal(a, b)
            after = packed(ctx)
            assert np.array_equal(after[:N], records)
            assert len(after) == (N + 1000 if grows else N)
            if grows:
                assert np.array_equal(after["id"][N:], more["id"])
                roomy.append(more)
            got, want = ctx.step(3), roomy.step(3)
        finally:
            del taken
            torch.cuda.empty_cache()
        assert got.records.tobytes() == want.records.tobytes()
        for a, b in zip(ctx.get_state(), roomy.get_state()):
            assert np.array_equal(a, b)


def test_adjoint_records_make_room(capi):
    """The records that an adjoint's forward sweep keeps (0.85 GB here) give way to a
    growth that needs their memory, and the reverse sweep takes its checkpoints
    instead: equal to the bit, also when asked for twice."""
    import torch

    pop = capi.generate_population(0, 9, N + 1000)
    first = {k: v[:N] for k, v in pop.items()}
    more = {k: v[N:] for k, v in pop.items()}
    with capi.Context(capi.default_config(componentMask=capi.PROP_ALL)) as ctx:
        pairs, _ = ctx.adjoint_make_pairs(3, 4096, 1080)
        loss, miss, tca, _ = ctx.adjoint_forward(pairs, 1080, 64)
        dx, dbc, _ = ctx.adjoint_backward()
    with capi.Context(capi.default_config(componentMask=capi.PROP_ALL)) as ctx:
        ctx.upload(first)
        taken = leave_free(1200 << 20)
        try:
            got = ctx.adjoint_forward(pairs, 1080, 64)
            ctx.append(more)
            grads = [ctx.adjoint_backward()[:2] for _ in range(2)]
        finally:
            del taken
            torch.cuda.empty_cache()
        assert ctx.size() == N + 1000
        assert got[0] == loss and np.array_equal(got[1], miss) and np.array_equal(got[2], tca)
        for gx, gb in grads:
            assert np.array_equal(gx, dx) and np.array_equal(gb, dbc)
        assert np.array_equal(ctx.download()["id"], pop["id"])
