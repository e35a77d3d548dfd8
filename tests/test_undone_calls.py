"""A call that is undone -- its records do not fit the caller's buffer -- leaves the
population as it was: states, iteration and the order in which records leave."""
import ctypes

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


@pytest.mark.parametrize("every", [1, 4, 33])
@pytest.mark.parametrize("pair_capacity", [0, 1])
@pytest.mark.parametrize("undone", [1, 3, 40, 150])
def test_undone_step_keeps_the_order(capi, every, pair_capacity, undone):
    """Calls of one launch and of several, in graphs and launched one by one, with device
    buffers that hold the records and that overflow in the undone call first; each
    from two of the ring's buffers and both sort sets."""
    import torch

    n = 3001
    pop = capi.generate_population(0, 5, n)
    cfg = capi.default_config(componentMask=capi.PROP_ALL, timestepsPerCollisionDetection=every,
                              conjunctionThreshold=70.0, pairCapacity=pair_capacity)
    buf = torch.zeros(n * capi.STATE_RECORD_DTYPE.itemsize, dtype=torch.uint8, device="cuda")

    def packed(ctx):
        assert ctx.pack_layers(0, ctx.grid()[0][2], False, buf, n) == n
        return buf.cpu().numpy().tobytes()

    with capi.Context(cfg) as ctx:
        ctx.upload(pop)
        ctx.conjunctions(10.0)
        ctx.integrate(50)  # the order of the scan is not that of the state any more
        for _ in range(3):
            before, it = packed(ctx), ctx.iteration()
            ids = np.frombuffer(before, dtype=capi.STATE_RECORD_DTYPE)["id"]
            assert not np.array_equal(ids, np.sort(ids))
            got, stats = ctypes.c_size_t(), capi.StepStats()
            rc = capi.lib().ladds_gpu_step(ctx.handle, undone, None, 0, ctypes.byref(got), ctypes.byref(stats))
            scans = sum((it + i) % every == 0 for i in range(undone))
            assert (rc == capi.ERR_CAPACITY and got.value > 0) if scans else rc == 0
            if scans:
                assert ctx.iteration() == it
                assert packed(ctx) == before
            else:
                order = np.frombuffer(packed(ctx), dtype=capi.STATE_RECORD_DTYPE)["id"]
                assert np.array_equal(order, ids)
            ctx.step(every + 1)
