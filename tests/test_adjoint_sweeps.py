"""The adjoint's sweeps where they can go wrong: batches of three steps that do
not fill, blocks of 16 pairs and their remainders, component masks with and
without kernels of their own, and the reverse sweep over segments that is taken
when the records of a whole sweep are too large to be kept."""
import numpy as np
import pytest

from test_adjoint import DT, capi, oracle_pairs, pairs16, rel_norm, tangent_gradient, to_records  # noqa: F401


@pytest.mark.gpu
@pytest.mark.parametrize("mask", ["full", "default", "kepler_j2", "full_without_drag", "full_without_sun"])
@pytest.mark.parametrize("n,steps,ck", [(1, 1, 1), (1, 2, 64), (16, 3, 2), (17, 4, 3), (33, 16, 5), (17, 35, 64)])
def test_sweeps_of_masks(capi, oracle, mask, n, steps, ck):  # noqa: F811
    """Against the oracle's tangent-linear gradient.  The misses are 50 m to 2 km,
    the positions' rounding over these steps below 1e-10 km, so relative
    errors are below 1e-8; the bound is ten times that."""
    A = capi.PROP_ALL
    bits = {"full": A, "default": capi.KEP | capi.J2 | capi.C22 | capi.S22 | capi.SRP | capi.DRAG,
            "kepler_j2": capi.KEP | capi.J2, "full_without_drag": A & ~capi.DRAG, "full_without_sun": A & ~capi.SOL}[mask]
    rows = oracle_pairs(oracle, n, steps, seed=100 * n + steps)
    with capi.Context(capi.default_config(componentMask=bits, deltaT=DT)) as ctx:
        _, miss, step, _ = ctx.adjoint_forward(to_records(rows, capi), steps, ck)
        dx, dbc, _ = ctx.adjoint_backward()
    ref, at, _ = oracle.pair_losses(rows, steps, dt=DT, mask=bits)
    assert np.array_equal(step, at)
    assert np.max(np.abs(miss - ref)) <= 1e-7 * np.max(ref)
    g = tangent_gradient(oracle, rows, steps, bits)
    assert np.all(rel_norm(dx, g[:, :12]) < 1e-7)
    assert np.max(np.abs(dbc - g[:, 12:])) <= 1e-7 * max(np.max(np.abs(g[:, 12:])), 1e-30)


@pytest.mark.gpu
@pytest.mark.parametrize("ck", [100, 333])
def test_segments_equal_the_whole_sweep(capi, ck):  # noqa: F811
    """1400 steps of 4096 pairs go by segments, those of a few pairs in one
    sweep: the same kernels over the same records, so equal to the bit."""
    steps = 1400
    with capi.Context(capi.default_config(componentMask=capi.PROP_ALL)) as ctx:
        pairs, _ = ctx.adjoint_make_pairs(3, 4096, steps)
        _, miss, step, _ = ctx.adjoint_forward(pairs, steps, ck)
        dx, dbc, _ = ctx.adjoint_backward()
        for part in (slice(0, 16), slice(4079, 4096)):
            _, m, s, _ = ctx.adjoint_forward(pairs[part].copy(), steps, ck)
            gx, gb, _ = ctx.adjoint_backward()
            assert np.array_equal(m, miss[part]) and np.array_equal(s, step[part])
            assert np.array_equal(gx, dx[part]) and np.array_equal(gb, dbc[part])
