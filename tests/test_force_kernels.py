"""Force kernels on the GPU: the density table of the FP64 drag term at its
bins' and bands' edges and outside it, and the kernels compiled for a component
mask against the oracle and against each other."""
import numpy as np
import pytest

from helpers import to_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ladds_b200 import build, capi

    build.build_gpu()
    return capi


def at_altitudes(h, bc):
    n = len(h)
    one = np.ones(n)
    return dict(x=6378.137 + h, y=0 * one, z=0 * one, vx=0 * one, vy=7.0 * one, vz=0.5 * one, radius=0.1 * one,
                aom=1e-9 * one, bc_inv=bc * one, id=np.arange(n, dtype=np.uint64))


def test_density_table_edges(capi, oracle):
    """One step of 1 s with the drag at most 0.1 km/s^2 (the oracle's bands and
    exponential): below the table, every band edge and some bins from both sides,
    the middle of bins, the table's end at 2048 km and beyond.  The stage
    altitudes lie metres above those set, so no stage sits on an edge.  1e-9 km: the
    bound of a single FP64 step elsewhere in the suite; a density off by 1e-8
    would pass it at the lowest altitudes only if the drag were a tenth of this."""
    edges = np.array([0, 25, 30, 40, 50, 60, 70, 80, 90, 100, 110, 120, 130, 140, 150, 180, 200, 250, 300, 350, 400,
                      450, 500, 600, 700, 800, 900, 1000, 1001, 1500, 2047, 2048], dtype=float)
    h = np.concatenate([edges - 0.01, edges + 1e-6, edges + 0.5, [-5.0, -0.5, 2047.99, 5000.0]])
    rho = 1.225 * np.exp(-np.maximum(h, 0.0) / 8.0)
    pop = at_altitudes(h, np.minimum(0.02, 0.1 / (0.5e3 * rho * 50.0)))
    with capi.Context(capi.default_config(componentMask=capi.KEP | capi.DRAG, deltaT=1.0)) as ctx:
        ctx.upload(pop)
        ctx.integrate(1)
        got = ctx.get_state()
    from ladds_b200.population import as_population

    ref, moved = (to_oracle(oracle, {k: v.copy() for k, v in as_population(pop).items()}) for _ in range(2))
    oracle.propagate(ref, oracle.KEP | oracle.DRAG, 1.0, 1)
    oracle.propagate(moved, oracle.KEP, 1.0, 1)  # without the drag
    assert np.max(np.abs(ref.vy - moved.vy)) > 0.05  # the drag matters here
    for g, r in zip(got, (ref.x, ref.y, ref.z, ref.vx, ref.vy, ref.vz)):
        assert np.max(np.abs(g - r)) < 1e-9


@pytest.mark.parametrize("mask", ["full", "default", "full_without_moon", "j2_drag"])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 257, 1000])
def test_mask_kernels(capi, oracle, mask, precision, n):
    """Masks with and without a kernel of their own: 20 steps against the oracle,
    and the propagation before a scan against the multi-step kernel bit for bit."""
    m = dict(full=capi.PROP_ALL, default=capi.default_config().componentMask,
             full_without_moon=capi.PROP_ALL & ~capi.LUN, j2_drag=capi.KEP | capi.J2 | capi.DRAG)[mask]
    pop = capi.generate_population(0, 19, n)
    pop["activity"][::9] = capi.EVASIVE_PRESERVING
    states = []
    for steps in (1, 0):
        with capi.Context(capi.default_config(componentMask=m, precision=precision)) as ctx:
            ctx.upload(pop)
            if steps:
                for _ in range(20):
                    ctx.step(1)
            else:
                ctx.integrate(20)
            states.append(ctx.get_state())
    for a, b in zip(*states):
        assert np.array_equal(a, b)
    ref = to_oracle(oracle, pop)
    oracle.propagate(ref, m, 10.0, 20)
    for g, r in zip(states[1], (ref.x, ref.y, ref.z)):
        assert np.max(np.abs(g - r)) < (1e-9 if precision == 0 else 1e-6)


@pytest.mark.parametrize("mask", ["kepler", "full"])
def test_reciprocal_roots_over_their_range(capi, oracle, mask):
    """Distances from 100 km to 1e7 km and air-relative speeds down to a standstill
    (where the drag's root has no argument): one step of 1 s against the oracle.  1e-9 km and
    a few units in the last place of the largest positions."""
    bits = capi.KEP if mask == "kepler" else capi.PROP_ALL
    radius = np.concatenate([np.geomspace(1e2, 1e7, 241) if mask == "kepler" else np.geomspace(6500.0, 1e7, 241)])
    n = len(radius)
    pop = at_altitudes(radius - 6378.137, 0.01)
    pop["vy"] = np.where(np.arange(n) % 3 == 0, 7.292115146706979e-5 * radius, np.sqrt(398600.4418 / radius))
    pop["vz"] = 0.0 * radius
    with capi.Context(capi.default_config(componentMask=bits, deltaT=1.0)) as ctx:
        ctx.upload(pop)
        ctx.integrate(1)
        got = ctx.get_state()
    from ladds_b200.population import as_population

    ref = to_oracle(oracle, {k: v.copy() for k, v in as_population(pop).items()})
    oracle.propagate(ref, bits, 1.0, 1)
    for g, r in zip(got, (ref.x, ref.y, ref.z, ref.vx, ref.vy, ref.vz)):
        assert np.all(np.abs(g - r) < 1e-9 + 4e-15 * radius)
