"""Performance cases of the framework: what a user has it do, through its public entry points.

Six kinds of call, each over the sizes, precisions, force sets and options that are used:

  host       one iteration with the positions and velocities in host memory
             (Context.step_host), the call of a host that owns its container
  loop       the iterations of a LADDS-style host: integrate, burn-up removal,
             escape removal, conjunction scan, each a call of its own
  step       the device-resident loop (Context.step), then the state read back
  propagate  propagation without scans (Context.integrate), then the state
  scan       the conjunction scan of a state (Context.scan), fragment clouds in it
  adjoint    miss distances of conjunction pairs and their gradients

Populations are seeded draws of the benchmark's definitions: 0 (LEO debris),
2 (constellation shells and debris), 4 (dense small-debris shells).
"""
import math

import numpy as np
import torch

from ladds_b200 import capi

DEFAULT_SET = capi.KEP | capi.J2 | capi.C22 | capi.S22 | capi.SRP | capi.DRAG  # the default configuration's terms
FORCE_SETS = {"kepler_j2": capi.KEP | capi.J2, "default": DEFAULT_SET, "full": capi.PROP_ALL}
PRECISIONS = {"fp64": capi.PRECISION_FP64, "split": capi.PRECISION_SPLIT}
SCREENS = {"lists": capi.SCREEN_LISTS, "buffer": capi.SCREEN_BUFFER}


def listed():
    return [
        # the smallest call: one iteration of 10,000 objects whose arrays a host container owns (the
        # CPU-runnable workload of the tests: central body + J2); latency and launches count
        {"name": "host_10k", "kind": "host", "population": 0, "n": 10_000, "forces": "kepler_j2",
         "precision": "fp64", "pinned": False, "threshold": 0.1},
        # the same call at the benchmark's size with pinned arrays (its end-to-end form)
        {"name": "host_1m", "kind": "host", "population": 0, "n": 1_000_000, "forces": "full",
         "precision": "split", "pinned": True, "threshold": 0.1},
        # the hot-path loop of a host program, a few iterations per visit of its output routine; the
        # default configuration
        {"name": "loop_100k", "kind": "loop", "population": 0, "n": 100_003, "forces": "default",
         "precision": "fp64", "steps": 4, "threshold": 0.1},
        # today's tracked catalogue, device resident, in the default configuration: many short iterations
        {"name": "step_30k", "kind": "step", "population": 0, "n": 30_011, "forces": "default",
         "precision": "fp64", "steps": 128, "every": 1, "cell": 0.0, "screen": "lists", "threshold": 1.0},
        # constellation shells in a debris background, scanned every fourth iteration
        {"name": "step_250k_every4", "kind": "step", "population": 2, "n": 250_000, "forces": "full",
         "precision": "fp64", "steps": 128, "every": 4, "cell": 0.0, "screen": "lists", "threshold": 0.5},
        # the benchmark's workload
        {"name": "step_1m", "kind": "step", "population": 0, "n": 1_000_000, "forces": "full",
         "precision": "split", "steps": 128, "every": 1, "cell": 0.0, "screen": "lists", "threshold": 1.0},
        # the benchmark's constellation workload
        {"name": "step_2m", "kind": "step", "population": 2, "n": 2_004_224, "forces": "full",
         "precision": "split", "steps": 48, "every": 1, "cell": 0.0, "screen": "lists", "threshold": 0.5},
        # the benchmark's scale workload, in the form its autotuner picks (40 km cells, buffer screening)
        {"name": "step_8m", "kind": "step", "population": 4, "n": 8_000_000, "forces": "full",
         "precision": "split", "steps": 32, "every": 1, "cell": 40.00004, "screen": "buffer", "threshold": 0.2},
        # propagation between rare scans: two hours in binary64
        {"name": "propagate_fp64", "kind": "propagate", "population": 0, "n": 200_000, "forces": "full",
         "precision": "fp64", "steps": 720},
        # the same in split precision at the benchmark's size
        {"name": "propagate_split", "kind": "propagate", "population": 0, "n": 1_000_000, "forces": "full",
         "precision": "split", "steps": 240},
        # the scan of a state with fragment clouds under spawn protection (crowded cells, long rows)
        {"name": "scan_clouds", "kind": "scan", "population": 4, "n": 500_000, "clouds": 6, "fragments": 15_000,
         "threshold": 5.0},
        # the benchmark's differentiation workload
        {"name": "adjoint_4096", "kind": "adjoint", "pairs": 4096, "steps": 1080, "checkpoint": 64},
    ]


def _log_int(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi], odd about as often as even."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("host", "loop", "step", "step", "step", "propagate", "propagate", "scan", "adjoint"))
    forces = rng.choice(("default", "full", "full", "kepler_j2"))
    precision = rng.choice(("fp64", "split"))
    population = rng.choice((0, 0, 2))
    if kind == "host":
        return {"kind": kind, "population": population, "n": _log_int(rng, 10_000, 1_000_000), "forces": forces,
                "precision": precision, "pinned": rng.random() < 0.5, "threshold": 0.1}
    if kind == "loop":
        return {"kind": kind, "population": population, "n": _log_int(rng, 10_000, 1_000_000), "forces": forces,
                "precision": precision, "steps": rng.randint(1, 6), "threshold": 0.1}
    if kind == "propagate":
        n = _log_int(rng, 10_000, 2_000_000)
        return {"kind": kind, "population": population, "n": n, "forces": forces, "precision": precision,
                "steps": _log_int(rng, 16, min(1000, 240_000_000 // n))}
    if kind == "scan":
        return {"kind": kind, "population": rng.choice((0, 4)), "n": _log_int(rng, 60_000, 1_000_000),
                "clouds": rng.randint(0, 6), "fragments": _log_int(rng, 500, 15_000), "threshold": 5.0}
    if kind == "adjoint":
        return {"kind": kind, "pairs": _log_int(rng, 64, 4096), "steps": rng.randint(90, 1080),
                "checkpoint": rng.choice((32, 64, 64, 128))}
    n = _log_int(rng, 10_000, 4_000_000)
    every = rng.choice((1, 1, 1, 2, 4, 10))
    dense = n >= 1_500_000 and rng.random() < 0.5
    return {"kind": "step", "population": 4 if dense else population, "n": n, "forces": forces,
            "precision": precision, "steps": _log_int(rng, 8, max(9, min(160, 120_000_000 // n))), "every": every,
            "cell": 40.00004 if dense else 0.0, "screen": "buffer" if dense else "lists",
            "threshold": 0.2 if dense else 0.5}


# ---------------------------------------------------------------- inputs


def _clouds(population, count, fragments, seed):
    """Fragment clouds appended to a population: `fragments` objects each around a point of an orbit through
    it, spread mostly along the track as after a few revolutions; one parent id per cloud."""
    rng = np.random.default_rng(seed)
    pop = {k: [v] for k, v in population.items()}
    n = len(population["x"])
    for c in range(count):
        a = 6378.137 + rng.uniform(700.0, 1200.0) + rng.normal(0.0, 12.0, fragments)
        u = rng.uniform(0.0, 2.0 * math.pi) + rng.normal(0.0, 0.05, fragments)
        inc = rng.uniform(0.3, math.pi - 0.3) + rng.normal(0.0, 0.004, fragments)
        raan = rng.uniform(0.0, 2.0 * math.pi) + rng.normal(0.0, 0.004, fragments)
        speed = np.sqrt(398600.4418 / a)
        cu, su, ci, si, co, so = np.cos(u), np.sin(u), np.cos(inc), np.sin(inc), np.cos(raan), np.sin(raan)
        r = np.stack([co * cu - so * su * ci, so * cu + co * su * ci, su * si])
        v = np.stack([-co * su - so * cu * ci, -so * su + co * cu * ci, cu * si])
        kick = rng.normal(0.0, 0.01, (3, fragments))
        radius = np.exp(rng.uniform(math.log(0.01), math.log(0.1), fragments))
        mass = 2700.0 * (4.0 / 3.0) * math.pi * radius**3
        new = {"radius": radius, "aom": math.pi * radius**2 * 1e-6 / mass, "bc_inv": 2.2 * math.pi * radius**2 / mass,
               "id": np.arange(n, n + fragments, dtype=np.uint64),
               "parent": np.full(fragments, c, dtype=np.uint64), "activity": np.zeros(fragments, dtype=np.int8)}
        for k in range(3):
            new["xyz"[k]] = a * r[k]
            new["v" + "xyz"[k]] = speed * v[k] + kick[k]
        for k, parts in pop.items():
            parts.append(new[k])
        n += fragments
    return {k: np.concatenate(v) for k, v in pop.items()}


def _config(case):
    """The configuration of a case's context.  The near-threshold flags are a diagnostic of comparisons between
    precisions and are off, as in a run that only wants its conjunctions."""
    return capi.default_config(
        componentMask=FORCE_SETS[case.get("forces", "full")], precision=PRECISIONS[case.get("precision", "fp64")],
        conjunctionThreshold=case.get("threshold", 0.1), nearThresholdRel=0.0,
        timestepsPerCollisionDetection=case.get("every", 1), cellSize=case.get("cell", 0.0),
        scanScreen=SCREENS[case.get("screen", "lists")])


def _population(case, seed):
    pop = capi.generate_population(case["population"], seed, case["n"])
    if case.get("clouds"):
        pop = _clouds(pop, case["clouds"], case["fragments"], seed)
    return pop


def _record_buffer(n):
    """Records that the caller makes room for: several times what a pass over n objects finds."""
    return 1 << 15 if n >= 400_000 else 1 << 13


def prepare(case, seed):
    """The context with its population (or the pairs of the adjoint) and the buffers that the caller keeps: the
    records and the state arrays (the state read back, or the one that a host program owns)."""
    ctx = capi.Context(_config(case))
    state = {"kind": case["kind"], "case": case, "ctx": ctx}  # ctx owns the device memory
    if case["kind"] == "adjoint":
        state["pairs"] = _pairs(case, seed)
        return state
    pop = _population(case, seed)
    ctx.upload(pop)
    n = len(pop["x"])
    state["records"] = np.zeros(_record_buffer(n), dtype=capi.PAIR_DTYPE)

    def array(values):
        if not case.get("pinned", True):
            return values.copy()
        t = torch.empty(n, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()
        t[:] = values
        return t

    fields = ("x", "y", "z", "vx", "vy", "vz")
    state["state"] = [array(pop[k]) for k in fields]
    if case["kind"] == "host":
        state["in"] = [array(pop[k]) for k in fields]
    return state


def _pairs(case, seed):
    """Conjunction pairs: B crosses A's orbit near A's position at a time inside the propagated span (both at the
    start of it by two-body motion, so the miss distances are some tens of kilometres at most)."""
    rng = np.random.default_rng(seed)
    n, dt, mu = case["pairs"], 10.0, 398600.4418
    a = 6378.137 + rng.uniform(500.0, 1500.0, n)
    meet = rng.uniform(0.2, 0.8, n) * case["steps"] * dt
    u0, inc, raan = rng.uniform(0, 2 * math.pi, n), rng.uniform(0.2, math.pi - 0.2, n), rng.uniform(0, 2 * math.pi, n)
    rate = np.sqrt(mu / a**3)

    def circular(u):
        cu, su, ci, si, co, so = np.cos(u), np.sin(u), np.cos(inc), np.sin(inc), np.cos(raan), np.sin(raan)
        r = np.stack([co * cu - so * su * ci, so * cu + co * su * ci, su * si], 1)
        v = np.stack([-co * su - so * cu * ci, -so * su + co * cu * ci, cu * si], 1)
        return a[:, None] * r, (a * rate)[:, None] * v

    rA, vA = circular(u0)
    at, vAt = circular(u0 + rate * meet)
    # B at the meeting point: A's radius vector, the velocity turned about it; back to the start by two-body motion
    turn = rng.uniform(0.3, math.pi, n)[:, None]
    h = np.cross(at / a[:, None], vAt)
    vB = np.cos(turn) * vAt + np.sin(turn) * h
    back = -(rate * meet)[:, None]
    speed = (a * rate)[:, None]
    rB = np.cos(back) * at + np.sin(back) * vB * (a[:, None] / speed)
    vB0 = -np.sin(back) * at * (speed / a[:, None]) + np.cos(back) * vB
    pairs = np.zeros(n, dtype=capi.ADJ_PAIR_DTYPE)
    pairs["rA"], pairs["vA"] = rA, vA
    pairs["rB"] = rB + rng.normal(0.0, 0.3, (n, 3))
    pairs["vB"] = vB0 + rng.normal(0.0, 1e-4, (n, 3))
    for side in "AB":
        radius = np.exp(rng.uniform(math.log(0.01), math.log(5.0), n))
        mass = 2700.0 * (4.0 / 3.0) * math.pi * radius**3
        pairs["bcInv" + side] = 2.2 * math.pi * radius**2 / mass
        pairs["aom" + side] = math.pi * radius**2 * 1e-6 / mass
    return pairs


# ---------------------------------------------------------------- calls


def _columns(records, state):
    """Conjunction records as plain arrays of the record buffer's length, zeros after the last record."""
    n, size = len(records), len(state["records"])
    out = {"count": n, "ids": np.zeros((2, size), dtype=np.int64), "slots": np.zeros((2, size), dtype=np.int64),
           "step": np.zeros(size, dtype=np.int64), "flags": np.zeros(size, dtype=np.int64),
           "dl2": np.zeros(size), "point": np.zeros((size, 3))}
    n = min(n, size)
    for k, side in enumerate("AB"):
        out["ids"][k, :n] = records["id" + side][:n]
        out["slots"][k, :n] = records["slot" + side][:n]
    for k in ("step", "flags", "dl2", "point"):
        out[k][:n] = records[k][:n]
    return out


def _read_state(ctx, arrays):
    """The population's positions and velocities into the caller's own (pinned) arrays."""
    code = capi.lib().ladds_gpu_get_state(ctx.handle, len(arrays[0]), *[a.ctypes.data for a in arrays])
    if code:
        raise capi.LaddsError(code, "get_state failed")
    return arrays


def run(state):
    case, ctx, kind = state["case"], state["ctx"], state["kind"]
    if kind == "host":
        res = ctx.step_host(state["in"], state["state"], out=state["records"])
        return {"records": _columns(res.records, state), "state": state["state"]}
    if kind == "loop":
        found, removed = [], 0
        params = _scan_params(case)
        for _ in range(case["steps"]):
            ctx.integrate(1, allow_nonfinite=True)
            removed += len(ctx.remove_below(150.0)) + len(ctx.remove_escaping())
            found.append(ctx.scan(params))
        return {"records": _columns(np.concatenate(found), state), "state": _read_state(ctx, state["state"]),
                "removed": removed}
    if kind == "step":
        res = ctx.step(case["steps"], out=state["records"])
        return {"records": _columns(res.records, state), "state": _read_state(ctx, state["state"])}
    if kind == "propagate":
        ctx.integrate(case["steps"])
        return {"state": _read_state(ctx, state["state"])}
    if kind == "scan":
        return {"records": _columns(ctx.scan(_scan_params(case)), state)}
    loss, miss, tca, _ = ctx.adjoint_forward(state["pairs"], case["steps"], case["checkpoint"])
    dx, dbc, _ = ctx.adjoint_backward()
    return {"loss": loss, "miss": miss, "tca": tca.astype(np.int64), "dx": dx, "dbc": dbc}


def _scan_params(case):
    return capi.ScanParams(cutoff=80.0, dt=10.0, collisionDistanceFactor=1.0, minDetectionRadius=0.05,
                           evasionCutoff=0.1, conjunctionThreshold=case["threshold"], nearThresholdRel=0.0)


def work(case):
    """Bytes: the state (position, velocity, two constants, tag) read once, positions and velocities written once;
    operations: the force evaluations (208 each for the full set) and the drift and kick updates of every step."""
    flops_eval = {"kepler_j2": 34, "default": 132, "full": 208}
    if case["kind"] == "adjoint":
        # forward: one sweep; gradient: the sweep again and its transpose, at least as many operations
        objects = 2 * case["pairs"]
        return {"bytes": case["pairs"] * (128 + 8 + 4 + 96 + 16), "flops": objects * case["steps"] * 3 * (3 * 208 + 42)}
    n = case["n"] + case.get("clouds", 0) * case.get("fragments", 0)
    if case["kind"] == "scan":
        return {"bytes": n * (68 + 24), "flops": n * 10}
    steps = case.get("steps", 1)
    return {"bytes": n * (68 + 48), "flops": n * steps * (3 * flops_eval[case["forces"]] + 42)}


# ---------------------------------------------------------------- 64-bit values
#
# The force model and the Yoshida-4 step in plain torch, every operation in binary64.

_MU, _RE, _J2, _J3 = 398600.4418, 6378.137, 1.08262668e-3, -2.53265649e-6
_C22, _S22 = 2.43938357328313e-6 * math.sqrt(5 / 12), -1.40027370385934e-6 * math.sqrt(5 / 12)
_MU_SUN, _MU_MOON, _AU, _P_SRP, _W = 1.32712440018e11, 4902.800066, 149597870.7, 4.56e-6, 7.292115146706979e-5
_JD = 2459580.5
_ATM = ((0, 1.225, 7.249), (25, 3.899e-2, 6.349), (30, 1.774e-2, 6.682), (40, 3.972e-3, 7.554),
        (50, 1.057e-3, 8.382), (60, 3.206e-4, 7.714), (70, 8.770e-5, 6.549), (80, 1.905e-5, 5.799),
        (90, 3.396e-6, 5.382), (100, 5.297e-7, 5.877), (110, 9.661e-8, 7.263), (120, 2.438e-8, 9.473),
        (130, 8.484e-9, 12.636), (140, 3.845e-9, 16.149), (150, 2.070e-9, 22.523), (180, 5.464e-10, 29.740),
        (200, 2.789e-10, 37.105), (250, 7.248e-11, 45.546), (300, 2.418e-11, 53.628), (350, 9.518e-12, 53.298),
        (400, 3.725e-12, 58.515), (450, 1.585e-12, 60.828), (500, 6.967e-13, 63.822), (600, 1.454e-13, 71.835),
        (700, 3.614e-14, 88.667), (800, 1.170e-14, 124.64), (900, 5.245e-15, 181.05), (1000, 3.019e-15, 268.00))


def _ephemeris(tau):
    """Sun and Moon positions [km] and the Earth rotation angle tau seconds after the epoch."""
    deg, arc = math.pi / 180, math.pi / (180 * 3600)
    T = (_JD + tau / 86400.0 - 2451545.0) / 36525.0
    ce, se = math.cos(23.43929111 * deg), math.sin(23.43929111 * deg)
    s, c = math.sin, math.cos
    M = (357.5256 + 35999.049 * T) * deg
    lam = 282.94 * deg + M + (6892.0 * s(M) + 72.0 * s(2 * M)) * arc
    r = (149.619 - 2.499 * c(M) - 0.021 * c(2 * M)) * 1e6
    sun = (r * c(lam), r * s(lam) * ce, r * s(lam) * se)
    L0 = (218.31617 + 481267.88088 * T - 1.3972 * T) * deg
    el, lp = (134.96292 + 477198.86753 * T) * deg, (357.52543 + 35999.04944 * T) * deg
    F, D = (93.27283 + 483202.01873 * T) * deg, (297.85027 + 445267.11135 * T) * deg
    dl = (22640 * s(el) + 769 * s(2 * el) - 4586 * s(el - 2 * D) + 2370 * s(2 * D) - 668 * s(lp) - 412 * s(2 * F)
          - 212 * s(2 * el - 2 * D) - 206 * s(el + lp - 2 * D) + 192 * s(el + 2 * D) - 165 * s(lp - 2 * D)
          + 148 * s(el - lp) - 125 * s(D) - 110 * s(el + lp) - 55 * s(2 * F - 2 * D))
    lam = L0 + dl * arc
    beta = (18520 * s(F + lam - L0 + (412 * s(2 * F) + 541 * s(lp)) * arc) - 526 * s(F - 2 * D)
            + 44 * s(el + F - 2 * D) - 31 * s(-el + F - 2 * D) - 25 * s(-2 * el + F) - 23 * s(lp + F - 2 * D)
            + 21 * s(-el + F) + 11 * s(-lp + F - 2 * D)) * arc
    r = (385000 - 20905 * c(el) - 3699 * c(2 * D - el) - 2956 * c(2 * D) - 570 * c(2 * el) + 246 * c(2 * el - 2 * D)
         - 205 * c(lp - 2 * D) - 171 * c(el + 2 * D) - 152 * c(el + lp - 2 * D))
    x, y, z = r * c(beta) * c(lam), r * c(beta) * s(lam), r * s(beta)
    moon = (x, y * ce - z * se, y * se + z * ce)
    T0 = (_JD - 2451545.0) / 36525.0
    gmst = 67310.54841 + (876600.0 * 3600.0 + 8640184.812866) * T0 + 0.093104 * T0 * T0 - 6.2e-6 * T0**3
    gmst = math.fmod(gmst, 86400.0)
    theta = (gmst + (86400.0 if gmst < 0 else 0.0)) * (2 * math.pi / 86400.0) + _W * tau
    return sun, moon, theta


def _third_body(r, body, mu):
    s = torch.tensor(body, dtype=r.dtype, device=r.device)[:, None]
    d = s - r
    return mu * (d / (d * d).sum(0) ** 1.5 - s / (s * s).sum() ** 1.5)


def _acceleration(mask, r, v, aom, bc, tau, atm):
    """Acceleration of the objects at the columns of r and v (3 x n)."""
    sun, moon, theta = _ephemeris(tau)
    x, y, z = r
    r2 = (r * r).sum(0)
    inv2 = 1.0 / r2
    rn = torch.sqrt(r2)
    zero = torch.zeros_like(x)
    a = torch.zeros_like(r)
    if mask & capi.KEP:
        a = a - _MU * inv2 / rn * r
    if mask & capi.J2:
        k, q = -1.5 * _J2 * _MU * _RE**2 * inv2 * inv2 / rn, 5.0 * z * z * inv2
        a = a + k * r * torch.stack([1.0 - q, 1.0 - q, 3.0 - q])
    if mask & capi.J3:
        k, f = -2.5 * _J3 * _MU * _RE**3 * inv2**3 / rn, 3.0 * z - 7.0 * z**3 * inv2
        a = a + k * torch.stack([x * f, y * f, 6.0 * z * z - 7.0 * z**4 * inv2 - 0.6 * r2])
    if mask & (capi.C22 | capi.S22):
        C, S = (_C22 if mask & capi.C22 else 0.0), (_S22 if mask & capi.S22 else 0.0)
        c, s = math.cos(theta), math.sin(theta)
        xf, yf = c * x + s * y, c * y - s * x
        g, k = C * (xf * xf - yf * yf) + 2.0 * S * xf * yf, 3.0 * _MU * _RE**2 * inv2 * inv2 / rn
        ax = k * (2.0 * (C * xf + S * yf) - 5.0 * g * xf * inv2)
        ay = k * (2.0 * (S * xf - C * yf) - 5.0 * g * yf * inv2)
        a = a + torch.stack([c * ax - s * ay, s * ax + c * ay, -5.0 * k * g * z * inv2])
    if mask & capi.SOL:
        a = a + _third_body(r, sun, _MU_SUN)
    if mask & capi.LUN:
        a = a + _third_body(r, moon, _MU_MOON)
    if mask & capi.SRP:
        s = torch.tensor(sun, dtype=r.dtype, device=r.device)[:, None]
        u = r - s
        along = (r * s).sum(0) / math.sqrt(sum(t * t for t in sun))
        lit = ~((along < 0) & (r2 - along * along < _RE**2))
        a = a + torch.where(lit, 1e3 * _P_SRP * _AU**2 * aom * (u * u).sum(0) ** -1.5, zero) * u
    if mask & capi.DRAG:
        w = torch.stack([v[0] + _W * y, v[1] - _W * x, v[2]])
        h = rn - _RE
        band = (torch.searchsorted(atm[:, 0].contiguous(), h.detach(), right=True) - 1).clamp(min=0)
        base, rho0, scale = atm[band].T
        a = a - 0.5e3 * rho0 * torch.exp((base - h) / scale) * bc * torch.sqrt((w * w).sum(0)) * w
    return a


def _yoshida(mask, r, v, aom, bc, start, steps, atm, dt=10.0):
    """`steps` steps from iteration `start`; yields the state after each."""
    c1, c2, d1, d2 = 0.6756035959798288, -0.17560359597982883, 1.3512071919596575, -1.7024143839193153
    for i in range(start, start + steps):
        tau = i * dt
        for c, d in ((c1, d1), (c2, d2), (c2, d1)):
            tau += c * dt
            r = r + c * dt * v
            v = v + d * dt * _acceleration(mask, r, v, aom, bc, tau, atm)
        r = r + c1 * dt * v
        yield r, v


def _miss(rA, vA, rB, vB, dt=10.0):
    """Squared distance and point (of B, and the offset to A) of the closest approach of two segments that end at
    (r, v)."""
    oA, oB = rA - vA * dt, rB - vB * dt
    o, w = oA - oB, vA - vB
    t = (-(o * w).sum(0) / (w * w).sum(0)).clamp(0.0, dt)
    d = o + w * t
    return (d * d).sum(0), oB + vB * t + 0.5 * d


def _tensors(*arrays):
    where = "cuda" if torch.cuda.is_available() else "cpu"
    return [torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device=where) for x in arrays]


def _exact_records(pop, r, v, case):
    """The conjunctions of a state by testing every pair (passive objects without parents)."""
    n, found = r.shape[1], []
    radius = torch.as_tensor(pop["radius"], dtype=torch.float64, device=r.device)
    for i in range(0, n, 1024):
        A = torch.arange(i, min(i + 1024, n), device=r.device)
        d2 = sum((r[k, A, None] - r[k, None, :]) ** 2 for k in range(3))
        a, b = torch.nonzero((d2 <= 6400.0) & (A[:, None] < torch.arange(n, device=r.device)), as_tuple=True)
        a = A[a]
        dl2, point = _miss(r[:, a], v[:, a], r[:, b], v[:, b])
        limit = torch.maximum(torch.tensor(case["threshold"] ** 2, device=r.device, dtype=r.dtype),
                              ((radius[a] + radius[b]) / 1000.0) ** 2)
        keep = dl2 <= limit
        found.append((dl2[keep], point[:, keep]))
    dl2, point = torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found], 1).T
    size = _record_buffer(n)
    return (torch.nn.functional.pad(dl2, (0, size - len(dl2))),
            torch.nn.functional.pad(point, (0, 0, 0, size - len(dl2))))


def _exact_adjoint(case, seed, atm, dt=10.0, segment=24):
    p = _pairs(case, seed)
    n, steps, mask = case["pairs"], case["steps"], capi.PROP_ALL
    r, v, aom, bc = _tensors(np.concatenate([p["rA"], p["rB"]]).T, np.concatenate([p["vA"], p["vB"]]).T,
                             np.concatenate([p["aomA"], p["aomB"]]), np.concatenate([p["bcInvA"], p["bcInvB"]]))
    best = torch.full((n,), math.inf, dtype=torch.float64, device=r.device)
    arg = torch.zeros(n, dtype=torch.int64, device=r.device)
    marks = []
    with torch.no_grad():
        for s, (r1, v1) in enumerate(_yoshida(mask, r, v, aom, bc, 0, steps, atm)):
            if s % segment == 0:
                marks.append((s, r, v))
            r, v = r1, v1
            d2, _ = _miss(r[:, :n], v[:, :n], r[:, n:], v[:, n:])
            arg = torch.where(d2 < best, s + 1, arg)
            best = torch.minimum(best, d2)
    gr, gv, gb = torch.zeros_like(r), torch.zeros_like(v), torch.zeros_like(bc)
    for s, r0, v0 in reversed(marks):
        r0, v0, b0 = (t.detach().requires_grad_() for t in (r0, v0, bc))
        total = 0.0
        for k, (r, v) in enumerate(_yoshida(mask, r0, v0, aom, b0, s, min(segment, steps - s), atm)):
            here = torch.nonzero(arg == s + k + 1)[:, 0]
            if len(here):
                d2, _ = _miss(r[:, here], v[:, here], r[:, n + here], v[:, n + here])
                total = total + d2.sum()
        total = total + (gr * r).sum() + (gv * v).sum()
        gr, gv, more = torch.autograd.grad(total, (r0, v0, b0))
        gb = gb + more
    dx = torch.cat([gr[:, :n], gv[:, :n], gr[:, n:], gv[:, n:]]).T
    return {"loss": best.sum(), "miss": best, "tca": None, "dx": dx, "dbc": torch.stack([gb[:n], gb[n:]], 1)}


def exact(case, seed):
    """States in 64 bits for every kind that propagates, miss distances and points of the conjunctions where every
    pair can be tested, and the adjoint's loss and gradients."""
    atm, = _tensors(np.array(_ATM))
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed, atm)
    if case["kind"] == "scan":
        return None
    pop = _population(case, seed)
    r, v, aom, bc = _tensors(np.stack([pop["x"], pop["y"], pop["z"]]), np.stack([pop["vx"], pop["vy"], pop["vz"]]),
                             pop["aom"], pop["bc_inv"])
    mask = FORCE_SETS[case["forces"]]
    for r, v in _yoshida(mask, r, v, aom, bc, 0, case.get("steps", 1), atm):
        pass
    out = {"state": [*r, *v]}
    if case["kind"] != "propagate":
        out["records"] = {k: None for k in ("count", "ids", "slots", "step", "flags", "dl2", "point")}
    if case["kind"] == "loop":
        out["removed"] = None
    if case["kind"] == "host" and case["population"] == 0 and case["n"] <= 100_000:
        out["records"]["dl2"], out["records"]["point"] = _exact_records(pop, r, v, case)
    return out
