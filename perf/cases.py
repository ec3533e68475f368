"""Performance cases of the propagation and closest-approach library.

Each case is one piece of work a program gives the Python binding (opengpop_b200): propagation
calls from one object to a whole catalogue, uneven request batches, trajectories, closest-approach
jobs, state transition matrices, miss-distance gradients and plain force evaluations.

listed() are the fixed cases and draw() makes more of the same ranges; prepare() builds what a
program holds before the call (context, states), run() makes the call, work() counts what it
cannot do without and exact() gives 64-bit values in plain torch where there are such values.
"""
import math
import os

import numpy as np
import torch

import opengpop_b200 as G
from opengpop_b200 import orbits

START = orbits.EPOCH
DEV = "cuda:0"


def listed():
    return [
        # one satellite's owner asks for the next hour: the smallest call, all latency
        dict(name="one_object_1h", kind="propagate", n=1, degree=70, h=30.0, steps=120, mixed=False, mix=False),
        # the 1,024-object, 20x20, 60 s, 24 h configuration: a constellation for a day
        dict(name="constellation_20x20_24h", kind="propagate", n=1024, degree=20, h=60.0, steps=1440, mixed=False,
             mix=False),
        # an odd-sized LEO catalogue already on the device, plain FP64 at full degree
        dict(name="catalogue_fp64", kind="device", n=18501, degree=70, h=30.0, steps=240, mixed=False, mix=False),
        # a fragment cloud's part of a catalogue: mixed precision, middle degree, longer step
        dict(name="subset_mixed_36x36", kind="device", n=24001, degree=36, h=60.0, steps=240, mixed=True, mix=True),
        # the 65,536-object mixed-precision configuration (LEO, MEO, GEO), host arrays in and out
        dict(name="population_mixed", kind="propagate", n=65536, degree=70, h=30.0, steps=320, mixed=True, mix=True),
        # ephemeris generation: every step's position, velocity and acceleration kept
        dict(name="ephemeris", kind="trajectory", n=3000, degree=50, h=30.0, steps=360, mixed=False, mix=True),
        # a propagation service's queue: uneven requests, one launch
        dict(name="request_batch", kind="batch", n=256, degree=0, h=0.0, days=1.0, shapes=20240101, mixed=True,
             mix=True),
        # covariance propagation: 6x6 state transition matrices over three hours
        dict(name="transition_matrices", kind="stm", n=1000, degree=70, h=30.0, steps=360, mixed=False, mix=False),
        # manoeuvre planning: gradients of the miss distance of listed pairs over six hours
        dict(name="miss_gradients", kind="miss", n=1200, degree=70, h=30.0, steps=720, mixed=False, mix=False),
        # conjunction assessment: a tenth of a catalogue against all of it over one day
        dict(name="conjunctions_1d", kind="approach", n=2500, degree=70, h=30.0, steps=2880, mixed=False, mix=False,
             threshold=20e3),
        # the screen alone over ephemerides of another propagator, two fleets against each other
        dict(name="screen_ephemerides", kind="screen", n=6000, degree=4, h=30.0, steps=720, mixed=False, mix=False,
             threshold=10e3),
        # force evaluations for a caller's own integrator: acceleration and its Jacobian
        dict(name="force_and_jacobian", kind="force", n=100003, degree=70, h=0.0, steps=1, mixed=False, mix=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["propagate", "propagate", "device", "device", "trajectory", "batch", "stm", "miss",
                       "approach", "screen", "force"])
    degree = rng.choice([8, 20, 36, 50, 70, 70])
    h = rng.choice([10.0, 30.0, 30.0, 60.0])
    mixed = rng.random() < 0.5
    mix = rng.random() < 0.5
    if kind in ("propagate", "device"):
        n = _log(rng, 1, 65536)
        return dict(kind=kind, n=n, degree=degree, h=h, steps=_log(rng, 30, 1500 if n < 3000 else 300), mixed=mixed,
                    mix=mix)
    if kind == "trajectory":
        n = _log(rng, 1, 8000)
        return dict(kind=kind, n=n, degree=degree, h=h, steps=_log(rng, 30, 400), mixed=mixed, mix=mix)
    if kind == "batch":
        return dict(kind=kind, n=_log(rng, 2, 300), degree=0, h=0.0, days=rng.uniform(0.3, 1.0),
                    shapes=rng.randrange(1 << 30), mixed=mixed, mix=True)
    if kind == "stm":
        return dict(kind=kind, n=_log(rng, 1, 2000), degree=degree, h=h, steps=_log(rng, 30, 360), mixed=False, mix=mix)
    if kind == "miss":
        return dict(kind=kind, n=_log(rng, 1, 1500), degree=degree, h=30.0, steps=_log(rng, 200, 720), mixed=False,
                    mix=False)
    if kind == "approach":
        n = _log(rng, 20, 2500)  # few objects come near each other only in a wider sense
        return dict(kind=kind, n=n, degree=degree, h=30.0, steps=_log(rng, 200, 2000), mixed=mixed, mix=False,
                    threshold=min(2000e3, 50e6 / n))
    if kind == "screen":
        n = _log(rng, 30, 6000)
        return dict(kind=kind, n=n, degree=4, h=30.0, steps=_log(rng, 60, 720), mixed=False, mix=False,
                    threshold=min(2000e3, 60e6 / n))
    return dict(kind=kind, n=_log(rng, 1, 200000), degree=degree, h=0.0, steps=1, mixed=mixed, mix=mix)


def _states(n, seed, mix):
    return orbits.mixed_population(n, seed) if mix and n >= 10 else orbits.leo(n, seed)


def _requests(case, seed):
    """The batch's shapes (from case["shapes"]) with states of `seed`."""
    g = np.random.default_rng(case["shapes"])
    s = np.random.default_rng(seed)
    out = []
    for _ in range(case["n"]):
        n = int(round(math.exp(g.uniform(0.0, math.log(512.0)))))
        h = float(g.choice([10.0, 30.0, 60.0, 120.0]))
        dur = case["days"] / 7.0 * math.exp(g.uniform(math.log(3600.0), math.log(7 * 86400.0)))
        degree = int(g.choice([8, 20, 36, 70]))
        out.append(dict(start=START, h=h, steps=max(1, int(round(dur / h))), degree=degree, n=n,
                        seed=int(s.integers(1 << 30))))
    return out


def _cuda(x):
    return torch.tensor(x, dtype=torch.float64, device=DEV)


def _fleet(case, seed):
    """Sampled two-body ephemerides r, v, a [steps][n][3] of case["n"] objects on the device."""
    g = np.random.default_rng(seed)
    n = case["n"]
    el = [g.uniform(6.8e6, 7.4e6, n), g.uniform(0.0, 0.02, n)] + [
        np.radians(g.uniform(0.0, top, n)) for top in (180.0, 360.0, 360.0, 360.0)]
    a, e, inc, raan, argp, m0 = (_cuda(x) for x in el)
    t = torch.arange(1, case["steps"] + 1, dtype=torch.float64, device=DEV)[:, None] * case["h"]
    M = m0 + torch.sqrt(orbits.GM / a ** 3) * t
    E = M.clone()
    for _ in range(8):
        E = E - (E - e * torch.sin(E) - M) / (1.0 - e * torch.cos(E))
    cE, sE, fac = torch.cos(E), torch.sin(E), torch.sqrt(1.0 - e * e)
    x, y, rn = a * (cE - e), a * fac * sE, a * (1.0 - e * cE)
    vs = torch.sqrt(orbits.GM * a) / rn
    vx, vy = -vs * sE, vs * fac * cE
    cO, sO, cw, sw, ci, si = (f(z) for z in (raan, argp, inc) for f in (torch.cos, torch.sin))
    p = torch.stack([cO * cw - sO * sw * ci, sO * cw + cO * sw * ci, sw * si], -1)
    q = torch.stack([-cO * sw - sO * cw * ci, -sO * sw + cO * cw * ci, cw * si], -1)
    r = x[..., None] * p + y[..., None] * q
    v = vx[..., None] * p + vy[..., None] * q
    return r, v, -orbits.GM * r / (rn ** 3)[..., None]


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, kind, n = case, case["kind"], case["n"]
    s.ctx = G.Context(gravity_degree=case["degree"], precision=G.MIXED if case["mixed"] else G.FP64)
    if kind == "batch":
        s.reqs = []
        for q in _requests(case, seed):
            r, v = _states(q["n"], q["seed"], True)
            s.reqs.append(dict(start=q["start"], h=q["h"], steps=q["steps"], degree=q["degree"], r=r, v=v))
    elif kind == "miss":
        s.r, s.v, s.pairs = orbits.conjunction_pairs(n, seed)
    elif kind == "screen":
        s.tr, s.tv, s.ta = _fleet(case, seed)
        s.sets = (np.arange(n) >= n // 2).astype(np.uint32)
    elif kind == "approach":
        s.r, s.v = _states(n, seed, False)
        k = max(1, n // 10)
        s.sets = np.minimum(np.arange(n), k).astype(np.uint32)  # k single objects, then all the others
    else:
        s.r, s.v = _states(n, seed, case["mix"])
        if kind in ("device", "trajectory", "force"):
            s.r, s.v = _cuda(s.r), _cuda(s.v)
    return s


ROWS = 4096  # rows of a program's record buffers


def _records(recs, n=ROWS):
    """The records in fixed buffers, zero past the last record."""
    out = dict(count=len(recs), pair=np.zeros((n, 2), np.int64), distance=np.zeros(n), time=np.zeros(n),
               position_a=np.zeros((n, 3)), position_b=np.zeros((n, 3)))
    for i, q in enumerate(recs[:n]):
        out["pair"][i] = q.object_index1, q.object_index2
        out["distance"][i], out["time"][i] = q.distance, q.time
        out["position_a"][i], out["position_b"][i] = q.position_a, q.position_b
    return out


def run(s):
    c, ctx = s.case, s.ctx
    kind, h, steps, n = c["kind"], c["h"], c.get("steps", 0), c["n"]
    if kind == "propagate":
        return ctx.propagate(START, h, steps, s.r, s.v)
    if kind == "device":
        r, v = s.r.clone(), s.v.clone()
        ctx.propagate_device(START, h, steps, r, v)
        return r, v
    if kind == "trajectory":
        r, v = s.r.clone(), s.v.clone()
        out = [torch.empty(steps, 3, n, dtype=torch.float64, device=DEV) for _ in range(3)]
        ctx.propagate_trajectory(START, h, steps, r, v, *out)
        return r, v, out
    if kind == "batch":
        return [np.concatenate(x) for x in zip(*ctx.propagate_batch(s.reqs))]
    if kind == "stm":
        return ctx.stm(START, h, steps, s.r, s.v)
    if kind == "miss":
        return ctx.miss_gradient(START, h, steps, s.r, s.v, s.pairs)
    if kind == "approach":
        ca = ctx.closest_approach(START, h, s.r, s.v, s.sets)
        ca.propagate(steps)
        recs = _records(ca.find(c["threshold"]))
        ca.close()
        return recs
    if kind == "screen":
        # the objects' first states come from the ephemerides' owner, on the host
        zero = np.ones((n, 3))
        ca = ctx.closest_approach(None, h, zero, zero, s.sets, kind="external")
        ca.reserve(steps)
        ca.append(steps, s.tr, s.tv, s.ta)
        recs = _records(ca.find(c["threshold"]))
        ca.close()
        return recs
    acc = torch.empty_like(s.r)
    jac = torch.empty(n, 3, 3, dtype=torch.float64, device=DEV)
    ctx.gravity(s.r, acc)
    ctx.gravity_jacobian(s.r, jac)
    return acc, jac


# ---- what a pass cannot do without ----
# One gravity evaluation: per (n, m) term the two-term recursion (3 operations) and six sums, FMA =
# 2 flops; per column the cos/sin recursion and the combination.
def _evaluation(L):
    return 24 * max(0, (L + 1) * (L + 2) // 2 - 3) + 15 * L + 60


def _jacobian(L):
    return 44 * max(0, (L + 1) * (L + 2) // 2 - 3) + 100 * (L + 1) + 200


# Evaluations at distinct positions of one step: the corrector of a 10-60 s step stands still in 64
# bits after three.
EVALS = 3
STARTUP_EVALS = 80 + 9 + 8 * EVALS


def _propagation(n, steps, L):
    return float(n) * (steps * (EVALS * _evaluation(L) + 500) + STARTUP_EVALS * _evaluation(L))


def work(case):
    kind, n, L, steps = case["kind"], case["n"], case["degree"], case.get("steps", 0)
    state = 96.0 * n  # position and velocity in, position and velocity out
    if kind in ("propagate", "device"):
        return dict(bytes=state, flops=_propagation(n, steps, L))
    if kind == "trajectory":
        return dict(bytes=state + 72.0 * n * steps, flops=_propagation(n, steps, L))
    if kind == "batch":
        reqs = _requests(case, 0)
        return dict(bytes=sum(96.0 * q["n"] for q in reqs),
                    flops=sum(_propagation(q["n"], q["steps"], q["degree"]) for q in reqs))
    if kind == "stm":
        extra = n * (steps + STARTUP_EVALS) * (_jacobian(L) + 6 * 150.0)
        return dict(bytes=state + 288.0 * n, flops=_propagation(n, steps, L) + extra)
    if kind == "miss":  # propagation, the pairs' minimum, then one Jacobian per step of either object
        u = 2 * n
        extra = u * (steps + STARTUP_EVALS) * (_jacobian(L) + 300.0) + 9.0 * n * steps
        return dict(bytes=48.0 * u + 120.0 * n, flops=_propagation(u, steps, L) + extra)
    if kind == "approach":
        k = max(1, n // 10)
        pairs = k * (k - 1) / 2 + k * (n - k)
        return dict(bytes=48.0 * n, flops=_propagation(n, steps, L) + 9.0 * pairs * steps)
    if kind == "screen":
        k = n // 2
        return dict(bytes=72.0 * n * steps, flops=9.0 * k * (n - k) * steps)
    return dict(bytes=n * (48.0 + 24.0 + 72.0), flops=n * float(_evaluation(L) + _jacobian(L)))


# ---- 64-bit values without the library ----
def _field(L):
    """Fully normalised C, S up to degree L, GM and radius from the gravity file."""
    C, S = torch.zeros(L + 1, L + 1, dtype=torch.float64), torch.zeros(L + 1, L + 1, dtype=torch.float64)
    with open(os.path.join(G.DATA_DIR, "JGM3.gfc")) as f:
        for line in f:
            w = line.replace("D", "E").replace("d", "e").split() if line.startswith("gfc ") else line.split()
            if len(w) >= 2 and w[0] == "earth_gravity_constant":
                gm = float(w[1].replace("D", "E"))
            elif len(w) >= 2 and w[0] == "radius":
                radius = float(w[1].replace("D", "E"))
            elif len(w) >= 5 and w[0] in ("gfc", "gfct") and int(w[1]) <= L and int(w[2]) <= L:
                C[int(w[1]), int(w[2])], S[int(w[1]), int(w[2])] = float(w[3]), float(w[4])
    return C.to(DEV), S.to(DEV), gm, radius


def _potential(p, C, S, gm, radius, L):
    """Sum over the objects of GM/r (1 + sum (R/r)^n P(n, m) (C cos + S sin)), m > 0 by polynomials."""
    x, y, z = p[:, 0], p[:, 1], p[:, 2]
    r = torch.sqrt(x * x + y * y + z * z)
    eps, q = z / r, radius / r
    cx, sx = [torch.ones_like(x)], [torch.zeros_like(x)]
    for _ in range(L):
        c, s = cx[-1], sx[-1]
        cx.append((x * c - y * s) / r)
        sx.append((x * s + y * c) / r)
    cm, sm = torch.stack(cx, 1), torch.stack(sx, 1)  # (cos phi)^m cos/sin(m lambda)
    diag = [1.0, math.sqrt(3.0)]
    for m in range(2, L + 1):
        diag.append(diag[-1] * math.sqrt((2 * m + 1) / (2 * m)))
    total = torch.ones_like(r)
    p1 = p2 = None  # rows n - 1 and n - 2 of P / (cos phi)^m, columns 0..n-1 and 0..n-2
    for n in range(0, L + 1):
        m = torch.arange(0, n, dtype=torch.float64, device=p.device)
        row = torch.full((p.shape[0], 1), diag[n], dtype=torch.float64, device=p.device)
        if n > 0:
            low = torch.sqrt((4.0 * n * n - 1) / (n * n - m * m)) * eps[:, None] * p1
            if n > 1:
                b = torch.sqrt((2 * n + 1) * ((n - 1) ** 2 - m * m) / ((2 * n - 3) * (n * n - m * m)))
                low = low - b * torch.cat([p2, torch.zeros_like(p1[:, :1])], 1)
            row = torch.cat([low, row], 1)
        if n >= 2:
            total = total + q ** n * (row * (cm[:, :n + 1] * C[n, :n + 1] + sm[:, :n + 1] * S[n, :n + 1])).sum(1)
        p2, p1 = p1, row
    return (gm / r * total).sum()


def _force(case, seed):
    L = case["degree"]
    field = _field(L)
    pos, _ = _states(case["n"], seed, case["mix"])
    pos = _cuda(pos)
    acc, jac = [], []
    for part in pos.split(8192):
        p = part.clone().requires_grad_(True)
        (a,) = torch.autograd.grad(_potential(p, *field, L), p, create_graph=True)
        rows = [torch.autograd.grad(a[:, i].sum(), p, retain_graph=True)[0] for i in range(3)]
        acc.append(a.detach())
        jac.append(torch.stack(rows, 1))
    return torch.cat(acc), torch.cat(jac)


def _screened(case, seed):
    """Records of the two fleets below the threshold: sampled minimum, then the root of the range rate
    of the degree-8 polynomial through r, v, a at the three samples around it."""
    tr, tv, ta = _fleet(case, seed)
    n, steps, h = case["n"], case["steps"], case["h"]
    k = n // 2
    best = torch.full((k, n - k), float("inf"), dtype=torch.float64, device=DEV)
    at = torch.zeros((k, n - k), dtype=torch.int64, device=DEV)
    for i in range(steps):
        d2 = ((tr[i, :k, None, :] - tr[i, None, k:, :]) ** 2).sum(-1)
        new = d2 < best
        best, at = torch.where(new, d2, best), torch.where(new, i, at)
    # a chord cannot come nearer than the sample by more than the way both objects make in a step
    ia, ib = torch.nonzero(best < (case["threshold"] + 16e3 * h) ** 2, as_tuple=True)
    cs, ib = at[ia, ib], ib + k
    edge = (cs == 0) | (cs == steps - 1)
    mid = cs.clamp(1, steps - 2)
    u = torch.tensor([-1.0, 0.0, 1.0], dtype=torch.float64, device=DEV)
    e = torch.arange(9, dtype=torch.float64, device=DEV)
    rows = []
    for node in u:  # value, slope and curvature of each power at the node, time in steps
        rows += [node ** e, e * node ** (e - 1).clamp(min=0), e * (e - 1) * node ** (e - 2).clamp(min=0)]
    inv = torch.linalg.inv(torch.stack(rows))

    def poly(obj):
        data = []
        for node in (-1, 0, 1):
            data += [tr[mid + node, obj], tv[mid + node, obj] * h, ta[mid + node, obj] * h * h]
        return torch.einsum("ij,jpc->ipc", inv, torch.stack(data))

    A, B = poly(ia), poly(ib)

    def value(P, t, order=0):
        w = torch.ones_like(e)
        for o in range(order):
            w = w * (e - o)
        return torch.einsum("ip,ipc->pc", (w * t[:, None] ** (e - order).clamp(min=0)).T, P)

    t = torch.zeros(ia.shape[0], dtype=torch.float64, device=DEV)
    for _ in range(30):
        d, d1, d2 = (value(A - B, t, o) for o in range(3))
        t = t - (d * d1).sum(1) / ((d1 * d1).sum(1) + (d * d2).sum(1))
    pa, pb = value(A, t), value(B, t)
    time = t * h + (cs + 1) * h
    pa = torch.where(edge[:, None], tr[cs, ia], pa)
    pb = torch.where(edge[:, None], tr[cs, ib], pb)
    time = torch.where(edge, torch.where(cs == 0, 0.0, steps * h), time)
    dist = (pa - pb).norm(dim=1)
    keep = torch.nonzero(dist < case["threshold"])[:, 0]
    keep = keep[torch.argsort(ia[keep] * n + ib[keep])]
    pad = [torch.zeros((ROWS,) + x.shape[1:], dtype=torch.float64, device=DEV) for x in (dist, time, pa, pb)]
    for to, x in zip(pad, (dist, time, pa, pb)):
        to[:min(ROWS, len(keep))] = x[keep[:ROWS]]
    return dict(count=None, pair=None, distance=pad[0], time=pad[1], position_a=pad[2], position_b=pad[3])


def exact(case, seed):
    if case["kind"] == "force":
        return _force(case, seed)
    if case["kind"] == "screen":
        return _screened(case, seed)
    # a propagation is a discrete map through the Earth-orientation series: no plain counterpart
    return None
