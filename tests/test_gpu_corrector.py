"""The GJ8 corrector's early end gives what all n_corrections passes give: against the CPU oracle,
which runs every pass, over step sizes and pass counts on both sides of the rule (few passes or long
steps must keep the plain passes), with an orbit below the rule's altitude, in every walk."""
import os

import numpy as np
import pytest

import oracle_api as O

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)
STEPS = 40


def _tolerance(h):
    # an acceleration (about 9 m/s^2) is rounded to a few times 2e-15 on either side, and the GJ8 sums
    # add N of them twice; ten times that, and a position's last bits at 4.2e7 m
    return 1e-7 + 10 * h * h * STEPS ** 1.5 * 7e-15


def _population(n):
    from opengpop_b200 import orbits
    r, v = orbits.mixed_population(n, seed=31)
    low = orbits.R_EARTH * 1.003
    r[0], v[0] = [low, 0.0, 0.0], [0.0, np.sqrt(orbits.GM / low), 0.0]
    return r, v


def _context(walk, **kw):
    import opengpop_b200 as G
    old = os.environ.get("GPOP_WALK_MODE")
    os.environ["GPOP_WALK_MODE"] = str(walk)
    try:
        return G.Context(**kw)
    finally:
        if old is None:
            del os.environ["GPOP_WALK_MODE"]
        else:
            os.environ["GPOP_WALK_MODE"] = old


@pytest.mark.parametrize("walk", [1, 2, 3, 4])
@pytest.mark.parametrize("h,ncorr", [(10.0, 7), (30.0, 1), (30.0, 2), (30.0, 3), (30.0, 7), (60.0, 4),
                                     (120.0, 7), (300.0, 3), (300.0, 7), (30.0, 64)])
def test_passes(oracle_data, h, ncorr, walk):
    r, v = _population(41)
    ro, vo = O.propagate(oracle_data, "gravity", START, h, STEPS, r, v, ncorr=ncorr)
    ctx = _context(walk, n_corrections=ncorr)
    rr, vv = ctx.propagate(START, h, STEPS, r, v)
    ctx.close()
    assert np.abs(rr - ro).max() < _tolerance(h)
    assert np.abs(vv - vo).max() < _tolerance(h) / h + 1e-10


@pytest.mark.parametrize("ncorr", [2, 7])
def test_split_block_and_batch(oracle_data, ncorr):
    import opengpop_b200 as G
    n, pick = 38001, np.array([0, 1, 2047, 9999, 27000, 35000, 38000])
    r, v = _population(n)
    ro, _ = O.propagate(oracle_data, "gravity", START, 30.0, STEPS, r[pick], v[pick], ncorr=ncorr)
    ctx = G.Context(n_corrections=ncorr)
    rr, _ = ctx.propagate(START, 30.0, STEPS, r, v)
    assert np.abs(rr[pick] - ro).max() < _tolerance(30.0)
    reqs = [dict(start=START, h=30.0, steps=STEPS, degree=70, r=r[k], v=v[k])
            for k in (pick[:1], pick, np.arange(300))]
    out = ctx.propagate_batch(reqs)
    assert np.abs(out[0][0] - ro[:1]).max() < _tolerance(30.0)
    assert np.abs(out[1][0] - ro).max() < _tolerance(30.0)
    assert np.abs(out[2][0][:2] - ro[:2]).max() < _tolerance(30.0)
    ctx.close()
