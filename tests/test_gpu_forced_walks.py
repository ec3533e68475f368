"""The walks a default call no longer takes at these sizes, forced with GPOP_WALK_MODE: the split block's corrector and
its bad states, and lanes per group of two objects."""
import numpy as np
import pytest

import oracle_api as O
from gpu_util import dev, host

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)


def _context(monkeypatch, walk, **kw):
    import opengpop_b200 as G
    monkeypatch.setenv("GPOP_WALK_MODE", str(walk))
    try:
        return G.Context(**kw)
    finally:
        monkeypatch.delenv("GPOP_WALK_MODE")


@pytest.mark.parametrize("ncorr", [1, 2, 7])
def test_split_block_corrector(monkeypatch, oracle_data, ncorr):
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    n, steps, h = 38001, 40, 30.0
    assert G.split_block(n) == 5
    r, v = orbits.mixed_population(n, seed=31)
    low = orbits.R_EARTH * 1.003  # below the early end's altitude
    r[0], v[0] = [low, 0.0, 0.0], [0.0, np.sqrt(orbits.GM / low), 0.0]
    pick = np.array([0, 1, 2047, 9999, 23680, 27000, 35000, 38000])
    ro, vo = O.propagate(oracle_data, "gravity", START, h, steps, r[pick], v[pick], ncorr=ncorr)
    ctx = _context(monkeypatch, 2, n_corrections=ncorr)
    rr, vv = ctx.propagate(START, h, steps, r, v)
    ctx.close()
    # an acceleration (about 9 m/s^2) is rounded to a few times 2e-15 on either side, and the GJ8 sums add N of them
    # twice; ten times that, and a position's last bits at 4.2e7 m
    tol = 1e-7 + 10 * h * h * steps ** 1.5 * 7e-15
    assert np.abs(rr[pick] - ro).max() < tol and np.abs(vv[pick] - vo).max() < tol / h + 1e-10
    assert np.isfinite(rr).all()


@pytest.mark.parametrize("precision", [0, 1])
def test_bad_state_in_the_split_block(monkeypatch, precision):
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    n = 40000
    r0, v0 = orbits.mixed_population(n, 6)
    ctx = _context(monkeypatch, 2, precision=precision)
    rc, vc = dev(r0), dev(v0)
    ctx.propagate_device(START, 30.0, 12, rc, vc)
    for bad in (np.zeros(3), np.array([np.nan, 7e6, 0.0])):
        rb = r0.copy()
        rb[23456] = bad
        rd, vd = dev(rb), dev(v0)
        with pytest.raises(G.GpopError) as e:
            ctx.propagate_device(START, 30.0, 12, rd, vd)
        assert e.value.status == 1
        keep = np.arange(n) != 23456
        assert np.array_equal(host(rd)[keep], host(rc)[keep]) and np.array_equal(host(vd)[keep], host(vc)[keep])
    ctx.close()


@pytest.mark.parametrize("n,precision", [(4096, 0), (20000, 0), (9472, 1), (20000, 1)])
def test_lane_pairs(monkeypatch, oracle_data, n, precision):
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    assert G.walk_policy(n, 148, precision)[0] == 4
    r, v = orbits.mixed_population(n, seed=90 + n % 11)
    out = []
    for walk in (3, 4):
        ctx = _context(monkeypatch, walk, precision=precision)
        out.append(ctx.propagate(START, 30.0, 12, r, v))
        ctx.close()
    # FP64: rounding of reordered sums over 12 steps; mixed: FP32 rounding of the degree > 8 sums
    tol_r, tol_v = (1e-6, 1e-9) if precision == 0 else (1e-3, 1e-6)
    assert np.abs(out[1][0] - out[0][0]).max() < tol_r and np.abs(out[1][1] - out[0][1]).max() < tol_v
    if precision == 0:  # both launches of the walk
        pick = np.unique(np.clip(np.r_[0, 1, n // 2, 18943, 18944, n - 1, np.linspace(0, n - 1, 12).astype(int)], 0, n - 1))
        ro, vo = O.propagate(oracle_data, "gravity", START, 30.0, 12, r[pick], v[pick])
        assert np.abs(out[1][0][pick] - ro).max() < 1e-6 and np.abs(out[1][1][pick] - vo).max() < 1e-9
