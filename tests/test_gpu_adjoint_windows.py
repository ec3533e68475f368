"""The adjoint of so many objects that a checkpoint's segment takes two windows of Jacobians and the startup
tangents several pieces: each segment is run again once, and the gradients are those of the objects alone."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)


def test_one_run_per_segment():
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    n = 150001  # 60 steps of the first segment: 9.0 million Jacobians, 7.5 to a window
    r, v = orbits.mixed_population(n, seed=8)
    g = np.random.default_rng(2)
    rb, vb = g.standard_normal((n, 3)), 1e3 * g.standard_normal((n, 3))
    os.environ["GPOP_ADJOINT_STORE_MB"] = "0"
    try:
        ctx = G.Context(gravity_degree=2)
    finally:
        del os.environ["GPOP_ADJOINT_STORE_MB"]
    count = []
    for steps in (4, 64):
        before = ctx.kernel_launches
        gr, gv = ctx.propagate_vjp(START, 30.0, steps, r, v, rb, vb)
        count.append(ctx.kernel_launches - before)
    # 4 steps: a sweep of nothing; 64: the segment's run, two windows of a launch each for Jacobians and sweep
    assert count[1] - count[0] == 1 + 2 * 2 - 1
    pick = np.array([0, 65535, 65536, 131071, 131072, n - 1])  # on either side of the pieces
    sr, sv = ctx.propagate_vjp(START, 30.0, 64, r[pick], v[pick], rb[pick], vb[pick])
    ctx.close()
    # other kernels for other counts: positions to some 1e-15 of their size
    for a, b in ((gr[pick], sr), (gv[pick], sv)):
        assert (np.abs(a - b).max(axis=1) <= 1e-9 * np.abs(b).max(axis=1)).all()
    assert np.isfinite(gr).all() and np.isfinite(gv).all()



def test_matrices_in_pieces():
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    n, steps = 65536 + 300, 12
    r, v = orbits.mixed_population(n, seed=9)
    pick = np.array([0, 1, 65535, 65536, n - 1])  # on either side of the pieces
    ctx = G.Context(gravity_degree=8)
    got = ctx.stm(START, 30.0, steps, r, v)
    few = ctx.stm(START, 30.0, steps, r[pick], v[pick])
    ctx.close()
    for a, b in zip(got, few):  # other kernels for other counts, as above
        a, b = a[pick].reshape(len(pick), -1), b.reshape(len(pick), -1)
        assert (np.abs(a - b).max(axis=1) <= 1e-9 * np.abs(b).max(axis=1)).all()
    assert all(np.isfinite(x).all() for x in got)
