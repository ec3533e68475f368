"""Derivatives of propagations with few corrector passes, whose last evaluation is not at the step's position:
transition matrices, and the adjoint from stored positions and from checkpoints, against differences of the same
propagation in long double."""
import os

import numpy as np
import pytest

import oracle_api as O
import oracle_ld

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)


@pytest.mark.parametrize("h,ncorr", [(30.0, 1), (60.0, 1), (60.0, 3), (120.0, 1), (120.0, 3), (120.0, 7)])
def test_derivatives(h, ncorr):
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    n, steps = 6, 70  # two segments of checkpoints
    r, v = orbits.mixed_population(n, 5)
    ref = oracle_ld.stm(O.Data(degree=8), START, h, steps, r, v, ncorr)
    ctx = G.Context(gravity_degree=8, n_corrections=ncorr)
    phi = ctx.stm(START, h, steps, r, v)[2].reshape(n, 6, 6)
    # 70 steps' rounded tangents in sums of sums: 70^1.5 1.1e-16 = 6e-14, a block's cancelling parts
    # may be a hundred times its values
    tol = 1e-11
    top = np.abs(ref).reshape(n, 2, 3, 2, 3).max(axis=(2, 4)).repeat(3, axis=1).repeat(3, axis=2)  # of a block
    assert (np.abs(phi - ref) <= tol * top).all()
    g = np.random.default_rng(1)
    bar = np.concatenate([g.standard_normal((n, 3)), 1e3 * g.standard_normal((n, 3))], axis=1)
    expect = np.einsum("ni,nij->nj", bar, ref)
    size = np.einsum("ni,nij->nj", np.abs(bar), top)
    for mb in (None, "0"):
        if mb is not None:
            os.environ["GPOP_ADJOINT_STORE_MB"] = mb
        try:
            adj = G.Context(gravity_degree=8, n_corrections=ncorr)
        finally:
            os.environ.pop("GPOP_ADJOINT_STORE_MB", None)
        got = np.concatenate(adj.propagate_vjp(START, h, steps, r, v, bar[:, :3], bar[:, 3:]), axis=1)
        adj.close()
        assert (np.abs(got - expect) <= tol * size).all()
    ctx.close()
