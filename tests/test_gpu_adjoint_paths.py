"""The adjoint from checkpoints against the adjoint from stored positions, in one window of Jacobians and in
several; Jacobians of points at the sizes where their kernel changes."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)


def _context(degree, store_mb=None):
    import opengpop_b200 as G
    if store_mb is not None:
        os.environ["GPOP_ADJOINT_STORE_MB"] = str(store_mb)
    try:
        return G.Context(gravity_degree=degree)
    finally:
        os.environ.pop("GPOP_ADJOINT_STORE_MB", None)


def _bars(n, seed):
    g = np.random.default_rng(seed)
    return g.standard_normal((n, 3)), 1e3 * g.standard_normal((n, 3))


@pytest.mark.parametrize("steps", [1, 4, 5, 63, 64, 65, 130])
@pytest.mark.parametrize("n", [1, 3])
def test_checkpoints_equal_stored_positions(n, steps):
    from opengpop_b200 import orbits
    r, v = orbits.mixed_population(n, seed=steps)
    out = []
    for mb in (None, 0):
        ctx = _context(20, mb)
        out.append(np.concatenate(ctx.propagate_vjp(START, 30.0, steps, r, v, *_bars(n, 5)), axis=1))
        ctx.close()
    # the segments take the forward run's steps again: the same positions, the same recurrences
    assert np.abs(out[0] - out[1]).max() <= 1e-12 * np.abs(out[0]).max()


@pytest.mark.parametrize("store_mb", [None, 0])
def test_several_windows(store_mb):
    from opengpop_b200 import orbits
    n, steps = 40000, 200  # 8 million Jacobians: more than a window holds
    r, v = orbits.mixed_population(n, seed=3)
    rb, vb = _bars(n, 6)
    pick = np.array([0, 17, 20000, 39998, 39999])
    ctx = _context(4, store_mb)
    gr, gv = ctx.propagate_vjp(START, 30.0, steps, r, v, rb, vb)
    sr, sv = ctx.propagate_vjp(START, 30.0, steps, r[pick], v[pick], rb[pick], vb[pick])
    ctx.close()
    # other kernels for other counts: positions to some 1e-15 of their size
    for a, b in ((gr[pick], sr), (gv[pick], sv)):
        assert (np.abs(a - b).max(axis=1) <= 1e-9 * np.abs(b).max(axis=1)).all()
    assert np.isfinite(gr).all() and np.isfinite(gv).all()


@pytest.mark.parametrize("degree", [8, 70])
def test_jacobian_sizes(degree):
    import torch
    from opengpop_b200 import orbits
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    r, _ = orbits.mixed_population(sms * 300, seed=9)
    dev = torch.tensor(r, dtype=torch.float64, device="cuda")
    ctx = _context(degree)

    def jac(x):
        J = torch.full((x.shape[0], 3, 3), float("nan"), dtype=torch.float64, device="cuda")
        ctx.gravity_jacobian(x, J)
        return J

    for n in (2, 4 * sms, 8 * sms + 1, 64 * sms, 64 * sms + 1, 128 * sms - 1, 128 * sms, 128 * sms + 1, 300 * sms):
        J = jac(dev[:n].contiguous())
        assert torch.isfinite(J).all()
        for i in (0, n // 2, n - 1):  # one point: 32 lanes; sums of some 2,500 terms in another order
            one = jac(dev[i:i + 1].contiguous())[0]
            assert (J[i] - one).abs().max() <= 1e-12 * one.abs().max()
    ctx.close()
