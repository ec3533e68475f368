"""Derivatives when the device's free memory is short: the vector-Jacobian product goes back to checkpoints also
where memory runs out behind the stored trajectory, and windows of Jacobians get shorter."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)
MB = 1 << 20


def _occupy(leave):
    """A tensor that leaves `leave` bytes of the device free, to the allocation's 2 MB."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty(free - leave, dtype=torch.uint8, device="cuda")


def _context(store_mb=None):
    import os
    import opengpop_b200 as G
    if store_mb is not None:
        os.environ["GPOP_ADJOINT_STORE_MB"] = str(store_mb)
    try:
        return G.Context(gravity_degree=2)
    finally:
        os.environ.pop("GPOP_ADJOINT_STORE_MB", None)


# free beside the trajectory: the startup's tangents (14 KB an object) do not fit; they do, a window's 512 MB not
@pytest.mark.parametrize("beside", [48, 320])
def test_vjp(beside):
    import torch
    from opengpop_b200 import orbits
    n, steps = 10000, 2000
    r, v = orbits.mixed_population(n, seed=4)
    g = np.random.default_rng(3)
    rb, vb = g.standard_normal((n, 3)), 1e3 * g.standard_normal((n, 3))
    ctx = _context(0)
    ref = ctx.propagate_vjp(START, 30.0, steps, r, v, rb, vb)
    ctx.close()
    ctx = _context()
    ctx.propagate_vjp(START, 30.0, 5, r[:1], v[:1], rb[:1], vb[:1])  # loads the kernels
    hold = _occupy(48 * n * steps + beside * MB)
    got = ctx.propagate_vjp(START, 30.0, steps, r, v, rb, vb)
    del hold
    torch.cuda.empty_cache()
    ctx.close()
    for a, b in zip(got, ref):  # the same positions, the same recurrences
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()


def test_stm():
    import torch
    from opengpop_b200 import orbits
    n, steps = 10000, 2000  # windows of 447 steps, 215 and 322 MB
    r, v = orbits.mixed_population(n, seed=4)
    ctx = _context()
    ref = ctx.stm(START, 30.0, steps, r, v)
    ctx.close()
    ctx = _context()
    ctx.stm(START, 30.0, 5, r[:1], v[:1])
    hold = _occupy(450 * MB)
    got = ctx.stm(START, 30.0, steps, r, v)
    del hold
    torch.cuda.empty_cache()
    ctx.close()
    for a, b in zip(got, ref):
        assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
