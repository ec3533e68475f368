"""The bounded wait on the table's staging copy runs out in one warp of each block alone (the test setting
GPOP_TEST_FIRST_WAIT_WARP): the block leaves as one and the call returns the timeout, in the kernels whose teams
and blocks have barriers behind the wait as in the others. A context made without the setting works as before."""
import numpy as np
import pytest

from gpu_util import dev, host, zeros

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)


def _context(monkeypatch, walk=0, **kw):
    import opengpop_b200 as G
    monkeypatch.setenv("GPOP_TEST_FIRST_WAIT_WARP", "0")
    monkeypatch.setenv("GPOP_WALK_MODE", str(walk))
    try:
        return G.Context(**kw)
    finally:
        monkeypatch.delenv("GPOP_TEST_FIRST_WAIT_WARP")
        monkeypatch.delenv("GPOP_WALK_MODE")


def _times_out(call):
    import opengpop_b200 as G
    for _ in range(2):  # the error word is clear again after the first
        with pytest.raises(G.GpopError) as e:
            call()
        assert e.value.status == 5 and "every copy had landed" in str(e.value)


# teams of warps, lanes of a warp, columns over a block; then the walks by themselves (2 at 40,000: the split block)
@pytest.mark.parametrize("n,walk", [(1, 0), (700, 0), (2500, 0), (41, 1), (41, 2), (41, 3), (4000, 4), (40000, 2)])
@pytest.mark.parametrize("precision", [0, 1])
def test_propagation(monkeypatch, n, walk, precision):
    from opengpop_b200 import orbits
    r, v = orbits.leo(n, 9)
    ctx = _context(monkeypatch, walk, precision=precision)
    _times_out(lambda: ctx.propagate_device(START, 30.0, 8, dev(r), dev(v)))
    ctx.close()


def test_batch_with_teams(monkeypatch):
    from opengpop_b200 import orbits
    reqs = []
    for i, (n, steps) in enumerate([(1, 150), (40, 12), (100, 6)]):
        r, v = orbits.leo(n, i)
        reqs.append(dict(start=START, h=30.0, steps=steps, degree=70, r=r, v=v))
    ctx = _context(monkeypatch)
    before = ctx.kernel_launches
    _times_out(lambda: ctx.propagate_batch(reqs))
    assert ctx.kernel_launches - before == 2 * (1 + 3 + 2 * 7 + 2)  # a launch each for the items and the teams
    ctx.close()


def test_force_and_derivatives(monkeypatch):
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    r, v = orbits.leo(64, 9)
    ctx = _context(monkeypatch)
    acc, jac = zeros(64, 3), zeros(64, 3, 3)
    _times_out(lambda: ctx.gravity(dev(r), acc))
    _times_out(lambda: ctx.gravity_jacobian(dev(r), jac))
    _times_out(lambda: ctx.stm(START, 30.0, 8, r, v))
    _times_out(lambda: ctx.propagate_vjp(START, 30.0, 8, r, v, r, v))
    ctx.close()
    ctx = G.Context()
    rd, vd = dev(r), dev(v)
    ctx.propagate_device(START, 30.0, 8, rd, vd)
    assert np.isfinite(host(rd)).all()
    ctx.close()
