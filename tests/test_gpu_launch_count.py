"""gpop_kernel_launches counts what a propagation launches: frames, startup (the pipeline's kernels, or one with
compensated sums and analytic forces) and a launch per 64 steps."""
import ctypes as C

import pytest

from gpu_util import dev

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)


@pytest.mark.parametrize("precision,flags,startup", [(0, 0, 3 + 2 * 7), (1, 0, 3 + 2 * 7), (1, 8, 1)])
def test_propagation(precision, flags, startup):
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    r, v = orbits.leo(100, 3)
    ctx = G.Context(gravity_degree=20, precision=precision, flags=flags)
    rd, vd = dev(r), dev(v)
    calls = ((lambda: ctx.propagate_device(START, 30.0, 100, rd, vd), 0),
             (lambda: G.load_library().gpop_propagate_device_noalloc(
                 ctx._h, C.byref(G.as_time(START)), 30.0, 100, 100, rd.data_ptr(), vd.data_ptr(), None), 1))
    for call, extra in calls:  # the second: its epochs' arguments
        before = ctx.kernel_launches
        assert not call()
        assert ctx.kernel_launches - before == 1 + extra + startup + 2
    before = ctx.kernel_launches
    ctx.propagate_analytic("zero", 30.0, 10, rd, vd)
    assert ctx.kernel_launches - before == 1 + 1
    ctx.close()
