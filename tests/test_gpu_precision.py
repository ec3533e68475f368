"""Errors of 64-bit results against extended precision."""
import numpy as np
import pytest

import oracle_api as O
import oracle_ld
from gpu_util import dev, host, zeros

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [2, 8, 36, 70])
def test_force(degree):
    """The central term is a product of 1/r three times: its rounding must not be found in the result three times.
    Roundings of a = -GM/r^2 (L x/r - J) that are independent (five products and the norm's three, taken 1.5
    times; half a unit at most, some 0.42 of 2^-53 in the root mean square): 1.5e-16 of |a|. Quotients by a rounded
    r add its rounding three times: 2.04e-16."""
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    pos, _ = orbits.mixed_population(3000, 17)
    hi, lo = oracle_ld.gravity(O.Data(degree=degree), pos)
    ctx = G.Context(gravity_degree=degree)
    acc = zeros(len(pos), 3)
    ctx.gravity(dev(pos), acc)
    got = host(acc)
    ctx.close()
    err = np.linalg.norm((got - hi) - lo, axis=1) / np.linalg.norm(hi, axis=1)
    assert np.sqrt((err ** 2).mean()) < 2.0e-16


# a team of warps, lanes of a warp, the columns over a block, two objects per thread: by copies of the objects
@pytest.mark.parametrize("copies", [1, 5, 25, 350])
@pytest.mark.parametrize("h,degree", [(10.0, 36), (30.0, 36), (60.0, 20), (120.0, 8)])
def test_corrector_end(h, degree, copies):
    """The corrector that ends at the fixed point found with FP32 corrections of the last digits, in the steps and in
    the startup, against seven passes: both errors are those of rounded accelerations in the GJ8 sums, of one
    size, and the root mean squares of 160 objects scatter by some 6 % each."""
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    start, steps, n = (2024, 1, 1, 0, 0, 0.0), 400, 160
    r, v = orbits.leo(n, 23)
    data = O.Data(degree=degree)
    exact = oracle_ld.propagate(data, start, h, steps, r, v)
    passes = O.propagate(data, "gravity", start, h, steps, r, v)
    ctx = G.Context(gravity_degree=degree)
    got = ctx.propagate(start, h, steps, np.tile(r, (copies, 1)), np.tile(v, (copies, 1)))
    ctx.close()
    for x, p, e in zip(got, passes, exact):
        rms = [np.sqrt((np.linalg.norm(y[:n] - e, axis=1) ** 2).mean()) for y in (x, p)]
        assert rms[0] < 1.25 * rms[1], (rms, rms[0] / rms[1])
