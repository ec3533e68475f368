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
