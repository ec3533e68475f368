"""The startup pipeline at the sizes where its kernels change (groups of whole warps, lane groups, one
and two objects per thread, partial groups and warps) against the CPU oracle on picked objects: the
replayed startup steps and the first GJ8 steps, FP64, full and low degree, one and seven passes."""
import numpy as np
import pytest

import oracle_api as O

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)
STEPS = 6


@pytest.mark.parametrize("degree", [8, 20, 70])
@pytest.mark.parametrize("n", [1, 2, 74, 75, 149, 889, 1777, 7105, 18943, 18945, 38001])
def test_sizes(n, degree):
    import opengpop_b200 as G
    import torch
    from opengpop_b200 import orbits
    data = O.Data(degree=degree)
    r, v = orbits.mixed_population(n, seed=5 + n) if n > 9 else orbits.leo(n, 5 + n)
    pick = np.unique(np.concatenate([[0, n // 2, n - 1], np.random.default_rng(n).integers(0, n, 5)]))
    for ncorr in (1, 7):
        _, _, rs, vs, as_ = O.propagate(data, "gravity", START, 30.0, STEPS, r[pick], v[pick], ncorr=ncorr,
                                        per_step=True)
        ctx = G.Context(gravity_degree=degree, n_corrections=ncorr)
        rd, vd = (torch.tensor(x, dtype=torch.float64, device="cuda") for x in (r, v))
        tr = [torch.empty(STEPS, 3, n, dtype=torch.float64, device="cuda") for _ in range(3)]
        ctx.propagate_trajectory(START, 30.0, STEPS, rd, vd, *tr)
        gr, gv, ga = (x[:, :, torch.as_tensor(pick)].permute(0, 2, 1).cpu().numpy() for x in tr)
        # positions: a few last bits at 4.2e7 m (7.5e-9); accelerations: rounding of the sums (5e-15 of
        # 9 m/s^2) and da/dr 2.6e-6 times the position's
        assert np.abs(gr - rs).max() < 1e-7
        assert np.abs(gv - vs).max() < 1e-10
        assert np.abs(ga - as_).max() < 5e-13
        ctx.close()
