"""GJ8 steps with the gravity columns split over a block's warps, at the sizes where its sets change: pairs of
objects with 16, 8, 4 and 2 lanes, full sets, a set and a remainder, idle places at the end, the corrector state
in shared memory and in the state arrays; and the groups of lanes below them. FP64 against the CPU oracle on
picked objects, mixed precision against the two-object walk; every trajectory row."""
import os

import numpy as np
import pytest

import oracle_api as O

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)
STEPS = 9


def _trajectory(precision, degree, r, v, walk, ncorr):
    import opengpop_b200 as G
    import torch
    os.environ["GPOP_WALK_MODE"] = str(walk)
    try:
        c = G.Context(precision=precision, gravity_degree=degree, n_corrections=ncorr)
    finally:
        del os.environ["GPOP_WALK_MODE"]
    n = r.shape[0]
    rd, vd = (torch.tensor(x, dtype=torch.float64, device="cuda") for x in (r, v))
    tr = [torch.full((STEPS, 3, n), float("nan"), dtype=torch.float64, device="cuda") for _ in range(3)]
    c.propagate_trajectory(START, 30.0, STEPS, rd, vd, *tr)
    out = [t.permute(0, 2, 1).cpu().numpy() for t in tr]
    assert np.array_equal(out[0][-1], rd.cpu().numpy()) and np.array_equal(out[1][-1], vd.cpu().numpy())
    c.close()
    return out


@pytest.mark.parametrize("degree", [14, 36, 70])
@pytest.mark.parametrize("per_sm", [1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 72, 96, 97, 150, 230, 383])
def test_sets(per_sm, degree):
    import torch
    from opengpop_b200 import orbits
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for n in {per_sm * sms, per_sm * sms - sms // 2}:  # every block full, and idle places in the last ones
        r, v = orbits.mixed_population(n, seed=17 + per_sm)
        tr = _trajectory(0, degree, r, v, 0, 7)
        pick = np.unique(np.concatenate([[0, 1, n // 2, n - 2, n - 1], np.random.default_rng(n).integers(0, n, 6)]))
        _, _, rs, vs, as_ = O.propagate(O.Data(degree=degree), "gravity", START, 30.0, STEPS, r[pick], v[pick],
                                        per_step=True)
        # a few last bits at 4.2e7 m, and what they make of the accelerations (2.6e-6 / s^2)
        assert np.abs(tr[0][:, pick] - rs).max() < 1e-7
        assert np.abs(tr[1][:, pick] - vs).max() < 1e-10
        assert np.abs(tr[2][:, pick] - as_).max() < 5e-13
        assert all(np.isfinite(t).all() for t in tr)
        two = _trajectory(1, degree, r, v, 5, 7)
        mixed = _trajectory(1, degree, r, v, 0, 7)
        # FP32 rounding of the degree > 8 sums: 1e-7 of some 1e-5 m/s^2 over 9 steps of 30 s
        assert np.abs(mixed[0] - two[0]).max() < 1e-5 and np.abs(mixed[1] - two[1]).max() < 1e-7


@pytest.mark.parametrize("ncorr", [1, 2])
@pytest.mark.parametrize("n", [100, 1500, 20000])
def test_few_passes(n, ncorr):
    from opengpop_b200 import orbits
    r, v = orbits.mixed_population(n, seed=n)
    tr = _trajectory(0, 70, r, v, 0, ncorr)
    pick = np.array([0, n // 3, n - 1])
    _, _, rs, _, as_ = O.propagate(O.Data(), "gravity", START, 30.0, STEPS, r[pick], v[pick], ncorr=ncorr, per_step=True)
    assert np.abs(tr[0][:, pick] - rs).max() < 1e-7 and np.abs(tr[2][:, pick] - as_).max() < 5e-13
