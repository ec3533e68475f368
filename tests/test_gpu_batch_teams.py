"""Batches whose longest requests run on teams of warps: every request as its own propagate call (FP64 to the
rounding of reordered sums over these steps, mixed precision as in test_gpu_batch)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)
SHORT = [(40, 12, 60.0, 70), (3, 0, 30.0, 20), (100, 6, 10.0, 8)]
# (objects, steps, step size, degree) of the long requests: one lane group per SM and two; a team of one, two and
# three warps; degrees mixed in one launch; a batch of nothing else; five steps, the first after the startup's four
CASES = [[(1, 150, 30.0, 70)], [(3, 120, 30.0, 70), (2, 110, 60.0, 20)], [(45, 90, 30.0, 70)], [(70, 80, 30.0, 36)],
         [(5, 100, 60.0, 20)], [(2, 5, 30.0, 50)]]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_long_requests_on_teams(case, precision):
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    alone = case == len(CASES) - 1
    spec = CASES[case] + ([] if alone else SHORT)
    reqs = []
    for i, (n, steps, h, degree) in enumerate(spec):
        r, v = orbits.mixed_population(n, seed=17 * case + i)
        reqs.append(dict(start=START, h=h, steps=steps, degree=degree, r=r, v=v))
    ctx = G.Context(gravity_degree=70, precision=precision)
    before = ctx.kernel_launches
    outs = ctx.propagate_batch(reqs)
    # frames, startup (3 + 2 per corrector pass), and a launch each for the items and the teams
    assert ctx.kernel_launches - before == 1 + 3 + 2 * 7 + (1 if alone else 2)
    again = ctx.propagate_batch(reqs)  # the captured graph
    for (r1, v1), (r2, v2) in zip(outs, again):
        assert np.array_equal(r1, r2) and np.array_equal(v1, v2)
    tol_r, tol_v = (1e-6, 1e-9) if precision == 0 else (1e-3, 1e-6)
    for q, (r, v) in zip(reqs, outs):
        if q["steps"] == 0:
            continue
        ref = G.Context(gravity_degree=q["degree"])
        rr, vv = ref.propagate(START, q["h"], q["steps"], q["r"], q["v"])
        ref.close()
        assert np.linalg.norm(r - rr, axis=1).max() <= tol_r
        assert np.linalg.norm(v - vv, axis=1).max() <= tol_v
    ctx.close()
