"""The plan a batch runs by (gpop_batch_run_plan): the requests it names for teams are those a team launch takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)
# (objects, steps, step size, degree), and which of them run on teams of how many lanes. (In the second, 110 steps at
# 20x20 on a warp, 0.59 ms by the planner's rates, end before the team's 120 at 70x70, 0.77 ms: no team for them.)
CASES = [([(1, 20000, 10.0, 70), (4096, 20, 60.0, 8), (3, 20, 60.0, 70)], [96, 0, 0]),
         ([(3, 120, 30.0, 70), (2, 110, 60.0, 20), (40, 12, 60.0, 70), (100, 6, 10.0, 8)], [96, 0, 0, 0]),
         ([(5, 100, 60.0, 20), (40, 12, 60.0, 70)], [32, 0]),
         ([(20000, 6, 30.0, 70), (8000, 4, 30.0, 36)], [0, 0])]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_run_plan(case):
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    spec, expect = CASES[case]
    reqs = []
    for i, (n, steps, h, degree) in enumerate(spec):
        r, v = orbits.leo(n, i)
        reqs.append(dict(start=START, h=h, steps=steps, degree=degree, r=r, v=v))
    ctx = G.Context(gravity_degree=70)
    lanes, team, est = ctx.batch_run_plan(reqs)
    assert [int(p) if t else 0 for p, t in zip(lanes, team)] == expect
    assert all(1 <= p <= 32 and p & (p - 1) == 0 for p, t in zip(lanes, team) if not t) and est > 0
    if not any(expect):  # no teams: the plan of the grid alone
        grid, est_grid = ctx.batch_plan(reqs)
        assert np.array_equal(lanes, grid) and est == est_grid
    before = ctx.kernel_launches
    ctx.propagate_batch(reqs)
    # frames, startup (3 + 2 per corrector pass), the items, and the teams where there are any
    assert ctx.kernel_launches - before == 1 + 3 + 2 * 7 + 1 + (1 if any(expect) else 0)
    ctx.close()
