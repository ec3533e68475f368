"""Device blocks kept between jobs: the same results from reused blocks, memory given back when the context
closes, an object closed after its context."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

START = (2024, 1, 1, 0, 0, 0.0)


def _jobs(ctx, r, v, k):
    n = r.shape[0]
    ca = ctx.closest_approach(START, 30.0, r, v, np.minimum(np.arange(n), k).astype(np.uint32))
    ca.propagate(40)
    ca.propagate(7)  # the store grows: new blocks, the old ones given back
    recs = [(q.object_index1, q.object_index2, q.distance, q.time) for q in ca.find(5e6)]
    ca.close()
    pairs = np.array([[0, 1], [2, n - 1]], np.int32)
    return (recs, *ctx.stm(START, 30.0, 30, r, v), *ctx.miss_gradient(START, 30.0, 40, r, v, pairs))


def test_reused_blocks_change_nothing():
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    r, v = orbits.leo(90, 3)
    ctx = G.Context(gravity_degree=20)
    first = _jobs(ctx, r, v, 9)
    for m in (70, 91, 30):  # other sizes leave their values in the kept blocks
        _jobs(ctx, *orbits.leo(m, m), 5)
    again = _jobs(ctx, r, v, 9)
    ctx.close()
    assert first[0] == again[0] and len(first[0]) > 0
    for a, b in zip(first[1:], again[1:]):
        assert np.array_equal(a, b)


def test_memory_returns_with_the_context():
    import torch
    import opengpop_b200 as G
    from opengpop_b200 import orbits
    r, v = orbits.leo(600, 5)
    held = []
    for _ in range(3):
        ctx = G.Context(gravity_degree=8)
        _jobs(ctx, r, v, 500)
        ca = ctx.closest_approach(START, 30.0, r, v, np.arange(600, dtype=np.uint32))
        ctx.close()
        ca.close()  # after its context
        torch.cuda.synchronize()
        held.append(torch.cuda.mem_get_info()[0])
    assert held[0] - held[2] < 1 << 20
