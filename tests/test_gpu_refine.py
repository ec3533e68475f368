"""The refinement's two forms of the interpolants' divisions: lengths scaled by 2^400 leave the range of the
shared reciprocal, and scale every quotient exactly, so both runs must find the same approaches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _circles(n, steps, h, scale):
    import torch
    g = torch.Generator().manual_seed(n)
    rad = 7.0e6 + 4.0e5 * torch.rand(n, generator=g, dtype=torch.float64)
    q, _ = torch.linalg.qr(torch.randn(n, 3, 2, generator=g, dtype=torch.float64))
    w = torch.sqrt(3.986e14 / rad ** 3)
    ph = w * h * torch.arange(steps, dtype=torch.float64)[:, None] + 6.2 * torch.rand(n, generator=g, dtype=torch.float64)
    u, p = q[None, :, :, 0], q[None, :, :, 1]
    c, s = torch.cos(ph)[..., None], torch.sin(ph)[..., None]
    r = rad[None, :, None] * (c * u + s * p)
    v = (rad * w)[None, :, None] * (c * p - s * u)
    a = -(w * w)[None, :, None] * r
    return [(x * scale).to("cuda:0").contiguous() for x in (r, v, a)]


@pytest.mark.parametrize("n,steps,h", [(2, 3, 30.0), (65, 40, 30.0), (200, 64, 7.5)])
def test_shared_reciprocal_equals_division(n, steps, h):
    import opengpop_b200 as G
    ctx = G.Context(gravity_degree=4)
    found = []
    for scale in (1.0, 2.0 ** 400):
        ca = ctx.closest_approach(None, h, np.ones((n, 3)), np.ones((n, 3)), np.arange(n, dtype=np.uint32),
                                  kind="external")
        ca.append(steps, *_circles(n, steps, h, scale))
        found.append([(q.object_index1, q.object_index2, q.distance / scale, q.time) for q in ca.find(1e6 * scale)])
        ca.close()
    a, b = found
    assert [x[:2] for x in a] == [x[:2] for x in b] and (n == 2 or len(a) > 0)
    inner = [(x, y) for x, y in zip(a, b) if 0 < x[3] < steps * h]
    for x, y in inner:  # the root's tolerance is 1e-7 s on either side; the distance is stationary there
        assert abs(x[3] - y[3]) <= 2e-7
        assert abs(x[2] - y[2]) <= 1e-9 * max(x[2], 1.0) + 1e-6
    ctx.close()
