"""Points nearly in a line, whose walks can be thousands of steps long (a point that went the
same way at each of its attempts held its group for a third of a second), and concentric
spheres in full doubles.  Cells equal the lockstep rounds' (integers, no tolerance)."""
import numpy as np
import pytest
import torch

import del3d_b200 as d3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,noise", [(100000, 1e-9), (20000, 1e-14), (30000, 1e-4)])
def test_points_nearly_in_a_line(cuda, n, noise):
    rng = np.random.default_rng(7)
    pts = np.stack([rng.random(n), noise * rng.random(n), noise * rng.random(n)], 1)
    x = torch.from_numpy(pts).to(cuda)
    a, nv = d3.build_device(x)
    a = a.clone()
    b, nv2 = d3.build_device(x, schedule=1)
    assert nv == nv2 and torch.equal(a, b)


def test_concentric_spheres(cuda):
    """Regions of hundreds of tets, nearly all of their tests exact: they go in with room for
    large regions, hardly any through the lockstep rounds (9 of 10 at least; a third did not)."""
    rng = np.random.default_rng(7)
    pts = []
    for r in (1.0, 1.5, 2.0):
        v = rng.standard_normal((2500, 3))
        pts.append(v / np.linalg.norm(v, axis=1, keepdims=True) * r)
    x = torch.from_numpy(np.concatenate(pts)).to(cuda)
    stats = {}
    a, nv = d3.build_device(x, stats=stats)
    a = a.clone()
    b, nv2 = d3.build_device(x, schedule=1)
    assert nv == nv2 and torch.equal(a, b)
    assert stats["async_inserted"] >= 0.9 * nv, stats
