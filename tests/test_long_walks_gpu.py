"""Points nearly in a line, whose walks can be thousands of steps long (a point that went the
same way at each of its attempts held its group for a third of a second).  Cells equal the lockstep rounds' (integers, no tolerance)."""
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
