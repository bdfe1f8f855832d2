"""The variant of the insertion kernel for near points on a grid, with 8 and 16 lanes a group:
it takes the levels of builds most of whose points lie on grids of 659 to 2^20 steps, and
these widths need levels with 6000 and 12000 groups.  Cells equal the lockstep rounds' or
the CPU oracle's (integers, no tolerance), the tables are checked after every level."""
import numpy as np
import pytest
import torch

import del3d_b200 as d3
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [700001, 1300003])
def test_quantised_spheres(cuda, n):
    x = torch.from_numpy(d3.gen_sphere(n, 11, q=4096)).to(cuda)
    a, nv = d3.build_device(x, validate=True)
    a = a.clone()
    b, nv2 = d3.build_device(x, schedule=1)
    assert nv == nv2 and torch.equal(a, b)


@pytest.mark.parametrize("sets,n", [(13000, 40), (7000, 70)])
def test_many_small_sets_on_grids(cuda, sets, n):
    """Enough sets that the first levels already go to narrow groups; cospherical fives abound."""
    rng = np.random.default_rng(sets)
    v = np.array([[300, 500, 940], [0, 0, 1100], [660, 880, 0], [700, 100, 846]])
    p = v[rng.integers(0, 4, (sets, n))]
    p = np.take_along_axis(p, rng.permuted(np.tile(np.arange(3), (sets, n, 1)), axis=2), 2) * rng.choice([-1, 1], (sets, n, 3))
    p[:, ::3] = rng.integers(-1100, 1101, p[:, ::3].shape)
    sid = np.repeat(np.arange(sets), n)
    p = np.unique(np.concatenate([sid[:, None], p.reshape(-1, 3)], axis=1), axis=0)
    offs = np.concatenate([[0], np.cumsum(np.bincount(p[:, 0], minlength=sets))]).astype(np.int64)
    pts = np.ascontiguousarray(p[:, 1:], dtype=np.float64)
    cells, co, nv = d3.build_batch_device(torch.from_numpy(pts).to(cuda), offs, validate=True)
    cells = cells.cpu().numpy()
    for k in range(0, sets, sets // 60):
        want = oracle.orc_build(np.ascontiguousarray(pts[offs[k]:offs[k + 1]]))
        assert nv[k] == want["n_vertices"] and np.array_equal(cells[co[k]:co[k + 1]], want["cells"]), k
