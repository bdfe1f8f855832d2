"""The asynchronous insertion kernel at the sizes where its choices change: the
lanes a group gets (32, 16, 8 by the work of a level), regions beyond a group's
scratch, points left over at the last level.  Cells equal the lockstep rounds' -
another kernel and another insertion order - or the CPU oracle's, bit for bit
(integers; no tolerance), and the tet table's invariants hold after every level."""
import numpy as np
import pytest
import torch

import del3d_b200 as d3
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dist,n", [("uniform", 5), ("uniform", 33), ("clusters", 257), ("lattice", 4097),
                                    ("sphere", 30011), ("uniform", 150001), ("lattice", 320000),
                                    ("clusters", 700001), ("uniform", 1300003)])
def test_lane_choices_equal_rounds(cuda, dist, n):
    x = torch.from_numpy(d3.gen_set(dist, n, n % 97)).to(cuda)
    a, nv = d3.build_device(x, validate=True)
    a = a.clone()
    b, nv2 = d3.build_device(x, schedule=1)
    assert nv == nv2 and torch.equal(a, b)


@pytest.mark.parametrize("sets,n", [(13000, 40), (7000, 64), (300, 600)])
def test_many_small_sets(cuda, sets, n):
    """Enough sets that the first levels already go to narrow groups."""
    rng = np.random.default_rng(sets)
    pts = rng.random((sets * n, 3))
    offs = np.arange(sets + 1, dtype=np.int64) * n
    cells, co, nv = d3.build_batch_device(torch.from_numpy(pts).to(cuda), offs, validate=True)
    cells = cells.cpu().numpy()
    for k in range(0, sets, sets // 60):
        want = oracle.orc_build(pts[k * n:(k + 1) * n])
        assert nv[k] == n and np.array_equal(cells[co[k]:co[k + 1]], want["cells"]), k


@pytest.mark.parametrize("around", [200, 300, 600, 5000])
def test_regions_beyond_the_scratch(cuda, around):
    """Points on a sphere about a cloud, then the cloud: an early point's region holds
    nearly every tet (64, 128 and 256 fit a group of 8, 16 and 32 lanes)."""
    rng = np.random.default_rng(around)
    v = rng.standard_normal((around, 3))
    shell = 10.0 * v / np.linalg.norm(v, axis=1, keepdims=True)
    pts = np.concatenate([shell, rng.standard_normal((40, 3)) * 1e-3])
    want = oracle.orc_build(pts)
    d = d3.Delaunay()
    d.build(pts)
    assert np.array_equal(d.finite_cells(), want["cells"]) and np.array_equal(d.all_cells(), want["all"])


@pytest.mark.parametrize("around", [900, 1800, 4000])
def test_big_regions_that_overlap(cuda, around):
    """Sets whose inner points' regions hold thousands of tets of a shell (4096 is the
    widest group's room) and get in each other's way; on a grid, so that ties abound."""
    rng = np.random.default_rng(around)
    sets = []
    for k in range(6):
        v = rng.standard_normal((around, 3))
        shell = np.round(1024.0 * v / np.linalg.norm(v, axis=1, keepdims=True))
        inner = rng.integers(-20, 21, (15, 3))
        sets.append(np.unique(np.concatenate([shell, inner]), axis=0)[rng.permutation(around)[:around - 50]])
    cells, n_vertices = d3.build_batch(sets)
    for k, pts in enumerate(sets):
        want = oracle.orc_build(pts)
        assert n_vertices[k] == want["n_vertices"] and np.array_equal(cells[k], want["cells"]), k


def test_offset_lattice_and_caller_chunks(cuda):
    """A lattice away from the origin, and the worker densities a caller may ask for."""
    pts = d3.gen_lattice(9000) + [700.0, -300.0, 55.0]
    want = oracle.orc_build(pts)["cells"]
    x = torch.from_numpy(pts).to(cuda)
    for kw in ({}, {"chunk": 7}, {"chunk": 100000}, {"chunk": -1, "alpha_small": 1}, {"chunk": -500}):
        assert np.array_equal(d3.build_device(x, **kw)[0].cpu().numpy(), want), kw


def _grid_ball(radius, n, seed):
    """n distinct integer points on a few concentric integer spheres and in the planes of their poles:
    many exactly cospherical and cocircular groups, differences of up to 2 * radius."""
    rng = np.random.default_rng(seed)
    base = np.array([[radius, 0, 0], [radius * 3 // 5, radius * 4 // 5, 0], [radius // 3, radius * 2 // 3, radius * 2 // 3]])
    v = base[rng.integers(0, 3, 4 * n)]
    v = np.take_along_axis(v, rng.permuted(np.tile(np.arange(3), (4 * n, 1)), axis=1), 1) * rng.choice([-1, 1], (4 * n, 3))
    v = v // rng.choice([1, 2], (4 * n, 1))
    p = np.unique(np.concatenate([v, rng.integers(-radius, radius + 1, (n // 4, 3))]), axis=0)
    return rng.permutation(p)[:n].astype(np.float64)


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -10, 2.0 ** 40, 2.0 ** -199, 2.0 ** 189, 2.0 ** -210])
@pytest.mark.parametrize("radius", [315, 330, 1290, 1305, 5400, 60000])
def test_exact_by_differences(cuda, radius, scale):
    """Sets on either side of the lines up to which the filters are exact for the whole set (659 steps
    across for in_sphere, 110000 for orient3d) and for one test (2600 steps), at both ends of the scales."""
    pts = _grid_ball(radius, 300, radius) * scale
    pts += np.array([7.0, -3.0, 11.0]) * radius * scale
    want = oracle.orc_build(pts)
    d = d3.Delaunay()
    d.build(pts)
    assert np.array_equal(d.finite_cells(), want["cells"]) and np.array_equal(d.all_cells(), want["all"])
