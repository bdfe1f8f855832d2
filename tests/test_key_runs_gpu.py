"""Long runs of equal curve keys: spots far denser than the set's bounding cube, and many
copies of a point.  They are sorted again by their own bounding cubes, time and again, and
the call keeps its own order: cells, vertex counts and the index a repeated point keeps are
the CPU oracle's (integers, no tolerance)."""
import numpy as np
import pytest
import torch

import del3d_b200 as d3
import oracle

pytestmark = pytest.mark.gpu


def _uniform(n, seed=1):
    return np.random.default_rng(seed).random((n, 3))


def _spots(n, k, sizes, seed=2):
    """n points, k of them in each of a few spots of the given sizes."""
    rng = np.random.default_rng(seed)
    p = rng.random((n, 3))
    for j, size in enumerate(sizes):
        p[j * k:(j + 1) * k] = rng.random(3) + rng.random((k, 3)) * size
    return p[rng.permutation(n)]


def _nested(n, levels):
    """Clouds around the origin, each 2^-30 the size of the one before."""
    rng = np.random.default_rng(levels)
    return np.concatenate([rng.uniform(-1, 1, (n, 3)) * 2.0 ** (-30 * k) for k in range(levels)])


def _copies(p, counts, seed=3):
    """p with its first points repeated counts[k] times, shuffled."""
    q = np.concatenate([np.repeat(p[:len(counts)], counts, axis=0), p[len(counts):]])
    return q[np.random.default_rng(seed).permutation(len(q))]


CASES = {
    "outlier": lambda: np.concatenate([_uniform(3000), [[2.0 ** 30, 0.0, 1.0]]]),
    "far_outlier": lambda: np.concatenate([_uniform(2000), [[2.0 ** 70, 2.0 ** 69, 1.0]]]),
    "spots_33": lambda: _spots(4000, 33, [2.0 ** -40, 2.0 ** -45, 2.0 ** -30]),
    "spots_1000": lambda: _spots(6000, 1000, [2.0 ** -26, 2.0 ** -23, 2.0 ** -20]),
    "nested": lambda: _nested(300, 5),
    "copies_40": lambda: _copies(_uniform(1500), [40, 33, 32, 34, 2]),
    "copies_5000": lambda: _copies(_uniform(3000), [5000, 1000, 3]),
    "copies_in_a_spot": lambda: _copies(_spots(3000, 500, [2.0 ** -30])[::-1], [50] * 40),
    "copies_of_a_spot": lambda: np.concatenate([_spots(3000, 400, [2.0 ** -35])] * 2),
    "signed_zeros": lambda: np.concatenate([_uniform(900), np.zeros((40, 3)), -np.zeros((41, 3)), [[0.0, -0.0, 0.0]]]),
    "only_copies": lambda: np.tile([[1.0, 2.0, 3.0]], (100, 1)),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_cells_equal_oracle(cuda, case):
    pts = np.ascontiguousarray(CASES[case](), dtype=np.float64)
    want = oracle.orc_build(pts)
    d = d3.Delaunay()
    d.build(pts)
    assert d.number_of_vertices() == want["n_vertices"]
    assert np.array_equal(d.finite_cells(), want["cells"])
    assert np.array_equal(d.all_cells(), want["all"])


def test_batch(cuda):
    """All of them in one call, sets without runs between: every set as the oracle builds it."""
    sets = []
    for k, name in enumerate(sorted(CASES)):
        sets += [np.ascontiguousarray(CASES[name](), dtype=np.float64), _uniform(200 + k, k)]
    cells, nv = d3.build_batch(sets)
    for k, pts in enumerate(sets):
        want = oracle.orc_build(pts)
        assert nv[k] == want["n_vertices"] and np.array_equal(cells[k], want["cells"]), k


def test_non_finite_after_runs(cuda):
    for bad in (np.nan, np.inf):
        pts = np.concatenate([_uniform(500), np.full((200, 3), bad)])
        with pytest.raises(d3.Del3dError) as e:
            d3.Delaunay().build(pts)
        assert e.value.status == d3.ERR_INVALID_INPUT


@pytest.mark.parametrize("far", [2.0 ** 25, 2.0 ** 40])
def test_one_outlier_does_not_cost_the_order(cuda, far):
    """One point far off puts all others into one cell of the grid.  Ordering them again takes
    the radix sort once more and a few passes over flags: two to three times the order, at most
    six here (min of five builds); the spatial sort and its coordinate sorts took sixteen."""
    pts = _uniform(300000)
    plain = torch.from_numpy(pts).to(cuda)
    pts = pts.copy()
    pts[7] = far
    outlier = torch.from_numpy(pts).to(cuda)

    def order_ms(x):
        best = 1e9
        for _ in range(5):
            stats = {}
            d3.build_device(x, stats=stats)
            best = min(best, stats["ms_order"])
        return best

    assert order_ms(outlier) <= 6.0 * order_ms(plain)
