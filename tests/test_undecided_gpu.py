"""Sets with many tests that neither the filters nor 64-bit integers decide: lattices whose
steps are no power of two, surfaces in full doubles, clumps far smaller than the set.  Cells
equal the CPU oracle's or, for the larger sets, the lockstep rounds' (integers, no
tolerance).  And nearly all points go in asynchronously: a point given up at such a test
goes to a pass with the exact stage, not behind passes that cannot decide it either, from
which most points came to the lockstep rounds (1471 rounds for the 30^3 lattice).  The
lines: 1 point in 100 to the rounds, and two attempts given up a point (one without and one
with the 64-bit test)."""
import numpy as np
import pytest
import torch

import del3d_b200 as d3
import oracle

pytestmark = pytest.mark.gpu


def _lattice(m):
    a = np.arange(m)
    return np.stack(np.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 3).astype(np.float64)


def _rotated(p):
    q, _ = np.linalg.qr(np.random.default_rng(9).standard_normal((3, 3)))
    return p @ q


def _sphere(n):
    v = np.random.default_rng(n).standard_normal((n, 3))
    return v / np.linalg.norm(v, axis=1, keepdims=True)


def _clump(n, k, size):
    p = np.random.default_rng(k).random((n, 3))
    p[:k] = 0.3 + p[:k] * size
    return p


CASES = {
    "lattice_12_tenths": (lambda: _lattice(12) * 0.1, True),
    "lattice_9_rotated": (lambda: _rotated(_lattice(9)), True),
    "sphere_900": (lambda: _sphere(900), True),
    "clump_300_of_3000": (lambda: _clump(3000, 300, 1e-9), True),
    "lattice_30_tenths": (lambda: _lattice(30) * 0.1, False),
    "lattice_31_rotated": (lambda: _rotated(_lattice(31)), False),
    "sphere_30000": (lambda: _sphere(30000), False),
    "clump_2000_of_100000": (lambda: _clump(100000, 2000, 1e-9), False),
    "clump_half_of_50000": (lambda: _clump(50000, 25000, 2.0 ** -30), False),
}


@pytest.mark.parametrize("case", sorted(CASES))
def test_undecided_points_go_in(cuda, case):
    make, small = CASES[case]
    pts = np.ascontiguousarray(make())
    x = torch.from_numpy(pts).to(cuda)
    stats = {}
    cells, nv = d3.build_device(x, stats=stats)
    cells = cells.clone()
    if small:
        want = oracle.orc_build(pts)
        assert nv == want["n_vertices"] and np.array_equal(cells.cpu().numpy(), want["cells"])
    else:
        b, nv2 = d3.build_device(x, schedule=1)
        assert nv == nv2 and torch.equal(cells, b)
    assert stats["async_inserted"] >= 0.99 * (nv - 4), stats
    assert stats["deferred_points"] <= 2 * nv, stats


def test_batch_and_validate(cuda):
    """Sets with and without such tests together, the tables checked after every level."""
    sets = [_lattice(9) * 0.1, d3.gen_uniform(3000, 1), _sphere(700), d3.gen_lattice(1000), _rotated(_lattice(8)),
            _clump(6000, 500, 1e-9), d3.gen_uniform(9000, 2)]
    offs = np.concatenate([[0], np.cumsum([len(s) for s in sets])]).astype(np.int64)
    x = torch.from_numpy(np.concatenate(sets)).to(cuda)
    cells, co, nv = d3.build_batch_device(x, offs, validate=True)
    cells = cells.cpu().numpy()
    for k, pts in enumerate(sets):
        want = oracle.orc_build(np.ascontiguousarray(pts))
        assert nv[k] == want["n_vertices"] and np.array_equal(cells[co[k]:co[k + 1]], want["cells"]), k
