"""Hull facets whose vertices are collinear but for rounding.  The reference's in-circle
filter can be wrong on them for a point in their plane; met in an unlucky order, that gives
conflict regions that touch themselves along an edge (the build ended with an internal
error) or other cells.  Sets of tenths in which the last point's region does so when it goes
in last (by the oracle's predicates), at scales that change the order the build takes them
in: cells equal the CPU oracle's, which are the same for every order of these points that
was tried (integers, no tolerance)."""
import numpy as np
import pytest

import del3d_b200 as d3
import oracle

pytestmark = pytest.mark.gpu

SETS = [
    [(1, 0, 13), (4, 3, 13), (13, 12, 13), (15, -1, 13), (10, -6, 13), (18, -4, 13), (11, 13, 9), (15, 3, 11),
     (6, 9, 7), (21, 10, 11), (0, 12, 7), (21, 18, 10), (5, 7, 13)],
    [(3, 4, 27), (7, 8, 27), (15, 16, 27), (14, 11, 27), (16, 7, 27), (17, 11, 27), (9, 7, 27), (12, 1, 27),
     (24, 23, 18), (13, 25, 22), (7, 1, 23), (6, 8, 25), (28, 0, 25), (11, 25, 22), (8, 11, 27)],
    [(4, 9, 26), (10, 18, 26), (14, 24, 26), (13, 4, 26), (15, 22, 26), (9, 15, 26), (3, 8, 21), (23, 20, 25),
     (18, 22, 24), (0, 16, 20), (5, 10, 22), (7, 12, 22), (5, 23, 26)],
    [(4, 8, 12), (12, 16, 12), (24, 28, 12), (18, 8, 12), (27, 2, 12), (29, 18, 12), (2, 10, 11), (3, 0, 6),
     (19, 23, 8), (22, 18, 10), (27, 0, 9), (9, 24, 5), (13, 24, 12)],
    [(3, 7, 20), (7, 11, 20), (15, 19, 20), (4, 2, 20), (17, 14, 20), (8, 11, 20), (17, 17, 20), (10, 9, 20),
     (29, 17, 19), (10, 8, 16), (1, 15, 11), (6, 9, 13), (28, 27, 11), (20, 20, 17), (5, 12, 20)],
    [(3, 2, 20), (9, 8, 20), (18, 17, 20), (12, 2, 20), (22, 14, 20), (1, 19, 18), (15, 16, 12), (27, 27, 11),
     (29, 14, 12), (5, 11, 17), (24, 8, 15), (11, 12, 20)],
    [(9, 1, 24), (13, 5, 24), (21, 13, 24), (11, 2, 24), (19, 10, 24), (21, 1, 24), (23, -4, 24), (22, 12, 24),
     (21, 0, 24), (17, 20, 16), (12, 2, 18), (29, 4, 15), (19, 24, 17), (6, 25, 21), (0, 1, 15), (11, 12, 24)],
    [(3, 1, 27), (7, 4, 27), (15, 10, 27), (20, 5, 27), (18, 6, 27), (16, -2, 27), (5, 2, 27), (20, 7, 22), (21,
     1, 21), (22, 1, 22), (18, 24, 25), (19, 17, 23), (3, 15, 20), (3, 11, 27)],
]


@pytest.mark.parametrize("many", [True, False])
def test_hull_slivers(cuda, many):
    sets = [np.array(s, dtype=np.float64) * 0.1 * 2.0 ** k for s in SETS for k in range(-30, 31)]
    if not many:
        sets = sets[:120]                          # few enough sets for the levels in shared memory
    cells, n_vertices = d3.build_batch(sets)
    for k, pts in enumerate(sets):
        want = oracle.orc_build(pts)
        assert n_vertices[k] == want["n_vertices"] and np.array_equal(cells[k], want["cells"]), k
