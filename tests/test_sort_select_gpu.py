"""The spatial sort's quickselects against the CPU oracle's order, bit for bit: ranges on
both sides of the 8192 elements that are finished in shared memory, and the long chains
of a pass whose pivot comes last, on runs of equal coordinates and without."""
import numpy as np
import pytest

import del3d_b200 as d3
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,grid", [(70000, 3), (200000, 7), (300000, 0), (1500000, 64)])
def test_sort_selects_of_every_size(cuda, n, grid):
    rng = np.random.default_rng(n)
    pts = rng.integers(0, grid, (n, 3)).astype(np.float64) + rng.random((n, 3)) * 2.0 ** -30 if grid else rng.random((n, 3))
    if grid == 7:
        pts = np.floor(pts)
    assert np.array_equal(d3.spatial_sort(pts), oracle.orc_spatial_sort(pts))
