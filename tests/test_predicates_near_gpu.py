"""in_sphere queries of points on a common grid, on both sides of the distance up to
which they are decided in 64-bit integers (2600 steps) and of the scales that allows,
with repeated points and exact ties: signs equal the CPU oracle's (no tolerance)."""
import numpy as np
import pytest

import del3d_b200 as d3
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -20, 2.0 ** 100, 2.0 ** -200, 2.0 ** -201, 2.0 ** 191])
@pytest.mark.parametrize("reach", [3, 40, 1300, 1301, 2600, 2601, 100000])
@pytest.mark.parametrize("perturbed", [True, False])
def test_grid_queries(cuda, reach, scale, perturbed):
    rng = np.random.default_rng(reach)
    n = 4000
    # Half: corners of boxes (cospherical) and the odd repeat; half: anywhere in a cube of `reach` steps.
    corner = rng.integers(-reach, 1, (n, 1, 3))
    size = rng.integers(1, reach + 1, (n, 1, 3))
    box = corner + size * rng.integers(0, 2, (n, 5, 3))
    free = rng.integers(0, reach + 1, (n, 5, 3))
    pts = np.where(rng.random((n, 1, 1)) < 0.5, box, free) + rng.integers(-(1 << 18), 1 << 18, (n, 1, 3))
    # (an odd step among the coordinates fixes the grid)
    pts[:, 0, 0] |= 1
    flat = np.ascontiguousarray(pts.reshape(-1, 3) * scale)
    idx = np.arange(5 * n, dtype=np.int32).reshape(n, 5)
    idx[::50, 4] = idx[::50, 1]
    kind = "in_sphere" if perturbed else "in_sphere_unperturbed"
    got = (d3.in_sphere if perturbed else d3.in_sphere_unperturbed)(flat, idx)
    want = oracle.orc_predicate(kind, flat, idx)
    assert np.array_equal(got, want)
