"""The build's own insertion order (one radix sort of set | level | Hilbert keys):
cells, vertex counts and the index a repeated point keeps must be the CPU
oracle's bit for bit (tolerance none: integers) where the keys are hardest -
repeated points, runs of equal keys up to and beyond the length that is looked
through, extents that underflow or overflow the grid, flat and tiny sets."""
import numpy as np
import pytest

import del3d_b200 as d3
import oracle

pytestmark = pytest.mark.gpu


def _clump(n, k):
    """n points, k of them so close together that they share a grid cell (each distinct)."""
    p = np.random.default_rng(n + k).random((n, 3))
    p[:k] = 0.3 + np.random.default_rng(k).integers(1, 1 << 20, (k, 3)) * 2.0 ** -48
    return p


def _copies(n, k):
    """n points, one of them k times over, in random places."""
    rng = np.random.default_rng(n * k)
    p = rng.random((n, 3))
    p[rng.permutation(n)[:k]] = p[0]
    return p


CASES = {
    "four": lambda: np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]]),
    "n63": lambda: d3.gen_uniform(63, 1),
    "n64": lambda: d3.gen_uniform(64, 1),
    "n65": lambda: d3.gen_uniform(65, 1),
    "clump_31": lambda: _clump(700, 31),
    "clump_33": lambda: _clump(700, 33),
    "clump_300": lambda: _clump(700, 300),
    "copies_2": lambda: _copies(900, 2),
    "copies_32": lambda: _copies(900, 32),
    "copies_33": lambda: _copies(900, 33),
    "copies_400": lambda: _copies(900, 400),
    "every_point_twice": lambda: np.repeat(d3.gen_uniform(1500, 4), 2, axis=0)[np.random.default_rng(1).permutation(3000)],
    "signed_zeros": lambda: np.random.default_rng(5).integers(-2, 3, (400, 3)) * np.random.default_rng(6).choice(
        [1.0, -1.0], (400, 3)),
    "huge_extent": lambda: np.random.default_rng(7).uniform(-1, 1, (300, 3)) * 2.0 ** 60,
    "tiny_extent": lambda: np.random.default_rng(8).uniform(-1, 1, (300, 3)) * 2.0 ** -60,
    "flat_slab": lambda: np.random.default_rng(9).random((2000, 3)) * [1.0, 1.0, 2.0 ** -30],
    "far_point": lambda: np.concatenate([d3.gen_uniform(500, 3), [[2.0 ** 40, 0.0, 1.0]]]),
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


def test_batch_of_every_case(cuda):
    """One call over all of them (one set's fall-back takes the whole call's), empty sets between."""
    sets = [np.zeros((0, 3))]
    for name in sorted(CASES):
        sets += [np.ascontiguousarray(CASES[name](), dtype=np.float64), np.zeros((0, 3))]
    for batch in (sets, [s for s in sets if len(s) in (0, 4, 63, 64, 65, 300, 3000)]):
        cells, nv = d3.build_batch(batch)
        for k, pts in enumerate(batch):
            want = oracle.orc_build(pts) if len(pts) else {"cells": np.zeros((0, 4), np.int32), "n_vertices": 0}
            assert nv[k] == want["n_vertices"] and np.array_equal(cells[k], want["cells"]), k


@pytest.mark.parametrize("doubled", [[], [0], [6], [1, 2, 5], list(range(7))])
def test_batch_with_copies_in_some_sets(cuda, doubled):
    """The sets with repeated points alone go through the reference's order: every set of a
    batch must come out as the oracle builds it, whichever sets hold copies."""
    sizes = [700, 5, 1200, 4, 1, 2500, 333]
    sets = [d3.gen_uniform(n, 20 + k) for k, n in enumerate(sizes)]
    for k in doubled:
        sets[k] = np.concatenate([sets[k], sets[k][::2]])
    cells, n_vertices = d3.build_batch(sets)
    for k, pts in enumerate(sets):
        want = oracle.orc_build(np.ascontiguousarray(pts))
        assert n_vertices[k] == want["n_vertices"]
        assert np.array_equal(cells[k], want["cells"])
