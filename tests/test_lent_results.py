"""Arrays over the library's result blocks: a block goes back once, when the last
array over it is gone, and beyond the bound results are copied instead."""
import ctypes
import gc

import numpy as np
import pytest

import del3d_b200 as d3


class _Res(ctypes.Structure):
    _fields_ = [("p", ctypes.POINTER(ctypes.c_int32))]


@pytest.mark.parametrize("limit,lent", [(1 << 20, True), (47, False), (48, True)])
def test_block_lives_as_long_as_its_arrays(monkeypatch, limit, lent):
    monkeypatch.setattr(d3._Owned, "LIMIT", limit)
    buf = (ctypes.c_int32 * 12)(*range(12))
    freed = []
    own = d3._Owned(_Res(ctypes.cast(buf, ctypes.POINTER(ctypes.c_int32))), lambda r: freed.append(1), 48)
    a = own.array(own._res.p, np.int32, 12).reshape(3, 4)
    empty = own.array(own._res.p, np.int32, 0)
    part = a[1:]
    del own, a
    gc.collect()
    assert freed == ([] if lent else [1]) and empty.shape == (0,)
    assert part.flags.writeable and np.array_equal(part, np.arange(4, 12).reshape(2, 4))
    del part
    gc.collect()
    assert freed == [1] and d3._Owned._held == 0


@pytest.mark.gpu
def test_results_survive_later_builds(cuda):
    want = []
    kept = []
    for k in range(6):
        d = d3.Delaunay()
        d.build(d3.gen_uniform(3000 + k, k))
        kept.append((d.finite_cells(), d.all_cells(), *d.incident_csr()))
        want.append([x.copy() for x in kept[-1]])
        del d
    cells, _ = d3.build_batch([d3.gen_uniform(500, k) for k in range(4)])
    again, _ = d3.build_batch([d3.gen_uniform(500, k) for k in range(4)])
    assert all(np.array_equal(a, b) for a, b in zip(cells, again))
    for a, b in zip(kept, want):
        assert all(np.array_equal(x, y) for x, y in zip(a, b))
