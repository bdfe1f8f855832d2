"""Lending results: a finaliser that runs while the bookkeeping's lock is held, and how much
is lent to a program that keeps its results."""
import ctypes
import gc
import threading

import numpy as np
import pytest

import del3d_b200 as d3


class _Res(ctypes.Structure):
    _fields_ = [("p", ctypes.POINTER(ctypes.c_int32))]


def _result(n=12):
    buf = (ctypes.c_int32 * n)(*range(n))
    return d3._Owned(_Res(ctypes.cast(buf, ctypes.POINTER(ctypes.c_int32))), lambda r: buf and None, 4 * n)


def test_a_result_may_end_while_another_begins():
    """The collector can end a result that sits in a cycle at any point of any thread, also
    in the middle of making another one."""
    done = threading.Event()

    def work():
        cycle = []
        cycle.append((cycle, _result()))
        del cycle
        with d3._Owned._mu:
            gc.collect()
        done.set()

    threading.Thread(target=work, daemon=True).start()
    assert done.wait(10.0)
    assert d3._Owned._held == 0


@pytest.fixture
def small_limits(monkeypatch):
    for name, value in {"FIRST": 200, "FIRST_RESULTS": 5, "MOST_RESULTS": 12, "LIMIT": 1000, "_back": 0,
                        "_back_results": 0}.items():
        monkeypatch.setattr(d3._Owned, name, value, raising=False)
    gc.collect()


def test_kept_results_are_copied_beyond_the_first(small_limits):
    """Blocks that do not come back would have to be pinned anew for every result."""
    kept = [_result() for _ in range(30)]                      # 48 bytes each
    assert [k.lent for k in kept] == [True] * 4 + [False] * 26
    arrays = [k.array(k._res.p, np.int32, 12) for k in kept]
    assert all(np.array_equal(a, np.arange(12)) and a.flags.owndata != k.lent for a, k in zip(arrays, kept))
    del kept, arrays
    gc.collect()
    kept = [_result() for _ in range(30)]                      # 4 * 48 bytes came back: 392
    assert sum(k.lent for k in kept) == 8 and d3._Owned._held == 8 * 48
    del kept
    gc.collect()
    kept = [_result() for _ in range(30)]                      # 776
    assert sum(k.lent for k in kept) == 12                     # (MOST_RESULTS)
    del kept
    gc.collect()
    assert d3._Owned._held == 0


def test_small_results_are_bounded_in_number(small_limits):
    kept = [_result(1) for _ in range(30)]
    assert sum(k.lent for k in kept) == 5
    del kept
    gc.collect()
    assert d3._Owned._held == 0
