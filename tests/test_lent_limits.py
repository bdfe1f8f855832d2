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
