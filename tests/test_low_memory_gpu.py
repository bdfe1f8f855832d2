"""Calls that fit the device's last free memory: they were accepted with scratch of their
own size, so they still are (results equal those of the same call with room)."""
import gc

import numpy as np
import pytest
import torch

import del3d_b200 as d3

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _queries(dev, nq, k):
    pts = torch.rand((100000, 3), dtype=torch.float64, device=dev)
    idx = torch.empty((nq, k), dtype=torch.int32, device=dev)
    for part in idx.split(1 << 25):
        part.copy_(torch.randint(0, len(pts), part.shape, dtype=torch.int32, device=dev))
    idx[:1000, k - 1] = idx[:1000, 0]            # some for the exact stage
    return pts, idx, torch.zeros(nq, dtype=torch.int8, device=dev)


def _call(pts, idx, kind, out):
    return d3.library().d3g_predicates_device(pts.data_ptr(), pts.shape[0], idx.data_ptr(), idx.shape[0], kind,
                                              out.data_ptr(), None, None)


def _fill(leave):
    """Takes the device's memory but for `leave` bytes."""
    hold = []
    for _ in range(4):
        torch.cuda.synchronize()
        more = torch.cuda.mem_get_info()[0] - leave
        if more >= 4 * MB:
            hold.append(torch.empty(more // (2 * MB) * (2 * MB), dtype=torch.uint8, device="cuda"))
    free = torch.cuda.mem_get_info()[0]
    if abs(free - leave) > 8 * MB:
        pytest.skip(f"{free} bytes free where {leave} were wanted: the device is shared")
    return hold


def _with_only(leave, nq, k, kind):
    pts, idx, out = _queries("cuda", nq, k)
    want = torch.zeros_like(out)
    assert _call(pts, idx, kind, want) == d3.OK  # (also loads the kernels, with their stack)
    gc.collect()
    torch.cuda.empty_cache()
    d3.release_cached_memory()
    hold = _fill(leave)
    status = _call(pts, idx, kind, out)
    detail = d3.library().d3g_last_error()
    del hold
    torch.cuda.empty_cache()
    d3.release_cached_memory()
    assert status == d3.OK, detail
    assert torch.equal(out, want)


def test_a_block_of_its_own_size(cuda):
    """Cached blocks come in steps of up to a sixteenth; a request that only fits as it is gets
    that.  4104 MiB of queue, 4352 with the step, and 4240 free."""
    nq = 4104 * MB // 8
    _with_only(8 * nq + 136 * MB, nq, 4, d3.ORIENT3D)


def test_in_sphere_without_a_second_queue(cuda):
    """The queue of calls for the exact stage has room for one entry a query (0.8 GB here); the
    64-bit stage's second one is done without where there is no room for it."""
    nq = 100_000_000
    _with_only(8 * nq + 300 * MB, nq, 5, d3.IN_SPHERE)
