"""The counters of tests that the filter left uncertain and of exact ties.  On an integer
lattice every uncertain test is a tie (the determinants are exact, and one that is not zero
is certified), so the two counts are equal, also where one group of lanes makes tens of
thousands of them a lane in one launch (no tolerance)."""
import pytest
import torch

import del3d_b200 as d3

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kw", [(32768, {"chunk": 100000}), (8000, {"chunk": 100000}), (32768, {})])
def test_every_uncertain_test_is_a_tie(cuda, n, kw):
    stats = {}
    d3.build_device(torch.from_numpy(d3.gen_lattice(n)).to(cuda), stats=stats, **kw)
    assert stats["tie_breaks"] == stats["uncertain_tests"] > n
