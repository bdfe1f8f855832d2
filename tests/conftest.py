import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (runs on the B200 box)")


@pytest.fixture(scope="session")
def cuda():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def _word01(seed, n):
    """n words of MT19937(seed) as word * 2^-32, the reference's tests' generator (tests/pointsets.h:36-45)."""
    return np.random.RandomState(seed)._bit_generator.random_raw(n).astype(np.float64) * 2.0 ** -32


def _lattice(nx, ny, nz):
    return np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 3).astype(
        np.float64)


def _box_shell(m):
    p = _lattice(m + 1, m + 1, m + 1)
    return p[(p.min(1) == 0) | (p.max(1) == m)]


def _no_reference(*_args, **_kw):
    pytest.skip("the compiled reference (oracle/_ref) is not built")


@pytest.fixture(autouse=True)
def without_the_reference(monkeypatch):
    """Where the compiled reference is not built, the CPU oracle takes its place (tests/test_oracle.py holds the two
    equal wherever it is), and the sets made here take that of those of its point sets whose pinned orders
    (tests/test_sort_gpu.py) they have; a test that needs anything else of it is skipped."""
    import oracle

    if oracle.ref_available():
        return
    monkeypatch.setattr(oracle, "ref_build", oracle.orc_build)
    monkeypatch.setattr(oracle, "ref_spatial_sort", oracle.orc_spatial_sort)
    monkeypatch.setattr(oracle, "ref_predicate", oracle.orc_predicate)
    monkeypatch.setattr(oracle, "ps_random_cube", lambda n, seed=4: _word01(seed, 3 * n).reshape(n, 3))
    monkeypatch.setattr(oracle, "ps_lattice", _lattice)
    monkeypatch.setattr(oracle, "ps_box_shell", _box_shell)
    monkeypatch.setattr(oracle, "ps_rng_below", lambda seed, m, n: (_word01(seed, n) * m).astype(np.int64))
    for name in ("exact_predicate", "ref_circumcenters", "ps_cylinder", "ps_sphere", "ps_torus"):
        monkeypatch.setattr(oracle, name, _no_reference)


def random_idx(rng, n_pts, n_q, k):
    return rng.integers(0, n_pts, size=(n_q, k)).astype(np.int32)
