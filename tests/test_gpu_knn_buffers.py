"""Exact k-NN where candidate buffers are too short or too many: queries among thousands of copies of a
row, which alone go through the sorted lists.  Ids and distances equal the FP32 screening's."""
import numpy as np
import pytest

from test_gpu_exact_knn import _knn

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("screening", ["auto", "split"])
@pytest.mark.parametrize("k,d,near,exclude", [(10, 33, 1, False), (10, 128, 3, True), (100, 20, 130, False),
                                              (100, 96, 1, True)])
def test_only_queries_among_copies_take_the_lists(efg, k, d, near, exclude, screening):
    rng = np.random.default_rng(k + d)
    n, nq, first = 140_011, 2_000, 1_000
    x = rng.integers(0, 100, (n, d)).astype(np.float32)
    copy = rng.integers(200, 256, d).astype(np.float32)  # far from the other rows and queries
    x[5_000:10_000] = copy
    if exclude:  # a run of base rows, of which `near` are copies
        rows = np.arange(first, first + nq)
        x[first + 11:first + 11 + near] = copy
        q = x[rows].copy()
    else:
        q = rng.integers(0, 100, (nq, d)).astype(np.float32)
        q[::nq // near][:near] = copy
        q[::nq // near][:near, 0] -= 3
    f32 = _knn(efg, x, q, k, "fp32", exclude=exclude, first_row=first if exclude else 0)
    tc = _knn(efg, x, q, k, screening, exclude=exclude, first_row=first if exclude else 0)
    assert efg.knn_stats().list_queries == near
    assert np.array_equal(tc[0], f32[0]) and np.array_equal(tc[1], f32[1])
