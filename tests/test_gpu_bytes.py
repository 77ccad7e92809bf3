"""Byte rows (a base of integers in [0, 255], at most 258 dimensions): the graph built over them and
the searches against the oracle, which computes in FP32 on the float rows -- exact on such data, so
everything must be equal.  The dimensions are the edges of 16-byte chunks and of the 258 limit; one
set has a single value outside the bytes, which must be noticed."""
import numpy as np
import pytest

from efanna_gb300 import datasets

pytestmark = pytest.mark.gpu


def _rows(n, d, seed):
    x = datasets.mixture_u8(n, d, seed=seed) if d >= 8 else \
        np.random.default_rng(seed).integers(0, 256, (n, d)).astype(np.float32)
    x[0, :] = 255.0
    x[1, :] = 0.0
    return x


@pytest.mark.parametrize("d,odd", [(2, None), (15, None), (16, None), (17, None), (100, None), (257, None), (258, None),
                                   (259, None), (64, 256.0), (64, 0.5), (64, -1.0)])
def test_byte_graph_and_search_match_oracle(efg, oracle_lib, d, odd):
    O = oracle_lib
    n = 1501
    x = _rows(n, d, seed=d)
    q = datasets.mixture_u8(40, d, seed=d, queries=True) if d >= 8 else _rows(40, d, seed=99)
    if odd is not None:
        x[n - 2, d - 1] = odd
    q[3, 0] += 0.25  # a query that is no byte row
    p = dict(trees=4, merge_level=3, epochs=3, check=25, L=30, K=10, S=10)
    idx = efg.Index(x, efg.IndexParams(**p))
    idx.build_index()
    rc, g, forest, _ = O.build_graph(x, O.make_params(K=10, S=10, L=30, check_k=25, epochs=3, trees=4, merge_level=3),
                                     O.CANON)
    assert rc == 0
    assert np.array_equal(idx.graph(), g.astype(np.uint32))
    idx.set_search_params(3, 150, 30, 4)
    ptr, ids = O.graph_csr_from_dense(g)
    ref = O.search(x, forest, ptr, ids, q, k=10, epochs=3, init_num=150, extend_to=30, trees=4, mode=O.CANON)
    got = idx.knn_search(10, q)
    rows = [i for i in range(len(q)) if i != 3]  # (query 3's distances are not integers: FP32 order may differ)
    assert np.array_equal(got[rows], ref[rows])
    assert len(set(got[3].tolist()) & set(ref[3].tolist())) >= 9


@pytest.mark.parametrize("d,K", [(3, 10), (16, 10), (17, 40), (128, 33), (257, 10), (258, 70), (259, 10)])
def test_byte_kgraph_search_matches_oracle(efg, oracle_lib, d, K):
    """Search method 1 over byte rows: graph rows below, at and beyond a warp, the list at its capacity."""
    O = oracle_lib
    n = 1501
    x = _rows(n, d, seed=d)
    q = datasets.mixture_u8(40, d, seed=d, queries=True) if d >= 8 else _rows(40, d, seed=99)
    q[3, 0] += 0.25  # a query that is no byte row
    L = max(30, K + 10)
    idx = efg.Index(x, efg.IndexParams(trees=4, merge_level=3, epochs=3, check=25, L=L, K=K, S=10))
    idx.build_index()
    rc, g, forest, _ = O.build_graph(x, O.make_params(K=K, S=10, L=L, check_k=25, epochs=3, trees=4, merge_level=3),
                                     O.CANON)
    assert rc == 0
    ptr, ids = O.graph_csr_from_dense(g)
    rows = [i for i in range(len(q)) if i != 3]
    for epochs, pool, extend, k in [(3, 300, 40, 10), (2, 150, 75, 1), (1, 200, 33, 100)]:
        idx.set_search_params(epochs, pool, extend, 4, -1, 1)
        got = idx.knn_search(k, q)
        ref, _, _ = O.search_kgraph(x, forest, ptr, ids, q, k=k, epochs=epochs, init_num=pool, extend_to=extend,
                                    trees=4, mode=O.CANON)
        assert np.array_equal(got[rows], ref[rows]), (epochs, pool, extend, k)
        assert len(set(got[3].tolist()) & set(ref[3].tolist())) >= 0.9 * k
