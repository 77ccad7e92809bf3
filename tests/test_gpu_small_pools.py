"""Searches with small pools, whose warps descend several trees together in a buffer larger than the pool's
ids: ids are the oracle's for tree counts around the warps' number, and the candidate bound still holds."""
import numpy as np
import pytest

from efanna_gb300 import datasets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("trees", [1, 7, 8, 9, 16, 17, 33, 64])
@pytest.mark.parametrize("point", [(2, 10, 5), (2, 50, 10), (3, 120, 30), (4, 600, 100)])
def test_small_pools_match_oracle(efg, oracle_lib, tmp_path, trees, point):
    O = oracle_lib
    x = datasets.mixture_u8(12_007, 40, seed=5)
    q = datasets.mixture_u8(300, 40, seed=5, queries=True)
    idx = efg.Index(x, efg.IndexParams(trees=4, merge_level=4, epochs=3, check=25, L=30, K=10, S=10))
    idx.build_index()
    idx.build_trees(trees)
    idx.save_trees(str(tmp_path / "t"))
    forest = O.Forest.load(str(tmp_path / "t"))
    gp, gi = idx.graph_csr()
    k = min(10, point[2])
    for queries in (q, q + np.float32(0.25)):
        idx.set_search_params(*point, trees)
        got = idx.knn_search(k, queries)
        ref = O.search(x, forest, gp, gi, queries[:40], k=k, epochs=point[0], init_num=point[1], extend_to=point[2],
                       trees=trees, mode=O.CANON)
        assert np.array_equal(got[:40], ref)


def test_candidate_bound_of_a_small_pool(efg):
    x = datasets.mixture_u8(12_007, 40, seed=5)
    q = datasets.mixture_u8(300, 40, seed=5, queries=True)
    idx = efg.Index(x, efg.IndexParams(trees=4, merge_level=4, epochs=3, check=25, L=30, K=10, S=10))
    idx.build_index()
    idx.build_trees(16)
    idx.set_search_params(2, 50, 40, 16)
    idx.set_search_candidate_cap(1)  # the pool's 50 ids, or the descent's frontier
    with pytest.raises(efg.EfannaError):
        idx.knn_search(10, q)
    idx.set_search_candidate_cap(0)
    assert idx.knn_search(10, q).shape == (300, 10)
