"""The search's two forms of the visited set -- a bitmap of the base, and a table with its hand-over to
global scratch -- give the same ids: a batch of at most one query per SM takes the bitmap where a
larger one may not."""
import numpy as np
import pytest

from efanna_gb300 import datasets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,point", [(31, (2, 20, 10)), (33, (3, 30, 30)), (4097, (4, 600, 100)),
                                     (1_000_003, (4, 1500, 300))])
def test_bitmap_and_table_agree(efg, n, point):
    x = datasets.mixture_u8(n, 16, seed=n % 97)
    q = datasets.mixture_u8(400, 16, seed=n % 97, queries=True)
    L = min(20, max(10, n // 3))
    idx = efg.Index(x, efg.IndexParams(trees=4, merge_level=0 if n < 100 else 4, epochs=2, check=10, L=L, K=10, S=8))
    idx.build_index()
    idx.set_search_params(*point, 4)
    whole = idx.knn_search(10, q)
    st = idx.search_stats()
    parts = np.concatenate([idx.knn_search(10, q[i:i + 50]) for i in range(0, 400, 50)])
    assert np.array_equal(whole, parts)
    one = idx.knn_search(10, q[:1])
    assert np.array_equal(one, whole[:1]) and st.queries == 400


def test_table_that_fills_within_an_epoch(efg, oracle_lib, tmp_path):
    """The table form where one epoch brings more new ids than the table has room for (uniform data: nearly
    all neighbours are new): the query goes to the overflow pass, and its ids are the oracle's."""
    O = oracle_lib
    rng = np.random.default_rng(7)
    x = rng.integers(0, 256, (1_000_003, 20)).astype(np.float32)
    q = rng.integers(0, 256, (600, 20)).astype(np.float32)
    idx = efg.Index(x, efg.IndexParams(trees=8, merge_level=8, epochs=3, check=32, L=40, K=32, S=10))
    idx.build_index()
    idx.save_trees(str(tmp_path / "t"))
    forest = O.Forest.load(str(tmp_path / "t"))
    gp, gi = idx.graph_csr()
    idx.set_search_params(6, 4000, 400, 8)
    got = idx.knn_search(10, q)
    ref = O.search(x, forest, gp, gi, q[:40], k=10, epochs=6, init_num=4000, extend_to=400, trees=8, mode=O.CANON)
    assert np.array_equal(got[:40], ref)
    for i in range(0, 600, 200):
        assert np.array_equal(idx.knn_search(10, q[i:i + 200]), got[i:i + 200])
    assert idx.search_stats().overflow_queries > 0
