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
