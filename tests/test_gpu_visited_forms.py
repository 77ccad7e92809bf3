"""The search's visited set as a bitmap and as a table, over the same queries: a small base searched
with pools and extends so large that a batch of many queries takes the table (its two CTAs do not fit on
an SM and it expects to visit more ids than the base has), while at most one query per SM takes the
bitmap.  The statistics tell which form ran: only a table is outgrown."""
import numpy as np
import pytest

from efanna_gb300 import datasets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [12, 96])
@pytest.mark.parametrize("epochs,pool,extend,outgrown", [
    (4, 16_000, 700, "overflow_queries"),   # the pool itself is more than the table takes: the overflow pass
    (4, 9_000, 2_000, "migrated_queries"),  # the first expansion is: the table moves to global scratch
])
def test_outgrown_tables_give_the_bitmaps_ids(efg, oracle_lib, tmp_path, d, epochs, pool, extend, outgrown):
    O = oracle_lib
    n, nq, one_wave = 20_011, 400, 100
    x = datasets.mixture_u8(n, d, seed=d)
    q = datasets.mixture_u8(nq, d, seed=d, queries=True)
    idx = efg.Index(x, efg.IndexParams(trees=4, merge_level=4, epochs=3, check=10, L=30, K=10, S=10))
    idx.build_index()
    idx.build_trees(32)
    idx.save_trees(str(tmp_path / "t"))
    forest = O.Forest.load(str(tmp_path / "t"))
    gp, gi = idx.graph_csr()
    idx.set_search_params(epochs, pool, extend, 32)
    table = idx.knn_search(10, q)
    st = idx.search_stats()
    assert getattr(st, outgrown) == nq
    bitmap = idx.knn_search(10, q[:one_wave])
    st = idx.search_stats()
    assert st.overflow_queries == 0 and st.migrated_queries == 0
    assert np.array_equal(table[:one_wave], bitmap)
    ref = O.search(x, forest, gp, gi, q[:20], k=10, epochs=epochs, init_num=pool, extend_to=extend, trees=32,
                   mode=O.CANON)
    assert np.array_equal(table[:20], ref)
