"""Searches at the limit of the shared memory a query may take: what the FP32 rows allow, a byte base allows
too (the query's bytes come on top)."""
import numpy as np
import pytest

from efanna_gb300 import datasets

pytestmark = pytest.mark.gpu

# 128 dimensions, degree 10, results beyond 2048: 512 bytes of query, 40 per extended id for the candidates,
# 2 x 4096 x 8 for the lists, 16 per extended id for the rows read, of 220 KB
LIMIT = (220 * 1024 - 512 - 2 * 4096 * 8) // 56


@pytest.mark.parametrize("data", ["bytes", "floats"])
def test_largest_extend(efg, oracle_lib, tmp_path, data):
    O = oracle_lib
    x = datasets.mixture_u8(5_000, 128, seed=4)
    q = datasets.mixture_u8(40, 128, seed=4, queries=True)
    if data == "floats":
        x, q = x + np.float32(0.5), q + np.float32(0.5)
    idx = efg.Index(x, efg.IndexParams(trees=8, merge_level=3, epochs=3, check=25, L=30, K=10, S=10))
    idx.build_index()
    idx.save_trees(str(tmp_path / "t"))
    forest = O.Forest.load(str(tmp_path / "t"))
    gp, gi = idx.graph_csr()
    for extend in (LIMIT - 1, LIMIT):
        idx.set_search_params(1, 3_000, extend, 8)
        got = idx.knn_search(20, q)
        ref = O.search(x, forest, gp, gi, q[:10], k=20, epochs=1, init_num=3_000, extend_to=extend, trees=8, mode=O.CANON)
        assert np.array_equal(got[:10], ref)
    idx.set_search_params(1, 3_000, LIMIT + 1, 8)
    with pytest.raises(efg.EfannaError):
        idx.knn_search(20, q)
