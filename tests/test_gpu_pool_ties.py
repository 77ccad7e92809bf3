"""The search's pool selection over data of few distinct distances, where thousands of the pool's keys are
tied at the distance it cuts at: the ids are the oracle's, and ties cost no more than a share of the search."""
import statistics

import numpy as np
import pytest

from efanna_gb300 import datasets

pytestmark = pytest.mark.gpu


def _index(efg, x):
    idx = efg.Index(x, efg.IndexParams(trees=8, merge_level=4, epochs=2, check=25, L=30, K=10, S=10))
    idx.build_index()
    return idx


@pytest.mark.parametrize("kind", ["few rows", "binary", "one row"])
@pytest.mark.parametrize("pool,extend", [(40, 33), (1000, 32), (2000, 200), (2000, 256), (1999, 513)])
def test_tied_pools_match_oracle(efg, oracle_lib, tmp_path, kind, pool, extend):
    O = oracle_lib
    rng = np.random.default_rng(pool + extend)
    n, d = 20_011, 24
    x, q = np.zeros((n, d), np.float32), np.zeros((200, d), np.float32)
    cols = {"few rows": 4, "binary": d, "one row": 0}[kind]
    x[:, :cols] = rng.integers(0, 2, (n, cols))
    q[:, :cols] = rng.integers(0, 2, (200, cols))
    idx = _index(efg, x)
    idx.save_trees(str(tmp_path / "t"))
    forest = O.Forest.load(str(tmp_path / "t"))
    gp, gi = idx.graph_csr()
    idx.set_search_params(2, pool, extend, 8)
    got = idx.knn_search(20, q)
    ref = O.search(x, forest, gp, gi, q[:25], k=20, epochs=2, init_num=pool, extend_to=extend, trees=8, mode=O.CANON)
    assert np.array_equal(got[:25], ref)


def test_ties_do_not_dominate_the_search(efg):
    """4000 queries, pools of 2000: rows of 16 kinds against rows that hardly tie.  (Ranking each tied key
    over the whole pool took five times as long as the rest of the search.)"""
    n, d, nq = 200_000, 32, 4_000
    rng = np.random.default_rng(0)
    tied, q_tied = np.zeros((n, d), np.float32), np.zeros((nq, d), np.float32)
    tied[:, :4] = rng.integers(0, 2, (n, 4))
    q_tied[:, :4] = rng.integers(0, 2, (nq, 4))
    ms = []
    for x, q in ((tied, q_tied), (datasets.mixture_u8(n, d, seed=1), datasets.mixture_u8(nq, d, seed=1, queries=True))):
        idx = _index(efg, x)
        idx.set_search_params(1, 2000, 200, 8)
        runs = []
        for _ in range(7):
            idx.knn_search(10, q)
            runs.append(idx.search_stats().device_ms)
        ms.append(statistics.median(runs))
        idx.close()
    assert ms[0] < 2.5 * ms[1], ms
