"""The join's records (per-target buckets, overflow list) and their merge into the pools, against the
oracle's state after an iteration: many records at one distance, repeated records, targets with more
records than a bucket holds, an overflow list that has to grow, pools of every slot count.

All data are small integers, so distances are exact and the states must be equal."""
import numpy as np
import pytest

from test_gpu_join_tc import _state_diff

pytestmark = pytest.mark.gpu


def _start(O, n, d, vals, L, check, seed, reverse_cap=100):
    x = np.random.default_rng(seed).integers(0, vals, (n, d)).astype(np.float32)
    params = dict(trees=4, merge_level=2, epochs=3, check=check, L=L, K=10, S=10, reverse_cap=reverse_cap)
    p = O.make_params(K=10, S=10, L=L, check_k=check, epochs=3, trees=4, merge_level=2, reverse_cap=reverse_cap)
    forest = O.Forest.build(x, 4, S=10, mode=O.CANON)
    rc, st = O.nnd_init(x, forest, p, max(L, 20) + reverse_cap, O.CANON)
    assert rc == 0
    return x, params, p, st


def _long_lists(st, rng, nodes, nn, no, hub=None):
    for i in nodes:
        ids = rng.choice(st.n, nn + no, replace=False)
        if hub is not None and hub not in ids:
            ids[0] = hub
        st.new_ids[i, :nn] = ids[:nn]
        st.old_ids[i, :no] = ids[nn:]
        st.new_cnt[i], st.old_cnt[i] = nn, no


@pytest.mark.parametrize("build", ["fp32", "bf16"])
@pytest.mark.parametrize("L,check", [(30, 25), (31, 60), (33, 25), (64, 40), (120, 200), (200, 25)])
@pytest.mark.parametrize("d,vals", [(3, 3), (16, 8)])
def test_tied_records_match_oracle(efg, oracle_lib, d, vals, L, check, build):
    """Few distinct distances: windows of tied records, duplicates within and across batches, records
    that land in the overflow slot."""
    O = oracle_lib
    x, params, p, cur = _start(O, 1500, d, vals, L, check, seed=L + d)
    idx = efg.Index(x, efg.IndexParams(**params))
    idx.set_build_precision(build)
    for it in range(3):
        nxt, pairs = O.nnd_iterate(x, cur, p, it, O.CANON)
        g = cur.copy()
        assert idx.nnd_iterate(g, it) == pairs
        assert _state_diff(nxt, g) is None, (it, _state_diff(nxt, g))
        cur = nxt


@pytest.mark.parametrize("build", ["fp32", "bf16"])
@pytest.mark.parametrize("nodes,nn,no,hub", [(500, 60, 20, 7), (1500, 130, 0, None)])
def test_overflowing_buckets_match_oracle(efg, oracle_lib, nodes, nn, no, hub, build):
    """One node in many long lists (its records overflow its bucket), and lists so long that the
    overflow list itself is too short and the join runs again."""
    O = oracle_lib
    x, params, p, st = _start(O, 1500, 24, 50, 30, 25, seed=1, reverse_cap=200)
    rng = np.random.default_rng(2)
    _long_lists(st, rng, rng.choice(st.n, nodes, replace=False), nn, no, hub)
    idx = efg.Index(x, efg.IndexParams(**params))
    idx.set_build_precision(build)
    nxt, pairs = O.nnd_iterate(x, st, p, 0, O.CANON)
    g = st.copy()
    assert idx.nnd_iterate(g, 0) == pairs
    assert _state_diff(nxt, g) is None, _state_diff(nxt, g)


@pytest.mark.parametrize("reverse_cap", [5, 31, 32, 33, 64])
def test_reverse_lists_match_oracle(efg, oracle_lib, reverse_cap):
    """Reverse lists below, at and beyond a warp's lanes, sampled and whole."""
    O = oracle_lib
    x, params, p, cur = _start(O, 2000, 6, 40, 30, 25, seed=9, reverse_cap=reverse_cap)
    idx = efg.Index(x, efg.IndexParams(**params))
    for it in range(2):
        nxt, pairs = O.nnd_iterate(x, cur, p, it, O.CANON)
        g = cur.copy()
        assert idx.nnd_iterate(g, it) == pairs
        assert _state_diff(nxt, g) is None, (it, _state_diff(nxt, g))
        cur = nxt
