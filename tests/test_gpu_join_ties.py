"""Merging records at one distance by the thousand: rows of a few kinds, every one with hundreds of copies,
and check_k on either side of the pool's capacity, where it decides whether a record in the overflow
slot or a duplicate counts as found.  States are the oracle's; the time stays in proportion."""
import time

import numpy as np
import pytest

from test_gpu_join_records import _long_lists, _start
from test_gpu_join_tc import _state_diff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("build", ["fp32", "bf16"])
@pytest.mark.parametrize("L,check", [(30, 30), (30, 31), (30, 32), (40, 41), (64, 65), (64, 66), (100, 101),
                                     (150, 200), (200, 25)])
@pytest.mark.parametrize("d,vals", [(1, 2), (2, 2), (4, 2)])
def test_rows_of_few_kinds_match_oracle(efg, oracle_lib, d, vals, L, check, build):
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
@pytest.mark.parametrize("L,check", [(30, 25), (30, 31), (30, 40), (150, 100)])
def test_a_hub_among_few_kinds_matches_oracle(efg, oracle_lib, L, check, build):
    """One node in 600 lists of 80: thousands of its records at each of three distances."""
    O = oracle_lib
    x, params, p, st = _start(O, 1500, 2, 2, L, check, seed=3, reverse_cap=200)
    rng = np.random.default_rng(4)
    _long_lists(st, rng, rng.choice(st.n, 600, replace=False), 60, 20, 7)
    idx = efg.Index(x, efg.IndexParams(**params))
    idx.set_build_precision(build)
    nxt, pairs = O.nnd_iterate(x, st, p, 0, O.CANON)
    g = st.copy()
    assert idx.nnd_iterate(g, 0) == pairs
    assert _state_diff(nxt, g) is None, _state_diff(nxt, g)


def test_copies_do_not_dominate_the_build(efg):
    """100,000 rows of 16 kinds against as many that differ: within 20 times (170 when the merge sorted its way
    through all of a hub's tied records 32 at a time)."""
    n, d = 100_000, 24
    rng = np.random.default_rng(0)
    copies = np.zeros((n, d), np.float32)
    copies[:, :4] = rng.integers(0, 2, (n, 4))
    s = []
    for x in (copies, rng.integers(0, 256, (n, d)).astype(np.float32)):
        idx = efg.Index(x, efg.IndexParams(K=10, L=30, check=25, S=10, trees=4, merge_level=4, epochs=4))
        idx.build_index()
        t0 = time.perf_counter()
        idx.build_index()
        s.append(time.perf_counter() - t0)
        idx.close()
    assert s[0] < 20 * s[1], s
