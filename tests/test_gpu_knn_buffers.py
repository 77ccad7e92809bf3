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


def _classes(rng, n, nq, d, classes, order):
    """Rows and queries of `classes` distant classes; the rows class by class or in turn."""
    centres = rng.integers(0, 200, (classes, d))
    of = np.arange(n) * classes // n if order == "sorted" else np.arange(n) % classes
    x = centres[of] + rng.integers(0, 50, (n, d))
    q = centres[rng.integers(0, classes, nq)] + rng.integers(0, 50, (nq, d))
    return x.astype(np.float32), q.astype(np.float32)


@pytest.mark.parametrize("n,nq,k,order,classes", [
    (20_000, 300, 10, "sorted", 4), (60_011, 300, 100, "sorted", 10), (7_000, 200, 104, "sorted", 5),
    (60_011, 300, 100, "in turn", 2), (1 << 16, 300, 10, "sorted", 8), (1 << 18, 500, 10, "in turn", 16),
    (1 << 18, 500, 100, "in turn", 8), (300_000, 300, 10, "sorted", 30)])
def test_bounds_hold_whatever_the_order_of_the_rows(efg, n, nq, k, order, classes):
    """Rows in class order and classes in turn: the bounds' groups and samples reach every class, so that no
    query finds a whole class under its bound."""
    x, q = _classes(np.random.default_rng(n + k), n, nq, 64, classes, order)
    for screening in ("auto", "split"):
        tc = _knn(efg, x, q, k, screening)
        assert efg.knn_stats().list_queries == 0
        f32 = _knn(efg, x, q, k, "fp32")
        assert np.array_equal(tc[0], f32[0]) and np.array_equal(tc[1], f32[1])


@pytest.mark.parametrize("n", [544, 545, 607, 1_791, 2_063, 4_300, 28_799])
@pytest.mark.parametrize("k,d", [(1, 5), (10, 64), (10, 129)])
def test_strided_groups_at_their_edges(efg, n, k, d):
    """Boxes of 16 and 64 rows a prime number apart, with empty columns at their ends."""
    rng = np.random.default_rng(n + d)
    x = rng.integers(0, 256, (n, d)).astype(np.float32)
    q = rng.integers(0, 256, (150, d)).astype(np.float32)
    for screening in ("auto", "split"):
        tc = _knn(efg, x, q, k, screening)
        f32 = _knn(efg, x, q, k, "fp32")
        assert np.array_equal(tc[0], f32[0]) and np.array_equal(tc[1], f32[1])


@pytest.mark.parametrize("n,k,copies", [(400, 10, 0), (5_000, 10, 0), (40_000, 10, 0), (140_011, 100, 5_000),
                                        (60_011, 100, 0), (20_000, 10, 3_000)])
@pytest.mark.parametrize("nq,groups", [(1_300, 1), (1_300, 2), (1_281, 1), (513, 2)])
@pytest.mark.parametrize("exclude", [False, True])
def test_queries_in_blocks(efg, n, k, copies, nq, groups, exclude):
    """Candidate buffers for 256 or 512 queries at a time: even and ragged last blocks, with queries in
    several blocks that overrun their buffers."""
    rng = np.random.default_rng(n + nq)
    d, first = 24, 50
    x = rng.integers(0, 100, (n, d)).astype(np.float32)
    if exclude:
        nq = min(nq, n - first)
        if copies:
            x[first:first + nq:199] = 220
        q = x[first:first + nq].copy()
    else:
        q = rng.integers(0, 100, (nq, d)).astype(np.float32)
        if copies:
            q[::199] = 220
    if copies:
        x[n - copies:] = 220
    X, Q = torch.from_numpy(x).cuda(), torch.from_numpy(q).cuda()
    ids = torch.full((nq, k), -7, dtype=torch.int32, device="cuda")
    dist = torch.full((nq, k), -1.0, dtype=torch.float32, device="cuda")
    per = 8 * (4096 if k == 100 else 2048)  # bytes of a query's buffer
    f32 = _knn(efg, x, q, k, "fp32", exclude=exclude, first_row=first)
    efg._check(efg.lib().efg_brute_force_knn_within(X.data_ptr(), n, d, d, Q.data_ptr(), nq, d, k, int(exclude), first,
                                                    ids.data_ptr(), dist.data_ptr(), groups * 256 * per + 100, None))
    torch.cuda.synchronize()
    assert efg.knn_stats().list_queries == (-(-nq // 199) if copies else 0)
    assert np.array_equal(ids.cpu().numpy(), f32[0]) and np.array_equal(dist.cpu().numpy(), f32[1])


def test_many_queries_with_little_memory(efg):
    """80,000 queries with 2.6 GB of candidate buffers between them where 1 GB is left: taken in blocks."""
    n, nq, d, k = 20_000, 80_000, 16, 100
    g = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randint(0, 256, (n, d), generator=g, device="cuda").float()
    Q = torch.randint(0, 256, (nq, d), generator=g, device="cuda").float()
    ids = torch.empty((nq, k), dtype=torch.int32, device="cuda")
    dist = torch.empty((nq, k), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    ballast = torch.empty(torch.cuda.mem_get_info()[0] - (1 << 30), dtype=torch.uint8, device="cuda")
    try:
        efg.brute_force_knn_device(X.data_ptr(), n, d, d, Q.data_ptr(), nq, d, k, ids.data_ptr(), dist.data_ptr())
        torch.cuda.synchronize()
    finally:
        del ballast
        torch.cuda.empty_cache()
    some = torch.arange(0, nq, 131, device="cuda")
    f32 = _knn(efg, X.cpu().numpy(), Q[some].cpu().numpy(), k, "fp32")
    assert np.array_equal(ids[some].cpu().numpy(), f32[0]) and np.array_equal(dist[some].cpu().numpy(), f32[1])


def test_sample_grows_with_the_base(efg):
    """45 million rows: a bound from 2^20 of them leaves more values under it (45 / 1.05 x 116 = 4980) than
    a buffer's 4096, so the sample has to be larger."""
    n, nq, d, k = 45_000_000, 64, 8, 100
    g = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randint(0, 256, (n, d), generator=g, device="cuda", dtype=torch.uint8).float()
    Q = torch.randint(0, 256, (nq, d), generator=g, device="cuda", dtype=torch.uint8).float()
    out = {}
    for screening in ("fp32", "auto"):
        ids = torch.empty((nq, k), dtype=torch.int32, device="cuda")
        dist = torch.empty((nq, k), dtype=torch.float32, device="cuda")
        efg.brute_force_knn_device(X.data_ptr(), n, d, d, Q.data_ptr(), nq, d, k, ids.data_ptr(), dist.data_ptr(),
                                   screening=screening)
        torch.cuda.synchronize()
        out[screening] = ids.cpu().numpy(), dist.cpu().numpy()
    assert efg.knn_stats().list_queries == 0
    assert np.array_equal(out["auto"][0], out["fp32"][0]) and np.array_equal(out["auto"][1], out["fp32"][1])
