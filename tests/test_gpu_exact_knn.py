"""The exact k-NN with its screening on the tensor cores (tcgen05 BF16 Gram tiles, FP32
accumulation, then the FP64 re-rank) against the FP32 CUDA-core screening and against numpy.

On byte-valued data BF16 holds every value and every FP32 partial sum of the Gram form is an
exact integer, so both screenings keep the same survivors and the results must be bit-identical.
On general float data the tensor-core path splits each value into hi + lo BF16 parts; the ids
after the FP64 re-rank must still be the exact ones."""
import numpy as np
import pytest

from efanna_gb300 import datasets

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _knn(efg, x, q, k, screening, exclude=False, first_row=0, stride=None, qstride=None, stream=0):
    n, d = x.shape
    ld = stride or (d + 3) // 4 * 4   # rows start on 16-byte boundaries
    qld = qstride or (d + 3) // 4 * 4
    xp = np.zeros((n, ld), np.float32)
    xp[:, :d] = x
    qp = np.zeros((q.shape[0], qld), np.float32)
    qp[:, :d] = q
    X, Q = torch.from_numpy(xp).cuda(), torch.from_numpy(qp).cuda()
    ids = torch.full((q.shape[0], k), -7, dtype=torch.int32, device="cuda")
    dist = torch.full((q.shape[0], k), -1.0, dtype=torch.float32, device="cuda")
    efg.brute_force_knn_device(X.data_ptr(), n, d, ld, Q.data_ptr(), q.shape[0], qld, k, ids.data_ptr(),
                               dist.data_ptr(), exclude_self=exclude, first_row=first_row, stream=stream,
                               screening=screening)
    torch.cuda.synchronize()
    return ids.cpu().numpy(), dist.cpu().numpy()


def _numpy_exact(x, q, k, exclude_rows=None):
    xd, qd = x.astype(np.float64), q.astype(np.float64)
    D = ((qd[:, None, :] - xd[None, :, :]) ** 2).sum(2)
    if exclude_rows is not None:
        D[np.arange(len(q)), exclude_rows] = np.inf
    order = np.lexsort((np.broadcast_to(np.arange(len(x)), D.shape), D), axis=1)[:, :k]
    return order.astype(np.int32), np.take_along_axis(D, order, 1)


@pytest.mark.parametrize("d", [1, 3, 32, 64, 100, 128, 200, 960])
@pytest.mark.parametrize("k", [1, 10, 100])
def test_tensor_core_equals_fp32_on_byte_data(efg, d, k):
    n, nq = 3000 + 77, 300
    x = datasets.mixture_u8(n, d, seed=d) if d >= 8 else np.random.default_rng(d).integers(0, 256, (n, d)).astype(
        np.float32)
    q = datasets.mixture_u8(nq, d, seed=d, queries=True) if d >= 8 else \
        np.random.default_rng(d + 1).integers(0, 256, (nq, d)).astype(np.float32)
    tc = _knn(efg, x, q, k, "auto")
    f32 = _knn(efg, x, q, k, "fp32")
    assert np.array_equal(tc[0], f32[0]) and np.array_equal(tc[1], f32[1])
    if d <= 128:
        ref_ids, ref_d = _numpy_exact(x, q, k)
        assert np.array_equal(tc[0], ref_ids)
        assert np.array_equal(tc[1], ref_d.astype(np.float32))


def test_split_form_on_byte_data_equals_plain(efg):
    x = datasets.mixture_u8(5000, 128, seed=3)
    q = datasets.mixture_u8(257, 128, seed=3, queries=True)
    plain = _knn(efg, x, q, 10, "auto")
    split = _knn(efg, x, q, 10, "split")
    assert np.array_equal(plain[0], split[0]) and np.array_equal(plain[1], split[1])


def test_exclude_self_strides_and_stream(efg):
    """exclude_self with a non-zero first row, padded row strides (dim 33 in rows of 36 floats) and
    a call on a non-default stream: identical to the FP32 screening and to numpy."""
    x = datasets.mixture_u8(4000, 33, seed=8)
    rows = np.arange(1500, 1500 + 400)
    s = torch.cuda.Stream()
    tc = _knn(efg, x, x[rows], 12, "auto", exclude=True, first_row=1500, stride=36, qstride=40,
              stream=s.cuda_stream)
    f32 = _knn(efg, x, x[rows], 12, "fp32", exclude=True, first_row=1500, stride=36, qstride=40)
    ref_ids, _ = _numpy_exact(x, x[rows], 12, exclude_rows=rows)
    assert np.array_equal(tc[0], f32[0]) and np.array_equal(tc[1], f32[1])
    assert np.array_equal(tc[0], ref_ids)
    assert not np.any(tc[0] == rows[:, None])


@pytest.mark.parametrize("gen,d", [("unit", 960), ("unit", 128), ("gauss", 96)])
def test_tensor_core_split_ids_exact_on_float_data(efg, gen, d):
    """Float data (the d = 960 unit-block generator; a Gaussian at d = 96): the split BF16 screening
    keeps the true neighbours among its survivors, so the ids after the FP64 re-rank equal numpy's
    exact FP64 order, and so do the FP32 screening's."""
    n, nq, k = 6000, 200, 100 if d == 960 else 10
    if gen == "unit":
        x = datasets.mixture_unit(n, d, block=16, seed=2)
        q = datasets.mixture_unit(nq, d, block=16, seed=2, queries=True)
    else:
        rng = np.random.default_rng(4)
        x = rng.standard_normal((n, d)).astype(np.float32)
        q = rng.standard_normal((nq, d)).astype(np.float32)
    tc = _knn(efg, x, q, k, "auto")
    ref_ids, ref_d = _numpy_exact(x, q, k)
    f32 = _knn(efg, x, q, k, "fp32")
    assert np.array_equal(tc[0], ref_ids)
    assert np.array_equal(tc[0], f32[0])
    assert np.allclose(tc[1], ref_d, rtol=1e-6, atol=0)


def test_tensor_core_full_size_equals_fp32(efg):
    """The benchmark's ground truth: 1M x 128 byte-valued base, 2,000 held-out queries, k = 10."""
    x = datasets.mixture_u8(1_000_000, 128, seed=0)
    q = datasets.mixture_u8(2000, 128, seed=0, queries=True)
    X, Q = torch.from_numpy(x).cuda(), torch.from_numpy(q).cuda()
    out = {}
    for screening in ("auto", "fp32"):
        ids = torch.zeros((2000, 10), dtype=torch.int32, device="cuda")
        dist = torch.zeros((2000, 10), dtype=torch.float32, device="cuda")
        efg.brute_force_knn_device(X.data_ptr(), 1_000_000, 128, 128, Q.data_ptr(), 2000, 128, 10, ids.data_ptr(),
                                   dist.data_ptr(), screening=screening)
        torch.cuda.synchronize()
        out[screening] = (ids.cpu().numpy(), dist.cpu().numpy())
    assert np.array_equal(out["auto"][0], out["fp32"][0])
    assert np.array_equal(out["auto"][1], out["fp32"][1])


@pytest.mark.parametrize("n,nq,k", [(129, 1, 104), (20_000, 3, 100), (33_001, 130, 104), (70_000, 300, 60)])
def test_few_queries_over_many_chunks(efg, n, nq, k):
    """A few queries with long lists: the base is cut into more chunks than 4096 keys per query would
    allow (one tile of rows at the least); byte data, so ids and distances equal the FP32 screening's."""
    x = datasets.mixture_u8(n, 40, seed=3)
    q = datasets.mixture_u8(nq, 40, seed=3, queries=True)
    tc = _knn(efg, x, q, k, "auto")
    f32 = _knn(efg, x, q, k, "fp32")
    assert np.array_equal(tc[0], f32[0]) and np.array_equal(tc[1], f32[1])


@pytest.mark.parametrize("n,nq,k,excl", [(17, 5, 1, False), (130, 260, 20, True), (543, 129, 10, False),
                                         (544, 64, 10, False), (2063, 257, 104, True), (2100, 1100, 104, False),
                                         (30_000, 900, 10, True), (130_000, 300, 104, False)])
@pytest.mark.parametrize("d", [5, 129, 300])
def test_bound_passes_at_their_edges(efg, n, nq, k, excl, d):
    """No bound, a bound from groups of 16 columns, of 64 and of whole tiles of the base, and from a sample;
    one and two query tiles per item, resident and streamed (d = 300 in the split form)."""
    rng = np.random.default_rng(n + d)
    x = rng.integers(0, 256, (n, d)).astype(np.float32)
    nq = min(nq, n) if excl else nq
    q = x[:nq].copy() if excl else rng.integers(0, 256, (nq, d)).astype(np.float32)
    k = min(k, n - 1)
    for screening in ("auto", "split"):
        tc = _knn(efg, x, q, k, screening, exclude=excl)
        f32 = _knn(efg, x, q, k, "fp32", exclude=excl)
        assert np.array_equal(tc[0], f32[0]) and np.array_equal(tc[1], f32[1])


@pytest.mark.parametrize("n", [3000, 60_000])
def test_many_equal_distances(efg, n):
    """More rows at one distance than a candidate buffer holds: the lists take the call."""
    x = np.zeros((n, 8), np.float32)
    x[::7, 3] = 1.0
    q = np.zeros((200, 8), np.float32)
    q[::2, 0] = 2.0
    tc = _knn(efg, x, q, 12, "auto")
    ref_ids, ref_d = _numpy_exact(x, q[:2], 12)
    for i in range(200):
        assert np.array_equal(tc[0][i], ref_ids[i % 2]) and np.array_equal(tc[1][i], ref_d[i % 2])


@pytest.mark.parametrize("n,nq", [(330_000, 4000), (520_000, 2000), (1_000_000, 3000)])
def test_long_lists_over_large_bases(efg, n, nq):
    """k = 100 over bases whose sample is cut or whose groups are doubled; ids and distances equal the FP32
    screening's, and the call does not end in the lists."""
    import torch
    x = torch.randint(0, 256, (n, 16), device="cuda", dtype=torch.int32).float()
    q = torch.randint(0, 256, (nq, 16), device="cuda", dtype=torch.int32).float()
    out = {}
    for screening in ("fp32", "auto"):
        ids = torch.zeros((nq, 100), dtype=torch.int32, device="cuda")
        dist = torch.zeros((nq, 100), dtype=torch.float32, device="cuda")
        efg.brute_force_knn_device(x.data_ptr(), n, 16, 16, q.data_ptr(), nq, 16, 100, ids.data_ptr(),
                                   dist.data_ptr(), screening=screening)
        torch.cuda.synchronize()
        out[screening] = (ids.cpu().numpy(), dist.cpu().numpy())
    assert efg.knn_stats().convert_ms > 0.05  # (the lists' rerun has nothing left to convert)
    assert np.array_equal(out["auto"][0], out["fp32"][0])
    assert np.array_equal(out["auto"][1], out["fp32"][1])
