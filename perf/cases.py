"""The work a user has this framework do, as measurable cases: graph builds, graph searches and
exact k-NN through the package's public entry points.

Three families:

* ``build``: rows in device memory -> an Index, its trees, the NN-descent graph, the graph as ids;
* ``search``: queries against an index that holds a graph and search trees (method 0, or method 1,
  "kgraph"), from host rows, from device rows or through a captured SearchPlan;
* ``knn``: the exact k nearest rows with their distances (ground truth, the learned form's traces).

``data`` names the values: ``bytes`` are integers in [0, 255] (SIFT-like descriptors), ``gauss`` a
float mixture with a decaying spectrum (deep descriptors), ``unit`` non-negative blocks that sum to
one (GIST-like).  Sizes and parameters are those of the benchmark and the tests, or lie between them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import efanna_gb300 as E

# graph parameters of the benchmark's workloads
G10 = dict(K=10, L=30, check=25, S=10, trees=8, merge_level=8, epochs=8)
G20 = dict(K=20, L=40, check=25, S=10, trees=8, merge_level=8, epochs=8)
G32 = dict(K=32, L=40, check=40, S=10, trees=8, merge_level=8, epochs=8)
G100 = dict(K=100, L=200, check=200, S=10, trees=8, merge_level=6, epochs=6)
SMALL = dict(K=10, L=30, check=25, S=10, trees=4, merge_level=4, epochs=5)
GRAPH_KEYS = ("K", "L", "check", "S", "trees", "merge_level", "epochs")


def listed():
    return [
        # an interactive lookup: one query, the reference configuration's own setting
        dict(name="search_one", family="search", data="bytes", n=1_000_000, d=128, **G10, entry="host",
             precision="fp32", method=0, search_trees=16, nq=1, k=10, rounds=4, pool=1200, extend=200),
        # the benchmark's search: a large batch at the recall@10 >= 0.95 setting
        dict(name="search_batch", family="search", data="bytes", n=1_000_000, d=128, **G10, entry="device",
             precision="fp32", method=0, search_trees=16, nq=10_000, k=10, rounds=4, pool=4000, extend=750),
        # the same search screened in FP8, from host rows to host ids
        dict(name="search_fp8", family="search", data="bytes", n=1_000_000, d=128, **G10, entry="host",
             precision="fp8", method=0, search_trees=16, nq=10_000, k=10, rounds=4, pool=4000, extend=750),
        # an odd-sized float set served in FP32: ragged rows, a few hundred queries
        dict(name="search_ragged", family="search", data="gauss", n=61_003, d=101, **G32, entry="device",
             precision="fp32", method=0, search_trees=8, nq=777, k=20, rounds=4, pool=1000, extend=100),
        # high-dimensional vectors screened in BF16, 100 neighbours per query
        dict(name="search_wide", family="search", data="unit", n=100_000, d=960, **G100, entry="device",
             precision="bf16", method=0, search_trees=8, nq=2_000, k=100, rounds=6, pool=3000, extend=300),
        # a serving batch through a captured plan: per-query k, pool and extend
        dict(name="search_plan", family="search", data="bytes", n=400_000, d=128, **G20, entry="plan",
             precision="fp32", method=0, search_trees=16, nq=256, k=100, rounds=8, pool=2000, extend=250),
        # the reference's other search method (best-first expansion)
        dict(name="search_kgraph", family="search", data="bytes", n=1_000_000, d=128, **G10, entry="device",
             precision="fp32", method=1, search_trees=16, nq=4_000, k=10, rounds=6, pool=4000, extend=500),
        # the benchmark's graph build
        dict(name="build_1m", family="build", data="bytes", n=1_000_000, d=128, **G10, precision="fp32"),
        # a small odd-sized float set indexed from scratch: launches and allocations count
        dict(name="build_small", family="build", data="gauss", n=20_011, d=100, **SMALL, precision="fp32"),
        # high-dimensional rows, K = 100, the join on the tensor cores (hi + lo products)
        dict(name="build_wide", family="build", data="unit", n=100_000, d=960, **G100, precision="bf16"),
        # the ground truth of the benchmark's queries
        dict(name="knn_truth", family="knn", data="bytes", n=1_000_000, d=128, nq=10_000, k=10),
        # exact neighbours of a few queries in a float set: k = 100, ragged rows
        dict(name="knn_few", family="knn", data="gauss", n=150_001, d=97, nq=300, k=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _rows(rng, data):
    """(n, d) of one set: at most 100M values, 10k to a million rows."""
    d = {"bytes": lambda: rng.choice([24, 32, 64, 96, 100, 127, 128, 192]),
         "gauss": lambda: _log(rng, 24, 200),
         "unit": lambda: 16 * rng.randint(6, 60)}[data]()
    return min(_log(rng, 10_000, 1_000_000), 100_000_000 // d), d


def _graph(rng, n):
    g = dict(SMALL) if n < 60_000 else dict(rng.choice([G10, G20, G32]))
    if n >= 200_000:
        g["epochs"] = rng.randint(5, 8)
    return g


def draw(rng):
    family = rng.choice(["build", "search", "search", "search", "knn"])
    data = rng.choice(["bytes", "bytes", "gauss", "unit"])
    n, d = _rows(rng, data)
    if family == "knn":
        k = rng.choice([1, 10, 10, 50, 100])
        nq = _log(rng, 1, 10_000)
        return dict(family="knn", data=data, n=n, d=d, nq=max(1, min(nq, int(8e11 / (n * d)))), k=k)
    if family == "build":
        return dict(family="build", data=data, n=n, d=d, **_graph(rng, n),
                    precision=rng.choice(["fp32", "fp32", "bf16"]))
    g = _graph(rng, n)
    entry = rng.choice(["host", "device", "device", "plan"])
    method = 1 if entry == "device" and rng.random() < 0.3 else 0
    extend = _log(rng, 40, min(700, 7500 // g["K"]))
    pool = min(int(extend * rng.uniform(4, 9)), 4000)
    k = rng.choice([1, 10, 10, 20, 50])
    return dict(family="search", data=data, n=n, d=d, **g, entry=entry,
                precision="fp32" if method else rng.choice(["fp32", "fp32", "bf16", "fp8"]), method=method,
                search_trees=rng.choice([4, 8, 16]), nq=_log(rng, 1, 8_000 if entry != "plan" else 500),
                k=min(k, extend), rounds=rng.randint(2, 5), pool=max(pool, extend), extend=extend)


def _generate(data, n, d, gen, params):
    """n x d float32 CUDA rows; the mixture's parameters come from ``params``, the draws from ``gen``."""
    if data == "bytes":
        weights, centres, sigma = params
        comp = torch.multinomial(weights, n, replacement=True, generator=gen)
        x = torch.randn((n, d), generator=gen, device="cuda")
        x.mul_(sigma[comp].unsqueeze(1)).add_(centres[comp])
        return x.clamp_(0.0, 255.0).round_()
    if data == "gauss":
        weights, centres, spectrum = params
        comp = torch.multinomial(weights, n, replacement=True, generator=gen)
        x = torch.randn((n, d), generator=gen, device="cuda")
        return x.mul_(spectrum[comp]).add_(centres[comp])
    weights, alpha = params
    out = torch.empty((n, d), dtype=torch.float32, device="cuda")
    for s in range(0, n, 1 << 16):
        e = min(n, s + (1 << 16))
        comp = torch.multinomial(weights, e - s, replacement=True, generator=gen)
        x = torch._standard_gamma(alpha[comp], generator=gen).view(e - s, d // 16, 16)
        out[s:e] = (x / x.sum(dim=2, keepdim=True)).view(e - s, d)
    return out


def _mixture(data, d, gen):
    comps = 64
    weights = torch.rand((comps,), generator=gen, device="cuda") + 0.2
    if data == "bytes":
        centres = torch._standard_gamma(torch.full((comps, d), 0.8, device="cuda"), generator=gen) * 25.0
        return weights, centres, torch.rand((comps,), generator=gen, device="cuda") * 20.0 + 10.0
    if data == "gauss":
        centres = torch.randn((comps, d), generator=gen, device="cuda") * 0.3
        decay = torch.arange(1, d + 1, device="cuda", dtype=torch.float32) ** -0.35
        scale = torch.rand((comps, 1), generator=gen, device="cuda") + 0.5
        order = torch.argsort(torch.rand((comps, d), generator=gen, device="cuda"), dim=1)
        return weights, centres, decay[order] * scale
    return weights, torch._standard_gamma(torch.full((comps, d), 2.0, device="cuda"), generator=gen) + 0.05


def _padded(x):
    """The same rows 16 bytes aligned (a row stride of a multiple of four values), as the k-NN wants them."""
    d = x.shape[1]
    return x if d % 4 == 0 else torch.nn.functional.pad(x, (0, -d % 4))[:, :d]


def _data(case, seed):
    """The base rows and the queries (held-out draws of the same mixture)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    params = _mixture(case["data"], case["d"], gen)
    x = _generate(case["data"], case["n"], case["d"], gen, params)
    q = _generate(case["data"], case["nq"], case["d"], gen, params) if "nq" in case else None
    return _padded(x), q if q is None else _padded(q)


def _index(x, case):
    p = E.IndexParams(**{key: case[key] for key in GRAPH_KEYS})
    return E.Index.from_device(x.data_ptr(), x.shape[0], x.shape[1], x.stride(0), p)


def _plan_params(case, seed):
    """Per-query (rounds, pool, extend, k) of a serving batch, up to the case's own values."""
    rng = np.random.default_rng(seed)
    nq, kmax = case["nq"], case["k"]
    k = rng.choice(np.array([1, 10, 50, 100]), nq).clip(1, kmax)
    extend = np.maximum(rng.integers(case["extend"] // 3 + 1, case["extend"] + 1, nq), k)
    pool = np.minimum((extend * rng.uniform(6.0, 10.0, nq)).astype(np.int64), case["pool"])
    return np.stack([np.full(nq, case["rounds"]), np.maximum(pool, extend), extend, k], 1).astype(np.int32)


def prepare(case, seed):
    x, q = _data(case, seed)
    state = dict(case=case, x=x, q=q)
    if case["family"] == "knn":
        state["ids"] = torch.empty((case["nq"], case["k"]), dtype=torch.int32, device="cuda")
        state["dists"] = torch.empty((case["nq"], case["k"]), dtype=torch.float32, device="cuda")
    elif case["family"] == "search":
        idx = _index(x, case)
        torch.cuda.current_stream().synchronize()
        idx.build_index()
        idx.build_trees(case["search_trees"])
        idx.set_search_precision(case["precision"])
        idx.set_search_params(case["rounds"], case["pool"], case["extend"], case["search_trees"],
                              search_method=case["method"])
        state["index"] = idx
        if case["entry"] == "device":
            state["out"] = torch.empty((case["nq"], case["k"]), dtype=torch.int32, device="cuda")
        else:
            state["q_host"] = np.ascontiguousarray(q.cpu().numpy())
        if case["entry"] == "plan":
            state["params"] = _plan_params(case, seed)
            limits = (case["rounds"], case["pool"], case["extend"], case["k"])
            state["plan"] = idx.search_plan(case["nq"], limits)
    torch.cuda.synchronize()
    return state


def run(state):
    case, x, q = state["case"], state["x"], state["q"]
    if case["family"] == "build":
        idx = _index(x, case)
        idx.set_build_precision(case["precision"])
        idx.build_index()
        graph = idx.graph().view(np.int32)  # ids below 2^30, in the type the search returns them in
        idx.close()
        return graph
    if case["family"] == "knn":
        E.brute_force_knn_device(x.data_ptr(), x.shape[0], x.shape[1], x.stride(0), q.data_ptr(), q.shape[0],
                                 q.stride(0), case["k"], state["ids"].data_ptr(), state["dists"].data_ptr(),
                                 stream=torch.cuda.current_stream().cuda_stream)
        return state["ids"], state["dists"]
    idx = state["index"]
    if case["entry"] == "plan":
        return state["plan"].run(state["q_host"], state["params"])
    if case["method"] == 1:  # this method keeps an enlarged pool: every call starts from its own setting
        idx.set_search_params(case["rounds"], case["pool"], case["extend"], case["search_trees"], search_method=1)
    if case["entry"] == "host":
        return idx.knn_search(case["k"], state["q_host"])
    idx.knn_search_device(case["k"], q.data_ptr(), q.shape[0], q.stride(0), state["out"].data_ptr(),
                          torch.cuda.current_stream().cuda_stream)
    return state["out"]


def work(case):
    n, d = case["n"], case["d"]
    if case["family"] == "build":
        # pairs a join scores: the new and old lists hold up to a few S entries and their reverse ones
        pairs = n * case["epochs"] * 3.0 * case["S"] * (case["S"] + 0.25 * case["L"])
        return {"bytes": 4.0 * n * (d + case["K"]), "flops": 3.0 * d * pairs}
    nq, k = case["nq"], case["k"]
    if case["family"] == "knn":
        return {"bytes": 4.0 * (n + nq) * d + 8.0 * nq * k, "flops": 2.0 * nq * n * d}
    # rows scored per query: the pool, then the unvisited part of the expanded rows
    expanded = case["extend"] * (1 + 0.18 * case["rounds"])
    scored = case["pool"] + 0.28 * expanded * case["K"]
    value = {"fp32": 4, "bf16": 2, "fp8": 1}[case["precision"]]
    rows = min(float(n), nq * scored)
    lists = min(float(n), nq * expanded)
    return {"bytes": rows * d * value + lists * case["K"] * 4.0 + nq * 4.0 * (d + k), "flops": 3.0 * d * nq * scored}


def exact(case, seed):
    """The k-NN distances in 64 bits; a search or a build returns ids alone."""
    if case["family"] != "knn":
        return None
    x, q = _data(case, seed)
    x = x.double()
    xn = (x * x).sum(1)
    k = case["k"]
    out = torch.empty((case["nq"], k), dtype=torch.float64, device="cuda")
    step = max(1, int(2e9 / (8 * case["n"])))
    for s in range(0, case["nq"], step):
        b = q[s:s + step].double()
        # candidates from the Gram form, their distances from the differences themselves
        near = torch.topk(xn - 2.0 * (b @ x.T), min(k + 8, case["n"]), dim=1, largest=False).indices
        for i in range(0, b.shape[0], 64):
            part = b[i:i + 64]
            diff = x[near[i:i + 64]] - part.unsqueeze(1)
            out[s + i:s + i + part.shape[0]] = (diff * diff).sum(2).sort(dim=1).values[:, :k]
    return None, out
