"""Builds with little device memory left: where the join's buckets and overflow list do not fit, its
records are counted first and written to their places by a second run, and the graph is the same."""
import numpy as np
import pytest

from efanna_gb300 import datasets

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("data,precision", [("bytes", "fp32"), ("gauss", "fp32"), ("gauss", "bf16")])
def test_build_with_little_memory(efg, data, precision):
    n, d = 100_000, 96
    if data == "bytes":
        x = datasets.mixture_u8(n, d, seed=1)
    else:
        x = (np.random.default_rng(1).standard_normal((n, d)) * np.arange(1, d + 1) ** -0.35).astype(np.float32)
    X = torch.from_numpy(x).cuda()
    graphs = []
    for left in (None, 2.25):  # GB left to the build; buckets, list and hub records together want three
        idx = efg.Index.from_device(X.data_ptr(), n, d, d, efg.IndexParams(
            K=100, L=200, check=200, S=10, trees=8, merge_level=6, epochs=3))
        idx.set_build_precision(precision)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        ballast = None
        if left:
            ballast = torch.empty(torch.cuda.mem_get_info()[0] - int(left * 2 ** 30), dtype=torch.uint8, device="cuda")
        try:
            idx.build_index()
            graphs.append(idx.graph())
        finally:
            del ballast
            idx.close()
            torch.cuda.empty_cache()
    assert np.array_equal(graphs[0], graphs[1])
