"""A search captured in a caller's CUDA graph when nothing has searched in FP32 before: the byte rows of the
base, which are made on first use, are not made inside the capture."""
import numpy as np
import pytest

from efanna_gb300 import datasets

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_first_fp32_search_inside_a_capture(efg, tmp_path):
    n, d, nq = 5_000, 64, 70
    x = datasets.mixture_u8(n, d, seed=2)
    q = datasets.mixture_u8(nq, d, seed=2, queries=True)
    built = efg.Index(x, efg.IndexParams(trees=4, merge_level=3, epochs=3, check=25, L=30, K=10, S=10))
    built.build_index()
    built.save_trees(str(tmp_path / "t"))
    built.save_graph(str(tmp_path / "g"))
    built.set_search_params(3, 400, 80, 4)
    want = built.knn_search(10, q)
    idx = efg.Index(x, efg.IndexParams(trees=4))
    idx.load_trees(str(tmp_path / "t"))
    idx.load_graph(str(tmp_path / "g"))
    idx.set_search_params(3, 400, 80, 4)
    Q = torch.from_numpy(q).cuda()
    out = torch.full((nq, 10), -7, dtype=torch.int32, device="cuda")
    idx.set_search_precision("bf16")  # a warm-up that allocates the search's scratch
    idx.knn_search_device(10, Q.data_ptr(), nq, d, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    idx.set_search_precision("fp32")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        idx.knn_search_device(10, Q.data_ptr(), nq, d, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        out.fill_(-7)
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want)
    assert np.array_equal(idx.knn_search(10, q), want)  # (over byte rows from here on)
    graph.replay()
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), want)
