"""The record buffers of the NN-descent join are sized for the join that runs: none of a build's joins
finds its overflow list too short and runs again, with byte rows and float rows, in FP32 and on the tensor
cores (whose first join runs in one piece where the distances are not exact)."""
import numpy as np
import pytest

from efanna_gb300 import datasets

pytestmark = pytest.mark.gpu

G10 = dict(K=10, L=30, check=25, S=10, trees=8, merge_level=6, epochs=3)
G20 = dict(K=20, L=40, check=25, S=10, trees=8, merge_level=6, epochs=3)
G32 = dict(K=32, L=40, check=40, S=10, trees=8, merge_level=6, epochs=3)
SMALL = dict(K=10, L=30, check=25, S=10, trees=4, merge_level=4, epochs=3)
L60 = dict(K=20, L=60, check=60, S=15, trees=8, merge_level=6, epochs=3)
G100 = dict(K=100, L=200, check=200, S=10, trees=8, merge_level=6, epochs=3)


def _rows(data, n, d):
    if data == "bytes":
        return datasets.mixture_u8(n, d, seed=d)
    if data == "unit":
        return datasets.mixture_unit(n, d, block=16, seed=d)
    rng = np.random.default_rng(d)
    return (rng.standard_normal((n, d)) * np.arange(1, d + 1) ** -0.35).astype(np.float32)


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("data,n,d", [("bytes", 20_011, 128), ("gauss", 20_011, 100), ("unit", 12_345, 192)])
@pytest.mark.parametrize("params", [G10, G20, G32, SMALL, L60, G100], ids=["g10", "g20", "g32", "small", "l60", "g100"])
def test_no_join_runs_again(efg, data, n, d, params, precision):
    idx = efg.Index(_rows(data, n, d), efg.IndexParams(**params))
    idx.set_build_precision(precision)
    idx.build_index()
    assert idx.build_stats().join_reruns == 0
