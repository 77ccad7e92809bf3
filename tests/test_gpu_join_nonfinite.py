"""The tensor-core join over a base with NaN, infinite and overflowing values: their distances are no
numbers, so their pairs make no records, and the graph is the FP32 join's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [32, 100, 128])
def test_rows_that_are_no_numbers(efg, d):
    n = 4_000
    rng = np.random.default_rng(d)
    x = rng.integers(0, 50, (n, d)).astype(np.float32)  # (squared norms below 2^22: other distances are exact)
    bad = {7: (3, np.nan), 1_001: (slice(None), np.nan), 2_002: (0, np.inf), 2_003: (slice(None), -np.inf),
           3_000: (1, 3e38), 3_998: (slice(None), -2e38), 3_999: (d - 1, 1e25)}
    for row, (cols, value) in bad.items():
        x[row, cols] = value
    graphs = []
    for precision in ("fp32", "bf16"):
        idx = efg.Index(x, efg.IndexParams(trees=4, merge_level=3, epochs=3, check=25, L=30, K=10, S=10))
        idx.set_build_precision(precision)
        idx.build_index()
        graphs.append(idx.graph())
        idx.close()
    assert np.array_equal(graphs[0], graphs[1])
    finite = np.setdiff1d(np.arange(n), list(bad))
    assert not np.isin(graphs[1][finite], list(bad)).any()
