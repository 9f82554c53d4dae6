"""kNN batches that mix queries with no result, fewer than k, exactly k, more (ties), and k beyond the filtered
search, below and above the room for the results after the first k; against the one-query-per-thread kernels."""
import numpy as np
import pytest

import octree_gb300 as otg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nq", [400, 3000])
def test_mixed_counts(dtype, nq):
    rng = np.random.default_rng(103)
    g = np.stack(np.meshgrid(*[np.arange(20.0)] * 3, indexing="ij"), -1).reshape(-1, 3)
    p = np.concatenate([g, 40 + rng.random((6000, 3)) * 20, 80 + rng.random((30, 3))])
    t = otg.Tree("points", dtype).create(p, max_depth=6, max_elements=16)
    q = np.concatenate([g[rng.integers(0, len(g), nq)], 40 + rng.random((nq, 3)) * 20, 80 + rng.random((nq, 3)), 200 + rng.random((50, 3))])
    q = q[rng.permutation(len(q))]
    ks = rng.choice([0, 1, 6, 8, 30, 60, 241], len(q)).astype(np.uint32)
    for k in (8, 40, ks):
        for md in (-1.0, 0.9, 1.5, 4.0):
            a, b = t.knn(q, k, max_distance=md), t.knn(q, k, max_distance=md, algo=otg.ALGO_PLAIN_FP64)
            assert all(np.array_equal(x, y) for x, y in zip(a, b)), (np.isscalar(k), md)
    n = np.diff(a[0].astype(np.int64))
    assert (n == 0).any() and (n > ks).any() and ((n < ks) & (n > 0)).any()
