"""Filtered kNN at the sizes where its order and its slots change: buffers of 32, 64 and 128 candidates, subtrees
tested whole, ties (more than k results), fewer points than k; against the one-query-per-thread kernels."""
import numpy as np
import pytest

import octree_gb300 as otg

pytestmark = pytest.mark.gpu


def check(t, q, k, **kw):
    a, b = t.knn(q, k, **kw), t.knn(q, k, algo=otg.ALGO_PLAIN_FP64, **kw)
    assert all(np.array_equal(x, y) for x, y in zip(a, b)), (k if np.isscalar(k) else "mixed", kw)
    return a


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("k", [1, 31, 32, 33, 63, 64, 65, 112, 113, 128, 129, 240])
def test_sizes(k, dtype):
    rng = np.random.default_rng(83)
    p = rng.random((20_000, 3)) * 100
    t = otg.Tree("points", dtype).create(p, max_depth=8, max_elements=20)
    q = np.concatenate([rng.random((200, 3)) * 100, p[:50], rng.random((20, 3)) * 400 - 150])
    check(t, q, k)
    check(t, q, k, max_distance=6.0)
    check(t, q, np.where(rng.random(len(q)) < 0.2, 0, rng.integers(1, k + 1, len(q))).astype(np.uint32))


@pytest.mark.parametrize("n", [1, 5, 20, 21, 95, 96, 97, 400])
def test_few_points(n):
    """Trees of about the size that is tested whole; k above the point count."""
    rng = np.random.default_rng(89)
    p = rng.random((n, 3)) * 10
    for elems in (1, 20):
        t = otg.Tree("points").create(p, max_depth=5, max_elements=elems)
        for k in (1, 8, 64, 200):
            off, ids, _ = check(t, rng.random((40, 3)) * 12 - 1, k)
            assert len(ids) == 40 * min(k, n)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_ties(dtype):
    """Lattice points and duplicates: results above k, equal keys in the final order."""
    rng = np.random.default_rng(97)
    g = np.stack(np.meshgrid(*[np.arange(16.0)] * 3, indexing="ij"), -1).reshape(-1, 3)
    p = np.concatenate([g, g[::3], g[:40]])[rng.permutation(len(g) + len(g[::3]) + 40)]
    t = otg.Tree("points", dtype).create(p, max_depth=6, max_elements=8)
    q = np.concatenate([g[rng.integers(0, len(g), 100)], g[rng.integers(0, len(g), 100)] + 0.5, rng.random((50, 3)) * 16])
    for k in (1, 7, 20, 60):
        off, ids, _ = check(t, q, k)
        assert len(ids) > len(q) * k
    check(t, q, rng.integers(0, 50, len(q)).astype(np.uint32))


def test_other_geometry_and_outside_points():
    rng = np.random.default_rng(101)
    p = rng.random((5000, 3)) * 100
    q = rng.random((200, 3)) * 100
    check(otg.Tree("points").create(p, max_depth=6, max_elements=20, box=np.array([[20.0, 20, 20, 70, 80, 90]])), q, 9)
    t = otg.Tree("points").create(p, max_depth=6, max_elements=20)
    t.insert(p[:700] * 0.9 + 4)
    check(t, q, 30)
