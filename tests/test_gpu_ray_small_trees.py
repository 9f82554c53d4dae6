"""First hits on point trees of about the size, and in batches of about the number of rays, from which one ray takes a
thread instead of a warp: against a forest's trees one by one in small batches."""
import numpy as np
import pytest

import octree_gb300 as otg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per", [1, 15, 16, 17, 31, 32, 33])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_forest(dtype, per):
    rng = np.random.default_rng(137)
    trees, rays = 64, 64
    p = (rng.random((trees * per, 3)) * 4).astype(dtype)
    f = otg.Forest("points", dtype).create(p, np.arange(trees + 1, dtype=np.uint64) * per, max_depth=4, max_elements=8)
    d = rng.normal(size=(trees * rays, 3))
    r = np.concatenate([rng.random((trees * rays, 3)) * 4, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(dtype)
    off, ids, dist = f.ray_first(r, np.arange(trees + 1, dtype=np.uint64) * rays, tol=0.3, tol_increment=0.01)  # 4096 rays
    assert len(ids) > 0
    for i in range(trees):
        a, b = i * rays, (i + 1) * rays
        t = otg.Tree("points", dtype).create(p[i * per : (i + 1) * per], max_depth=4, max_elements=8)
        o, k, e = t.ray_first(r[a:b], tol=0.3, tol_increment=0.01)
        s = slice(int(off[a]), int(off[b]))
        assert np.array_equal(off[a : b + 1] - off[a], o) and np.array_equal(ids[s], k) and np.array_equal(dist[s], e)
