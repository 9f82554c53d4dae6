"""Plane queries on trees that hold entities with coordinates that are no numbers or infinite (outside the given
space, so the root keeps them): the answers of the exact tests."""
import numpy as np
import pytest

import octree_gb300 as otg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind", ["points", "boxes"])
def test_planes(kind, dtype, bad):
    rng = np.random.default_rng(71)
    n, w = 3000, 3 if kind == "points" else 6
    c = rng.random((n, 3)) * 20
    h = 0.05 + rng.random((n, 3)) * 0.5
    ent = (c if kind == "points" else np.concatenate([c - h, c + h], 1)).astype(dtype)
    odd = rng.permutation(n)[:40]
    ent[odd, rng.integers(0, w, 40)] = bad
    ent[odd[:5]] = bad
    ent[odd[5:10], 0] = -bad
    t = otg.Tree(kind, dtype).create(ent, max_depth=6, max_elements=16, box=np.array([[-1.0, -1, -1, 21, 21, 21]]))
    nrm = rng.normal(size=(48 * 9, 3))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    nrm[::7] = [1, 0, 0]
    nrm[3::7] = [0, -1, 0]
    d = (nrm * rng.random((48 * 9, 3)) * 20).sum(1, keepdims=True)
    for per in (1, 6, 9):
        p = np.concatenate([d, nrm], 1)[: 48 * per].reshape(48, per, 4)
        single = np.ascontiguousarray(p[:, 0])
        for fn, q in ((t.frustum_culling, p), (t.plane_search, single), (t.plane_positive_segmentation, single)):
            for kw in ({}, {"tol": 0.25}):
                a, b = fn(q, **kw), fn(q, algo=otg.ALGO_PLAIN_FP64, **kw)
                assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]), (fn.__name__, per, kw)
