"""Frusta of about and above the planes that the FP32 tests take, against the exact kernels: equal ids."""
import numpy as np
import pytest

import octree_gb300 as otg
from test_gpu_planes import entities, queries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind", ["points", "boxes"])
def test_many_planes(kind, dtype):
    """Frusta of more planes than the FP32 tests take: the planes after them decide too."""
    rng = np.random.default_rng(59)
    ent = entities(rng, kind, 3000, 1.0, 0.0).astype(dtype)
    t = otg.Tree(kind, dtype).create(ent, max_depth=6, max_elements=16)
    for per in (8, 31, 32, 33, 40):
        p = queries(rng, ent, 24, per, False)
        p[:, :, 0] = -3 - 12 * rng.random((24, per))  # planes that cut little: the last ones cut most
        p[:, :, 0] += (p[:, :, 1:] * 10).sum(2)
        last = queries(rng, ent, 24, 1, True)[:, 0]
        p[:12, -1] = last[:12]
        for kw in ({}, {"tol": 0.25}):
            a, b = t.frustum_culling(p, **kw), t.frustum_culling(p, algo=otg.ALGO_PLAIN_FP64, **kw)
            assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]), (per, kw)
            assert len(a[1]) > 0
