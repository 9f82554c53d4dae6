"""Frustum and plane queries with FP32 tests and untested subtrees against the one-query-per-thread
kernels, which test every node and entity exactly: equal ids."""
import numpy as np
import pytest

import octree_gb300 as otg

pytestmark = pytest.mark.gpu


def unit(rng, n):
    d = rng.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def entities(rng, kind, n, scale, shift):
    c = rng.random((n, 3)) * 20 * scale + shift
    if kind == "points":
        return c
    h = (0.05 + rng.random((n, 3))) * 0.5 * scale
    return np.concatenate([c - h, c + h], 1)


def queries(rng, ent, n, per, aligned):
    """Planes through entity corners or anywhere; aligned ones have faces in common with boxes."""
    nrm = unit(rng, n * per)
    if aligned:
        nrm = np.zeros((n * per, 3))
        nrm[np.arange(n * per), rng.integers(0, 3, n * per)] = rng.choice([-1.0, 1.0], n * per)
    through = ent[rng.integers(0, len(ent), n * per), :3]
    return np.concatenate([(nrm * through).sum(1, keepdims=True), nrm], 1).reshape(n, per, 4)


def check(t, planes, **kw):
    single = np.ascontiguousarray(planes[:, 0])
    for fn, p in ((t.frustum_culling, planes), (t.plane_search, single), (t.plane_positive_segmentation, single)):
        a, b = fn(p, **kw), fn(p, algo=otg.ALGO_PLAIN_FP64, **kw)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]), (fn.__name__, kw)
        # the split shapes hand contained subtrees on as items
        for shape in (4 | 1 << 8, 2 | 2 << 8, 8 | 4 << 8):
            otg.autotune_force_shape(shape)
            try:
                c = fn(p, **kw)
            finally:
                otg.autotune_force_shape(-1)
            assert np.array_equal(c[0], b[0]) and np.array_equal(c[1], b[1]), (fn.__name__, kw, shape)


@pytest.mark.parametrize("scale,shift", [(1.0, 0.0), (1e-3, 1e3), (1e4, -3e5), (1.0, 2.0**24)])
@pytest.mark.parametrize("aligned", [False, True])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind", ["points", "boxes", "regular_boxes"])
def test_planes(kind, dtype, aligned, scale, shift):
    """The largest shift flattens the FP32 boxes, which leaves some of them in no reachable node."""
    rng = np.random.default_rng(43)
    ent = entities(rng, kind, 3000, scale, shift).astype(dtype)
    if kind == "regular_boxes" and aligned and not (dtype == np.float32 and shift == 2.0**24):
        space = np.array([[*(ent[:, :3].min(0) - scale), *(ent[:, 3:].max(0) + scale)]])
        t = otg.Tree(kind, dtype).create(ent, max_depth=6, max_elements=16, box=space)
    else:
        t = otg.Tree("boxes" if kind == "regular_boxes" else kind, dtype).create(ent, max_depth=6, max_elements=16)
    for per in (1, 6, 9) if shift == 0.0 else (1, 6):  # above 8 planes every test is exact
        p = queries(rng, ent, 24, per, aligned)
        for kw in ({}, {"tol": 0.0}, {"tol": 0.25 * scale}):
            check(t, p, **kw)


def test_entities_outside_their_nodes():
    """After set_entities a node says nothing about its entities: every one is tested."""
    rng = np.random.default_rng(47)
    ent = entities(rng, "boxes", 20_000, 1.0, 0.0)
    t = otg.Tree("boxes").create(ent, max_depth=6, max_elements=16)
    p = queries(rng, ent, 24, 6, False)
    check(t, p)
    t.set_entities(ent[rng.permutation(len(ent))])
    check(t, p)


def test_points_outside_the_space():
    rng = np.random.default_rng(53)
    ent = entities(rng, "points", 20_000, 1.0, 0.0)
    t = otg.Tree("points").create(ent, max_depth=6, max_elements=16, box=np.array([[4.0, 4, 4, 15, 15, 15]]))
    for per in (1, 6):
        check(t, queries(rng, ent, 24, per, False))
