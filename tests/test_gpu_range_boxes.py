"""RangeSearch and PickSearch on FP64 trees with FP32 tests against the one-query-per-thread kernels with exact
tests: equal ids, for boxes and queries on common lattice values and an ulp either side of them."""
import numpy as np
import pytest

import octree_gb300 as otg

pytestmark = pytest.mark.gpu


def nudge(rng, x):
    k = rng.random(x.shape)
    return np.where(k < 0.25, np.nextafter(x, np.inf), np.where(k < 0.5, np.nextafter(x, -np.inf), x))


def check(t, ranges, points, **kw):
    for mode in (otg.RANGE_INSIDE, otg.RANGE_OVERLAP):
        a, b = t.range_search(ranges, mode, **kw), t.range_search(ranges, mode, algo=otg.ALGO_PLAIN_FP64, **kw)
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]), (mode, kw)
    a, b = t.pick_search(points, **kw), t.pick_search(points, algo=otg.ALGO_PLAIN_FP64, **kw)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]), ("pick", kw)


@pytest.mark.parametrize("shift", [0.0, -1e3, 2.0**20, 1e9])
@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e4])
@pytest.mark.parametrize("kind", ["boxes", "regular_boxes", "points"])
def test_lattice(kind, scale, shift):
    rng = np.random.default_rng(103)
    lo = rng.integers(0, 24, (3000, 3)) * scale + shift
    ent = nudge(rng, lo) if kind == "points" else nudge(rng, np.concatenate([lo, lo + rng.integers(0, 4, (3000, 3)) * scale], 1))
    if kind != "points":
        ent = np.concatenate([np.minimum(ent[:, :3], ent[:, 3:]), np.maximum(ent[:, :3], ent[:, 3:])], 1)
    space = np.array([[*(np.full(3, shift) - 3 * scale), *(np.full(3, shift) + 33 * scale)]])
    t = otg.Tree(kind).create(ent, max_depth=5, max_elements=12, box=space)
    r = rng.integers(-1, 26, (400, 3)) * scale + shift
    ranges = nudge(rng, np.concatenate([r, r + rng.integers(0, 9, (400, 3)) * scale], 1))
    ranges[:3] = np.array([*(np.full(3, shift) - 9 * scale), *(np.full(3, shift) + 90 * scale)])
    points = nudge(rng, rng.integers(0, 28, (400, 3)) * scale + shift)
    points[:100] = ent[:100, :3]
    for kw in ({}, {"tol": 0.0}, {"tol": 0.5 * scale}, {"tol": 1e-9 * scale}):
        check(t, ranges, points, **kw)


@pytest.mark.parametrize("kind", ["boxes", "points"])
def test_random_and_other_geometry(kind):
    rng = np.random.default_rng(107)
    c, h = rng.random((20_000, 3)) * 60, rng.random((20_000, 3))
    ent = c if kind == "points" else np.concatenate([c - h, c + h], 1)
    t = otg.Tree(kind).create(ent, max_depth=7, max_elements=16)
    q, e = rng.random((600, 3)) * 60, rng.random((600, 3)) * 6
    q[:20] = 1e30
    ranges = np.concatenate([q - e, q + e], 1)
    check(t, ranges, q)
    check(t, ranges, ent[:600, :3])
    if kind == "boxes":
        t.set_entities(ent[rng.permutation(len(ent))])
        check(t, ranges, q)
