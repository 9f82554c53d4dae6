"""CollisionDetection by packets against the one-box-per-thread kernel with exact tests: equal pair lists,
at packet and run-length edges, for touching, nested and far boxes and for other geometry."""
import numpy as np
import pytest

import octree_gb300 as otg

pytestmark = pytest.mark.gpu


def check(a, b=None, **kw):
    if b is None:
        x, y = a.collision_self(**kw), a.collision_self(algo=otg.ALGO_PLAIN_FP64, **kw)
    else:
        x, y = a.collision_pair(b, **kw), a.collision_pair(b, algo=otg.ALGO_PLAIN_FP64, **kw)
    assert x.shape == y.shape and np.array_equal(x, y), kw
    return len(x)


def boxes(rng, n, side, lo, hi):
    c, h = rng.random((n, 3)) * side, rng.uniform(lo, hi, (n, 3))
    return np.concatenate([c - h, c + h], 1)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 65, 1000, 20_011])
def test_sizes(n, dtype):
    rng = np.random.default_rng(61)
    side = 2.0 * n ** (1 / 3)
    t = otg.Tree("boxes", dtype).create(boxes(rng, n, side, 0.1, 1.2), max_depth=7, max_elements=8)
    u = otg.Tree("boxes", dtype).create(boxes(rng, max(1, n // 3), side, 0.1, 2.0), max_depth=5, max_elements=20)
    for kw in ({}, {"tol": 0.0}, {"tol": 0.3}):
        check(t, **kw)
        check(t, u, **kw)
        check(u, t, **kw)


@pytest.mark.parametrize("shift", [0.0, 1e3, 2.0**20, -3e7])
@pytest.mark.parametrize("kind", ["boxes", "regular_boxes"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_touching_and_nearly(dtype, kind, shift):
    """Lattice boxes that touch, and boxes an ulp or two apart or deep."""
    rng = np.random.default_rng(67)
    g = np.stack(np.meshgrid(*[np.arange(14)] * 3, indexing="ij"), -1).reshape(-1, 3) + shift
    b = np.concatenate([g, g + 1], 1).astype(dtype)
    k = rng.random(b.shape)
    b = np.where(k < 0.2, np.nextafter(b, dtype(np.inf)), np.where(k < 0.4, np.nextafter(b, dtype(-np.inf)), b)).astype(dtype)
    space = np.array([[*(np.full(3, shift) - 8), *(np.full(3, shift) + 24)]])
    t = otg.Tree(kind, dtype).create(b, max_depth=6, max_elements=8, box=space)
    u = otg.Tree(kind, dtype).create(b[rng.permutation(len(b))[:900]], max_depth=6, max_elements=8, box=space)
    for kw in ({}, {"tol": 0.0}, {"tol": 0.25}):
        check(t, **kw)
        check(t, u, **kw)


@pytest.mark.parametrize("wide", [200, 1100])
def test_long_runs_and_large_boxes(wide):
    """A few boxes over everything: runs of pairs up to and above the counted order's limit, long walks one by one."""
    rng = np.random.default_rng(71)
    n = 3000
    b = boxes(rng, n, 40.0, 0.05, 0.4)
    b[:3] = [-1, -1, -1, 41, 41, 41]
    b[3 : 3 + wide] = boxes(rng, wide, 4.0, 2.0, 3.0)
    b = b[rng.permutation(n)]
    t = otg.Tree("boxes").create(b, max_depth=8, max_elements=16)
    assert check(t) > n
    check(t, otg.Tree("boxes").create(boxes(rng, 500, 40.0, 0.05, 6.0), max_depth=8, max_elements=16))


def test_few_pairs():
    """Fewer pairs than a quarter of the boxes: the radix order; and none."""
    rng = np.random.default_rng(73)
    t = otg.Tree("boxes").create(boxes(rng, 30_000, 100.0, 0.05, 0.3), max_depth=8, max_elements=16)
    assert 0 < check(t) < 30_000 / 4
    far = boxes(rng, 1000, 10.0, 0.1, 0.2) + 500.0
    assert check(t, otg.Tree("boxes").create(far, max_depth=5, max_elements=16)) == 0


def test_other_geometry():
    """After set_entities the pairs found are those whose box enters the other's node: both kernels walk the
    larger tree from the smaller, left one's boxes."""
    rng = np.random.default_rng(79)
    b = boxes(rng, 5000, 30.0, 0.1, 0.8)
    t = otg.Tree("boxes").create(b, max_depth=6, max_elements=16)
    u = otg.Tree("boxes").create(boxes(rng, 2000, 30.0, 0.1, 0.8), max_depth=6, max_elements=16)
    check(u, t)
    t.set_entities(b + 0.01)
    check(u, t)
    t.set_entities(b[rng.permutation(len(b))])
    check(u, t)
