"""Ray kernels with FP32 tests against the one-ray-per-thread kernels, which test every box exactly in
the tree's scalar type and walk RayIntersectedFirst's updates in order: the results are equal, ids and
distances bit for bit."""
import numpy as np
import pytest

import octree_gb300 as otg

pytestmark = pytest.mark.gpu


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def both(t, rays, **kw):
    for fn in (t.ray_all, t.ray_first):
        assert same(fn(rays, **kw), fn(rays, algo=otg.ALGO_PLAIN_FP64, **kw)), (fn.__name__, kw)


def directions(rng, n, kind):
    if kind == "axis":
        d = np.zeros((n, 3))
        d[np.arange(n), rng.integers(0, 3, n)] = rng.choice([-1.0, 1.0], n)
        return d
    d = rng.normal(size=(n, 3))
    if kind == "plane":
        d[np.arange(n), rng.integers(0, 3, n)] = 0.0
    if kind == "nearly":
        d[np.arange(n), rng.integers(0, 3, n)] *= 10.0 ** rng.uniform(-17, -5, n)
    return d / np.linalg.norm(d, axis=1, keepdims=True)


TOLERANCES = [{}, {"tol": 0.0}, {"tol": 0.25}, {"tol": 0.01, "tol_increment": 0.125}, {"tol": 0.01, "tol_increment": 3.0},
              {"max_distance": 7.5}, {"max_distance": 0.0}, {"tol": 0.5, "max_distance": 3.0}]


@pytest.mark.parametrize("kw", TOLERANCES, ids=[str(i) for i in range(len(TOLERANCES))])
@pytest.mark.parametrize("kind", ["random", "axis", "plane", "nearly"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_random_boxes(dtype, kind, kw):
    """Enough rays for the FP32 images (a few entity tests per entity); every third ray starts on a box corner."""
    rng = np.random.default_rng(23)
    n, nr = 3001, 401
    c, h = rng.random((n, 3)) * 20, 0.05 + rng.random((n, 3))
    b = np.concatenate([c - h, c + h], 1)
    t = otg.Tree("boxes", dtype).create(b, max_depth=6, max_elements=16)
    o = rng.random((nr, 3)) * 24 - 2
    o[::3] = b[rng.integers(0, n, len(o[::3])), 3:]
    both(t, np.concatenate([o, directions(rng, nr, kind)], 1), **kw)


@pytest.mark.parametrize("shift", [0.0, 1e3, 2.0**20, 1e9])
@pytest.mark.parametrize("scale", [1e-3, 1.0, 1e5])
def test_faces_within_rounding(shift, scale):
    """Lattice boxes that touch, rays along and within an ulp of their faces: the FP32 bounds cannot decide them."""
    rng = np.random.default_rng(29)
    g = np.stack(np.meshgrid(*[np.arange(12)] * 3, indexing="ij"), -1).reshape(-1, 3) * scale + shift
    b = np.concatenate([g, g + scale], 1)
    t = otg.Tree("boxes").create(b, max_depth=6, max_elements=8)
    nr = 600
    o = rng.integers(0, 13, (nr, 3)) * scale + shift
    o = np.where(rng.random((nr, 3)) < 0.3, np.nextafter(o, np.inf), np.where(rng.random((nr, 3)) < 0.3, np.nextafter(o, -np.inf), o))
    d = np.concatenate([directions(rng, 200, "axis"), directions(rng, 200, "plane"), directions(rng, 200, "nearly")])
    for kw in ({}, {"tol": 0.0}, {"tol": 0.3 * scale}):
        both(t, np.concatenate([o, d], 1), **kw)


@pytest.mark.parametrize("copies", [64, 128, 129, 700])
def test_many_candidates(copies):
    """Equal and nested boxes: candidate buffers at and above their 128 entries, and equal exits."""
    rng = np.random.default_rng(31)
    c = rng.random((6, 3)) * 10
    b = np.concatenate([np.repeat(np.concatenate([c - 1, c + 1], 1), copies, 0), np.concatenate([c - 2, c + 1], 1)])
    b = b[rng.permutation(len(b))]
    for dtype in (np.float64, np.float32):
        t = otg.Tree("boxes", dtype).create(b, max_depth=5, max_elements=16)
        o = rng.random((500, 3)) * 12 - 1
        for kw in ({}, {"tol": 0.125}):
            both(t, np.concatenate([o, directions(rng, 500, "random")], 1), **kw)


def test_points_and_other_geometry():
    """Point trees, and a box tree whose entities left their nodes, take the walk in its own order."""
    rng = np.random.default_rng(37)
    p = rng.random((4000, 3)) * 10
    rays = np.concatenate([rng.random((300, 3)) * 10, directions(rng, 300, "random")], 1)
    both(otg.Tree("points").create(p, max_depth=6, max_elements=16), rays, tol=0.3)
    b = np.concatenate([p - 0.2, p + 0.2], 1)
    t = otg.Tree("boxes").create(b, max_depth=6, max_elements=16)
    both(t, rays)
    t.set_entities(b[rng.permutation(len(b))])
    both(t, rays, tol=0.01)


def test_edge_rays():
    """Rays that are not normalised, not finite or far away; boxes that reach far out of the space."""
    rng = np.random.default_rng(41)
    c = rng.random((2000, 3)) * 10
    b = np.concatenate([c - 0.3, c + 0.3], 1)
    d = directions(rng, 400, "random")
    o = rng.random((400, 3)) * 10
    o[:40] *= 1e30
    o[40:60, 0] = 1e200
    d[60:80] *= 2.0
    d[80:85] = np.nan
    o[85:90, 1] = np.inf
    t = otg.Tree("boxes").create(b, max_depth=6, max_elements=16)
    both(t, np.concatenate([o, d], 1))
    b[:3, 3:] = 1e6
    t = otg.Tree("boxes").create(b, max_depth=6, max_elements=16, box=np.array([[0, 0, 0, 10, 10, 10.0]]))
    both(t, np.concatenate([o, d], 1))
