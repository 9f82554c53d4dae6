"""Queries where the device has little room for scratch: the stream-ordered pool is one of a fixed size."""
import contextlib
import ctypes as C

import numpy as np
import pytest

import octree_gb300 as otg

pytestmark = pytest.mark.gpu


class _Props(C.Structure):
    _fields_ = [("alloc", C.c_int), ("handles", C.c_int), ("location", C.c_int), ("device", C.c_int), ("win32", C.c_void_p),
                ("max_size", C.c_size_t), ("usage", C.c_ushort), ("reserved", C.c_ubyte * 54)]


@contextlib.contextmanager
def pool_of(size):
    """The device's current memory pool is a new one of at most `size` bytes."""
    cuda = C.CDLL("libcuda.so.1")
    dev, old, pool = C.c_int(), C.c_void_p(), C.c_void_p()
    assert cuda.cuDeviceGet(C.byref(dev), 0) == 0 and cuda.cuDeviceGetMemPool(C.byref(old), dev) == 0
    props = _Props(alloc=1, location=1, device=0, max_size=size)  # pinned, on the device
    assert cuda.cuMemPoolCreate(C.byref(pool), C.byref(props)) == 0
    assert cuda.cuDeviceSetMemPool(dev, pool) == 0
    try:
        yield
    finally:
        assert cuda.cuDeviceSetMemPool(dev, old) == 0 and cuda.cuMemPoolDestroy(pool) == 0


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_small_results(dtype):
    rng = np.random.default_rng(113)
    c = rng.random((20_000, 3)) * 100
    t = otg.Tree("boxes", dtype).create(np.concatenate([c - 0.1, c + 0.1], 1).astype(dtype), max_depth=7, max_elements=16)
    q = rng.random((4096, 3)) * 100
    ranges = np.concatenate([q - 1, q + 1], 1)
    d = rng.normal(size=(4096, 3))
    rays = np.concatenate([q, d / np.linalg.norm(d, axis=1, keepdims=True)], 1)
    calls = [lambda: t.range_search(ranges, 1), lambda: t.pick_search(q), lambda: t.ray_all(rays, max_distance=5.0), lambda: t.ray_first(rays)]
    want = [f() for f in calls]
    with pool_of(32 << 20):
        for f, w in zip(calls, want):
            assert all(np.array_equal(a, b) for a, b in zip(f(), w) if b is not None)
    assert sum(len(w[1]) for w in want) > 1000


def test_collisions():
    rng = np.random.default_rng(127)
    c, h = rng.random((1_000_000, 3)) * 100, 0.5 * (0.5 + rng.random((1_000_000, 3)))
    t = otg.Tree("boxes").create(np.concatenate([c - h, c + h], 1), max_depth=8, max_elements=20)
    want = t.collision_self()
    assert len(want) > 2_000_000
    with pool_of(160 << 20):
        assert np.array_equal(t.collision_self(), want)


def test_insert():
    """The new arrays are as large as the tree, not as the bound that a Create sizes its own by."""
    rng = np.random.default_rng(131)
    p, q = rng.random((1_000_000, 3)), rng.random((200_000, 3))
    box = np.array([[0.0, 0, 0, 1, 1, 1]])
    for limit in (1 << 30, 96 << 20):
        t = otg.Tree("points").create(p, max_depth=8, max_elements=20, box=box)
        with pool_of(limit):
            t.insert(q)
            off, ids, dist = t.knn(q[:100], 1)
            del t
        assert (dist == 0).all()
