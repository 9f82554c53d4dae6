"""Canonical order of query results (ids ascending, or (distance, id) ascending) at the run lengths
where the ordering changes: one warp's 32 items, its 256-item limit, a block's 8192-item limit, and
the bitmap order of dense results. Expected values come from numpy on inputs with exact arithmetic."""
import numpy as np
import pytest

import octree_gb300 as otg

pytestmark = pytest.mark.gpu

RUNS = [0, 1, 2, 31, 32, 33, 63, 64, 65, 255, 256, 257, 1000, 4097, 8192]


def csr(lists, dtype=np.uint32):
    off = np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.uint64)
    return off, np.concatenate(lists).astype(dtype) if len(lists) else np.zeros(0, dtype)


def clusters(runs, seed):
    """Points in unit cells at x = 4 i, runs[i] of them in cell i, in shuffled order; their cells."""
    rng = np.random.default_rng(seed)
    cell = rng.permutation(np.repeat(np.arange(len(runs)), runs))
    pts = rng.integers(0, 1 << 20, (len(cell), 3)) / 2.0**20
    pts[:, 0] += 4.0 * cell
    return pts, cell


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("runs", [RUNS, RUNS + [8193], RUNS[:6] * 40], ids=["block", "longer", "short"])
def test_id_runs(runs, dtype):
    """300k points beside the cells make the results sparse, so that they are ordered by runs."""
    pts, cell = clusters(runs, 11)
    rng = np.random.default_rng(12)
    far = rng.random((300_000, 3)) - [6.0, 0.0, 0.0]
    at = rng.permutation(len(pts) + len(far))
    pts, cell = np.concatenate([pts, far])[at], np.concatenate([cell, np.full(len(far), -1)])[at]
    t = otg.Tree("points", dtype).create(pts, max_depth=10, max_elements=16)
    r = np.zeros((len(runs), 6))
    r[:, 0], r[:, 3] = 4.0 * np.arange(len(runs)) - 1, 4.0 * np.arange(len(runs)) + 2
    r[:, 1:3], r[:, 4:6] = -1, 2
    off, ids, _ = t.range_search(r)
    eo, ei = csr([np.flatnonzero(cell == i) for i in range(len(runs))])
    assert np.array_equal(off, eo) and np.array_equal(ids, ei)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("runs", [RUNS, RUNS + [8193], RUNS[:6] * 40], ids=["block", "longer", "short"])
def test_distance_runs(runs, dtype):
    """Ray i meets a stack of runs[i] boxes at multiples of 1/4 (many equal distances)."""
    rng = np.random.default_rng(13)
    row = rng.permutation(np.repeat(np.arange(len(runs)), runs))
    x = rng.integers(1, 512, len(row)) / 4.0
    b = np.zeros((len(row), 6))
    b[:, 0], b[:, 3] = x, x + 0.25
    b[:, 1], b[:, 4] = 4.0 * row, 4.0 * row + 1
    b[:, 2], b[:, 5] = 0, 1
    t = otg.Tree("boxes", dtype).create(b, max_depth=8, max_elements=16)
    rays = np.zeros((len(runs), 6))
    rays[:, 1], rays[:, 2], rays[:, 3] = 4.0 * np.arange(len(runs)) + 0.5, 0.5, 1.0
    off, ids, dist = t.ray_all(rays, tol=0.0)
    lists = [np.flatnonzero(row == i) for i in range(len(runs))]
    lists = [l[np.lexsort((l, x[l]))] for l in lists]
    eo, ei = csr(lists)
    assert np.array_equal(off, eo) and np.array_equal(ids, ei)
    assert np.array_equal(dist, x[ei])


@pytest.mark.parametrize("step", [0.0, 2.0**-44, 2.0**-20, 2.0**40], ids=["equal", "near", "close", "wide"])
@pytest.mark.parametrize("distinct", [1, 2, 9, 1000])
def test_distance_ties(distinct, step):
    """Runs of equal distances and of distances that agree in their leading bits: 1 + step j, `distinct` of them."""
    rng = np.random.default_rng(23)
    runs = [2, 3, 12, 13, 31, 32, 33, 64, 65, 128, 129, 255, 256]
    row = rng.permutation(np.repeat(np.arange(len(runs)), runs))
    x = 1.0 + step * rng.integers(0, distinct, len(row))
    b = np.zeros((len(row), 6))
    b[:, 0], b[:, 3] = x, x + 1.0
    b[:, 1], b[:, 4] = 4.0 * row, 4.0 * row + 1
    b[:, 2], b[:, 5] = 0, 1
    t = otg.Tree("boxes").create(b, max_depth=6, max_elements=16)
    rays = np.zeros((len(runs), 6))
    rays[:, 1], rays[:, 2], rays[:, 3] = 4.0 * np.arange(len(runs)) + 0.5, 0.5, 1.0
    off, ids, dist = t.ray_all(rays, tol=0.0)
    lists = [np.flatnonzero(row == i) for i in range(len(runs))]
    eo, ei = csr([l[np.lexsort((l, x[l]))] for l in lists])
    assert np.array_equal(off, eo) and np.array_equal(ids, ei) and np.array_equal(dist, x[ei])


@pytest.mark.parametrize("n", [300, 8191, 8192, 8193, 70_001])
@pytest.mark.parametrize("nq", [1, 7])
def test_dense_ids(n, nq):
    """Half-spaces that take a third to all of the points: rows of bits, at their chunk edges."""
    rng = np.random.default_rng(17)
    pts = rng.integers(0, 1 << 20, (n, 3)) / 2.0**20
    t = otg.Tree("points").create(pts, max_depth=8, max_elements=16)
    planes = np.zeros((nq, 4))
    planes[:, 0] = np.linspace(-0.5, 0.7, nq)
    planes[:, 1] = 1.0
    off, ids, _ = t.plane_positive_segmentation(planes, tol=0.0)
    eo, ei = csr([np.flatnonzero(pts[:, 0] >= p) for p in planes[:, 0]])
    assert np.array_equal(off, eo) and np.array_equal(ids, ei)


def test_dense_ids_of_a_forest():
    """Rows of bits of different lengths, empty trees among them."""
    rng = np.random.default_rng(19)
    sizes = [9000, 0, 1, 8192, 0, 20_000, 3, 8193]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    pts = rng.integers(0, 1 << 20, (int(off[-1]), 3)) / 2.0**20
    f = otg.Forest("points").create(pts, off, max_elements=16)
    per = 2
    qoff = np.arange(len(sizes) + 1, dtype=np.uint64) * per
    planes = np.zeros((per * len(sizes), 2, 4))
    lo, hi = rng.integers(0, 256, per * len(sizes)) / 1024.0, 0.5 + rng.integers(0, 256, per * len(sizes)) / 512.0
    planes[:, 0, 0], planes[:, 0, 1] = lo, 1.0
    planes[:, 1, 0], planes[:, 1, 1] = -hi, -1.0
    got = f.frustum_culling(planes, qoff, tol=0.0)
    lists = []
    for q in range(per * len(sizes)):
        x = pts[int(off[q // per]) : int(off[q // per + 1]), 0]
        lists.append(np.flatnonzero((x >= lo[q]) & (x <= hi[q])))
    eo, ei = csr(lists)
    assert np.array_equal(got[0], eo) and np.array_equal(got[1], ei)


@pytest.mark.parametrize("nq", [1, 1023, 1024, 1025, 16384, 16385, 40_000])
def test_query_counts(nq):
    """Offsets scanned by one block up to 16384 queries, by tiles above; results read back through the pinned block
    and, above its 256 KiB, directly."""
    rng = np.random.default_rng(23)
    x = np.sort(rng.integers(0, 1 << 16, 5000))
    pts = np.stack([x / 64.0, np.full(len(x), 0.5), np.full(len(x), 0.5)], 1)
    t = otg.Tree("points").create(pts, max_depth=10, max_elements=8)
    lo = rng.integers(0, 1 << 16, nq)
    hi = lo + rng.integers(1, 200, nq)
    r = np.zeros((nq, 6))
    r[:, 0], r[:, 3], r[:, 4:] = lo / 64.0 - 1 / 128, hi / 64.0 - 1 / 128, 1
    off, ids, _ = t.range_search(r, tol=0.0)
    a, b = np.searchsorted(x, lo), np.searchsorted(x, hi)
    assert np.array_equal(off, np.concatenate([[0], np.cumsum(b - a)]))
    assert np.array_equal(ids, np.concatenate([np.arange(i, j) for i, j in zip(a, b)]))
