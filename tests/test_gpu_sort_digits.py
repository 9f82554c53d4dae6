"""Trees built by every form of the sort's passes (eight- and nine-bit digits, box keys without their
depth's upper bits, segmented passes of a forest) against the oracle, for even and skewed keys."""
import numpy as np
import pytest

import octree_gb300 as otg
from _compare import assert_nodes_equal
from _oracle_lib import KIND_BOXES, KIND_LOOSE_BOXES, KIND_POINTS, oracle

pytestmark = pytest.mark.gpu
NAME = {KIND_POINTS: "points", KIND_LOOSE_BOXES: "boxes", KIND_BOXES: "regular_boxes"}


def entities(rng, n, kind, spread, dtype):
    c = rng.random((n, 3)) * 100
    if spread == "few":  # lanes that share their digits
        c = rng.random((3, 3))[rng.integers(0, 3, n)] * 90 + 5
    elif spread == "sorted":
        c = c[np.argsort(c[:, 2])]
    if kind == KIND_POINTS:
        return c.astype(dtype)
    h = rng.uniform(0.01, 2.0, (n, 3)) * rng.choice([1.0, 1.0, 8.0], (n, 1))
    b = np.concatenate([np.clip(c - h, 0, 100), np.clip(c + h, 0, 100)], 1)
    if n > 4:
        b[n // 2] = [0, 0, 0, 100, 100, 100]  # a box as large as the space
        b[n // 3] = [100, 100, 100, 100, 100, 100] if kind == KIND_LOOSE_BOXES else b[0]  # centred on the far corner
    return b.astype(dtype)


@pytest.mark.parametrize("spread", ["even", "few", "sorted"])
@pytest.mark.parametrize("kind", [KIND_POINTS, KIND_LOOSE_BOXES, KIND_BOXES])
@pytest.mark.parametrize("depth", [1, 2, 3, 4, 5, 6, 7, 8, 9])
def test_depths(depth, kind, spread):
    rng = np.random.default_rng(300 + depth)
    dtype = np.float64 if depth % 2 else np.float32
    for n in (1, 33, 4095, 4097, 20_011):
        e = entities(rng, n, kind, spread, dtype)
        t = otg.Tree(NAME[kind], dtype).create(e, max_depth=depth, max_elements=8)
        assert_nodes_equal(t.nodes(), oracle().create(e, kind, depth, None, 8).nodes(), f"{depth} {kind} {spread} {n}")


@pytest.mark.parametrize("spread", ["even", "few"])
@pytest.mark.parametrize("kind", [KIND_POINTS, KIND_LOOSE_BOXES])
@pytest.mark.parametrize("depth", [4, 6, 7, 8])
def test_forest(depth, kind, spread):
    rng = np.random.default_rng(330 + depth)
    sizes = [1, 0, 4096, 4097, 8192, 300, 12_289]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    e = np.concatenate([entities(rng, n, kind, spread, np.float32) for n in sizes if n])
    f = otg.Forest(NAME[kind], np.float32).create(e, off, max_depth=depth, max_elements=8)
    nodes, tree = f.nodes(), f.node_trees()
    for i, n in enumerate(sizes):
        if not n:
            continue
        at = int(off[i])
        sel = np.nonzero(tree == i)[0]
        ids = [nodes["eids"][int(nodes["eoff"][k]) : int(nodes["eoff"][k + 1])].astype(np.int64) - at for k in sel]
        got = dict(keys=nodes["keys"][sel], min=nodes["min"][sel], size=nodes["size"][sel],
                   eoff=np.concatenate([[0], np.cumsum([len(x) for x in ids])]).astype(np.uint64), eids=np.concatenate(ids).astype(np.uint32))
        assert_nodes_equal(got, oracle().create(e[at : at + n], kind, depth, None, 8).nodes(), f"tree {i}")


@pytest.mark.parametrize("kind,dtype", [(KIND_POINTS, np.float32), (KIND_POINTS, np.float64), (KIND_LOOSE_BOXES, np.float32), (KIND_LOOSE_BOXES, np.float64)])
@pytest.mark.parametrize("n", [1, 682, 683, 2049, 5000])
def test_forest_geometry(kind, dtype, n):
    """A forest's gather at the edges of a block's units, from an aligned array and from one that starts a scalar later:
    a range that holds everything and one that holds some."""
    import torch

    rng = np.random.default_rng(350 + n)
    e = entities(rng, 3 * n, kind, "even", dtype)
    off = np.array([0, n, 2 * n, 3 * n], np.uint64)
    r = np.array([[-1.0] * 3 + [101.0] * 3, [20.0] * 3 + [60.0] * 3], dtype)
    w = e.shape[1]
    for shift in (0, 1):
        buf = torch.empty(3 * n * w + 2, device="cuda", dtype=torch.float64 if dtype == np.float64 else torch.float32)
        d = buf[shift : shift + 3 * n * w].view(3 * n, w)
        d.copy_(torch.as_tensor(e))
        f = otg.Forest(NAME[kind], dtype).create(d, off, max_depth=5, max_elements=8)
        o, ids = f.range_search(np.tile(r, (3, 1)), np.array([0, 2, 4, 6], np.uint64), otg.RANGE_INSIDE)[:2]
        for t in range(3):
            eo, ei = oracle().create(e[t * n : (t + 1) * n], kind, 5, None, 8).range_search(r, 0)[:2]
            a, b = int(o[2 * t]), int(o[2 * t + 2])
            assert np.array_equal(o[2 * t : 2 * t + 3] - o[2 * t], eo) and np.array_equal(ids[a:b], ei), (t, shift)


def test_forest_gather_of_large_trees():
    """A tree above the size up to which loads fetch ahead, beside a small one: the geometry in tree order is the entities'."""
    rng = np.random.default_rng(371)
    sizes = [64 * 2**20 // 24 + 1, 1000]
    n = sum(sizes)
    c = rng.random((n, 3), dtype=np.float32) * 100
    off = np.array([0, sizes[0], n], np.uint64)
    e = np.concatenate([c, c + np.float32(0.25)], 1)
    f = otg.Forest("boxes", np.float32).create(e, off)
    r = np.array([[10, 10, 10, 13, 14, 15], [0, 0, 0, 40, 40, 40]], np.float32)
    o, ids = f.range_search(r, np.array([0, 1, 2], np.uint64), otg.RANGE_INSIDE)[:2]
    for t in range(2):
        s = e[int(off[t]) : int(off[t + 1])]
        inside = np.flatnonzero(((s[:, :3] > r[t, :3]) & (s[:, 3:] < r[t, 3:])).all(1))
        assert np.array_equal(ids[int(o[t]) : int(o[t + 1])], inside), t
