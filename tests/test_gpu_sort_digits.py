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
