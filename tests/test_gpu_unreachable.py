"""Box trees with entities that no node holds (loose boxes whose centre lies in cell 2^D of the grid: flat boxes
on the max face of the space): queries that take a subtree whole must not return them. Against the oracle
and the one-query-per-thread kernels."""
import numpy as np
import pytest

import octree_gb300 as otg
from _compare import assert_csr_equal
from _oracle_lib import KIND_LOOSE_BOXES, oracle

pytestmark = pytest.mark.gpu

SHAPES = (-1, 2, 4 | 1 << 8, 2 | 2 << 8, 8 | 4 << 8)


def cases(dtype, n=2001):
    rng = np.random.default_rng(61)
    cen = rng.random((n, 3)) * 48 + 0.5
    h = rng.random((n, 3)) * 0.5
    b = np.concatenate([cen - h, cen + h], 1)
    ceiling = b.copy()
    ceiling[7] = [10, 10, 50, 12, 12, 50]
    corner = b.copy()
    corner[1] = [50, 50, 50, 50, 50, 50]
    corner[2] = [0, 0, 0, 0, 0, 0]
    space = np.array([0.0, 0, 0, 50, 50, 50])
    return {k: (v[0].astype(dtype), v[1]) for k, v in {
        "flat": (np.concatenate([cen, cen], 1), None),
        "ceiling": (ceiling, None),
        "ceiling_given_space": (ceiling, space),
        "corner": (corner, space),
    }.items()}


def frusta(dtype, n):
    """Boxes of six planes: around everything, up to just below the max faces, and around parts."""
    rng = np.random.default_rng(67)
    lo = np.full((n, 3), -1.0)
    hi = np.full((n, 3), 51.0)
    hi[n // 4 : n // 2] = 49.75  # holds the boxes of the nodes, not the ones on the max faces
    lo[n // 2 :] = rng.random((n - n // 2, 3)) * 20
    p = np.zeros((n, 6, 4))
    for a in range(3):
        p[:, 2 * a, 0], p[:, 2 * a, 1 + a] = lo[:, a], 1.0
        p[:, 2 * a + 1, 0], p[:, 2 * a + 1, 1 + a] = -hi[:, a], -1.0
    return p.astype(dtype)


@pytest.mark.parametrize("name", ["flat", "ceiling", "ceiling_given_space", "corner"])
@pytest.mark.parametrize("max_elem", [4, 24])
@pytest.mark.parametrize("n", [41, 2001])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_whole_subtrees_hold_no_unreachable_entity(dtype, n, max_elem, name):
    ent, space = cases(dtype, n)[name]
    t = otg.Tree("boxes", dtype).create(ent, max_depth=5, box=space, max_elements=max_elem)
    o = oracle().create(ent, KIND_LOOSE_BOXES, 5, space, max_elem)
    p = frusta(dtype, 64)
    single = np.ascontiguousarray(p[:, 0])
    want, side = o.frustum(p), o.plane_positive(single)
    for shape in SHAPES:
        otg.autotune_force_shape(shape)
        try:
            for _ in range(2):  # FP64 trees build their images once the queries are worth it
                assert_csr_equal(t.frustum_culling(p)[:2], want, f"{name} frustum {shape}")
            assert_csr_equal(t.plane_positive_segmentation(single)[:2], side, f"{name} positive side {shape}")
        finally:
            otg.autotune_force_shape(-1)
    assert_csr_equal(t.frustum_culling(p, algo=otg.ALGO_PLAIN_FP64)[:2], want, f"{name} plain frustum")
    assert_csr_equal(t.plane_positive_segmentation(single, algo=otg.ALGO_PLAIN_FP64)[:2], side, f"{name} plain positive side")
    assert np.array_equal(t.collision_self(), o.collide_self())
    assert np.array_equal(t.collision_pair(t), o.collide_pair(o))


def test_static_export_still_refuses_them():
    ent, space = cases(np.float64)["ceiling"]
    t = otg.Tree("boxes").create(ent, max_depth=5, box=space, max_elements=8)
    with pytest.raises(otg.OtgError, match="outside the grid"):
        t.export_static()


def check_forest(res, trees, spaces, p, per):
    for i, e in enumerate(trees):
        o = oracle().create(e, KIND_LOOSE_BOXES, 5, None if spaces is None else spaces[i], 8)
        a, b = i * per, (i + 1) * per
        r = res[0].astype(np.int64)[a : b + 1]
        assert_csr_equal((r - r[0], res[1][r[0] : r[-1]]), o.frustum(p[a:b]), f"tree {i}")


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_forest_and_plan(dtype):
    torch = pytest.importorskip("torch")
    trees = [e for e, _ in cases(dtype).values()] + [cases(dtype, 700)["flat"][0]]
    ent = np.concatenate(trees)
    off = np.concatenate([[0], np.cumsum([len(e) for e in trees])]).astype(np.uint64)
    per = 64
    p = np.concatenate([frusta(dtype, per)] * len(trees))
    qoff = np.arange(len(trees) + 1, dtype=np.uint64) * per
    space = np.tile(np.array([[0.0, 0, 0, 50, 50, 50]], dtype), (len(trees), 1))
    for spaces in (space, None):
        f = otg.Forest("boxes", dtype).create(ent, off, max_depth=5, boxes=spaces, max_elements=8)
        for _ in range(2):
            check_forest(f.frustum_culling(p, qoff), trees, spaces, p, per)
    plan = otg.ForestPlan(otg.Forest("boxes", dtype), torch.as_tensor(ent, device="cuda"), off, max_depth=5, max_elements=8,
                          planes=torch.as_tensor(p, device="cuda"), frustum_offsets=qoff, capacity_factor=4.0)
    for _ in range(2):
        plan.run()
        check_forest(plan.result(otg.ForestPlan.FRUSTUM), trees, None, p, per)
