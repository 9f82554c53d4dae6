"""Signs of zero in node geometry: of coordinates that are 0.0 and -0.0 a node keeps the first in order, as the
reference's std::min and std::max do."""
import numpy as np
import pytest

import octree_gb300 as otg
from _oracle_lib import KIND_LOOSE_BOXES, KIND_POINTS, oracle

pytestmark = pytest.mark.gpu


def assert_same_bits(t, o):
    gpu, ref = t.nodes(), o.nodes()
    order = np.argsort(gpu["keys"], kind="stable")
    assert np.array_equal(gpu["keys"][order], ref["keys"])
    for name in ("min", "size"):
        a, b = gpu[name][order], ref[name]
        assert np.array_equal(a, b) and np.array_equal(np.signbit(a), np.signbit(b)), name
    return ref


@pytest.mark.parametrize("max_depth,max_elem", [(1, 400), (4, 3), (6, 16)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_boxes(dtype, max_depth, max_elem):
    rng = np.random.default_rng(107)
    c = rng.random((3000, 3)) * 20 - 10
    h = rng.random((3000, 3))
    lo, hi = c - h, c + h
    side = rng.integers(0, 3, (3000, 3))  # many boxes end or begin at zero
    z = np.where(rng.random((3000, 3)) < 0.5, 0.0, -0.0)
    lo, hi = np.where(side == 1, z, lo), np.where(side == 2, z, hi)
    lo, hi = np.where((side == 2) & (lo >= 0), lo - 12, lo), np.where((side == 1) & (hi <= 0), hi + 12, hi)
    ent = np.concatenate([lo, hi], 1).astype(dtype)
    space = np.array([-24.0, -24, -24, 24, 24, 24])
    t = otg.Tree("boxes", dtype).create(ent, max_depth=max_depth, box=space, max_elements=max_elem)
    ref = assert_same_bits(t, oracle().create(ent, KIND_LOOSE_BOXES, max_depth, space, max_elem))
    if max_depth > 1:
        zeros = ref["min"] == 0
        assert (np.signbit(ref["min"]) & zeros).any() and (~np.signbit(ref["min"]) & zeros).any()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_root_box_of_outside_points(dtype):
    rng = np.random.default_rng(109)
    for trial in range(8):
        p = 1 + rng.random((500, 3)) * 9
        out = rng.permutation(500)[:200]
        p[out] = np.where(rng.random((200, 3)) < 0.2, np.where(rng.random((200, 3)) < 0.5, 0.0, -0.0), p[out])
        p = p.astype(dtype)
        space = np.array([0.5, 0.5, 0.5, 11, 11, 11])
        t = otg.Tree("points", dtype).create(p, max_depth=4, box=space, max_elements=8)
        assert_same_bits(t, oracle().create(p, KIND_POINTS, 4, space, 8))
