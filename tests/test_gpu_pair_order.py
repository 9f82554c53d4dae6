"""Order of collision pairs over the lengths at which it changes its way: runs sorted by rank, in registers, by a
block, and by radix sorts."""
import numpy as np
import pytest

import octree_gb300 as otg

pytestmark = pytest.mark.gpu


def groups(rng, lens, dtype):
    """Box i of the first tree holds lens[i] boxes of the second, and meets no others."""
    side = 10.0
    n = len(lens)
    edge = int(np.ceil(n ** (1 / 3)))
    at = np.stack(np.unravel_index(np.arange(n), (edge,) * 3), 1) * (2 * side)
    a = np.concatenate([at, at + side], 1)
    owner = np.repeat(np.arange(n), lens)
    c = at[owner] + 1 + rng.random((len(owner), 3)) * (side - 2)
    b = np.concatenate([c, c + 0.01], 1)
    p = rng.permutation(len(b))
    return a.astype(dtype), b[p].astype(dtype), owner[p]


@pytest.mark.parametrize(
    "lens",
    [[1, 2, 0, 63, 64, 65, 3, 128, 129, 255, 256], [64] * 40, [65] * 40, [1] * 100 + [257, 511, 512, 513, 1024, 1025, 0, 70], [8191, 8192, 5], [8193, 5, 300]],
)
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_runs(dtype, lens):
    a, b, owner = groups(np.random.default_rng(73), lens, dtype)
    ta = otg.Tree("boxes", dtype).create(a, max_depth=4, max_elements=8)
    tb = otg.Tree("boxes", dtype).create(b, max_depth=6, max_elements=16)
    ids = np.argsort(owner, kind="stable")
    assert np.array_equal(ta.collision_pair(tb), np.stack([owner[ids], ids], 1))
