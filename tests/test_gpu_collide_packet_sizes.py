"""Collisions of sparse and of dense boxes at counts around which the search's packets change their size, against
the search without packets."""
import numpy as np
import pytest

import octree_gb300 as otg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 37, 9727, 9728, 9729, 19_457, 38_911, 77_825, 155_647, 155_649])
@pytest.mark.parametrize("per", [3, 40])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_packet_sizes(dtype, per, n):
    rng = np.random.default_rng(79)
    c = rng.random((n, 3)) * 100
    h = 25.0 * (per / n) ** (1 / 3) * (0.5 + rng.random((n, 3)))
    ent = np.concatenate([c - h, c + h], 1).astype(dtype)
    t = otg.Tree("boxes", dtype).create(ent, max_depth=8, max_elements=16)
    assert np.array_equal(t.collision_self(), t.collision_self(algo=otg.ALGO_PLAIN_FP64))
    m = n // 3 + 1
    u = otg.Tree("boxes", dtype).create(ent[:m] + dtype(0.5), max_depth=7, max_elements=16)
    assert np.array_equal(t.collision_pair(u), t.collision_pair(u, algo=otg.ALGO_PLAIN_FP64))
