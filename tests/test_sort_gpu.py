"""Keys and the sorted order of the octree build, at the sizes where the keys
kernel changes its keys per thread and where tiles and blocks end, against a
float32 replay of the descent and a stable sort of its keys on the host."""
import numpy as np
import pytest

import nbody_gb300 as nb

pytestmark = pytest.mark.gpu
HALF, DEPTH = np.float32(4000.0), 21


def host_keys(x):
    """The octant path of each body (Octree::Add's descent) and its length, in
    float32; a path that meets a gap between float child bounds ends there."""
    inside = ((x >= -HALF) & (x < HALF)).all(1)
    lo = np.full(x.shape, -HALF, np.float32)
    size = np.full(len(x), HALF + HALF, np.float32)
    key, depth = np.zeros(len(x), np.uint64), np.zeros(len(x), np.int32)
    live = inside.copy()
    for _ in range(DEPTH):
        s = size * np.float32(0.5)
        mid = lo + s[:, None]
        top = mid + s[:, None]
        up = x >= mid
        live &= ~(up & ~(x < top)).any(1)
        size = np.where(up[:, 0], top[:, 0] - mid[:, 0], mid[:, 0] - lo[:, 0])
        lo = np.where(up, mid, lo)
        oct_ = (up * np.array([1, 2, 4], np.uint64)).sum(1, dtype=np.uint64)
        key = (key << np.uint64(3)) | np.where(live, oct_, np.uint64(0))
        depth += live
    key[~inside] = np.uint64(0xFFFFFFFFFFFFFFFF)
    return key, depth


@pytest.mark.parametrize("n", [2, 255, 257, 4095, 4097, 8193, 100003, 700001, 1300001])
@pytest.mark.parametrize("spread", [3.0, 5000.0])
def test_keys_and_order(n, spread):
    rng = np.random.default_rng(n)
    x = rng.normal(0.0, spread, (n, 3)).astype(np.float32)
    x[n // 2] = x[0]                       # a coincident pair: ties keep their input order
    x[rng.integers(0, n, n // 50)] = x[0]
    pm = np.concatenate([x, np.full((n, 1), 1.0 / n, np.float32)], 1)
    want, want_depth = host_keys(x)
    with nb.NBodySim(kind=nb.SIM_BARNES_HUT) as s:
        s.init_soa(pm, np.zeros_like(pm))
        keys, depth = s.tree_keys()
        np.testing.assert_array_equal(keys, want)
        np.testing.assert_array_equal(depth, want_depth)
        if (want_depth > 0).sum() >= 2:
            np.testing.assert_array_equal(s.tree_order(), np.argsort(want, kind="stable"))


def test_exported_order_after_a_force_pass():
    """A force pass sorts the bodies along the Hilbert curve; the exported
    order, nodes and statistics are still those of the octant paths."""
    pm, v = nb.seed_disk(5, 20000)
    with nb.NBodySim(kind=nb.SIM_BARNES_HUT, theta=0.5) as s, nb.NBodySim(kind=nb.SIM_BARNES_HUT, theta=0.5) as t:
        s.init_soa(pm, v)
        t.init_soa(pm, v)
        F = s.compute_forces()
        nodes, order, stats = s.tree_nodes(), s.tree_order(), s.tree_stats()
        np.testing.assert_array_equal(nodes, t.tree_nodes())
        np.testing.assert_array_equal(order, t.tree_order())
        assert stats == t.tree_stats()
        keys, _ = s.tree_keys()
        np.testing.assert_array_equal(order, np.argsort(keys, kind="stable"))
        np.testing.assert_array_equal(F, s.compute_forces())
