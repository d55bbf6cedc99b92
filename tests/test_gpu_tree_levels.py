"""The device tree against the same build in numpy: levels over all points and
levels inside one block, segments on both sides of the block's 1024 points, a
leaf size that changes the last level, tied coordinates."""
import numpy as np
import pytest

import vortrace_b200 as vt
from vortrace_b200 import _lib as L

pytestmark = pytest.mark.gpu


def _numpy_tree(pos, leaf):
    """perm of the tree: Morton order, then per level a stable sort of every
    segment along its widest dimension; segment k of level l holds
    [k n >> l, (k + 1) n >> l)."""
    n = len(pos)
    lo, hi = pos.min(0), pos.max(0)
    sc = 2097151.0 / (hi - lo)
    q = np.minimum(np.maximum((pos - lo) * sc, 0.0), 2097151.0).astype(np.uint64)
    key = np.zeros(n, np.uint64)
    for b in range(21):
        for d in range(3):
            key |= ((q[:, d] >> np.uint64(b)) & np.uint64(1)) << np.uint64(3 * b + d)
    perm = np.argsort(key, kind="stable")
    depth = 0
    while (n + (1 << depth) - 1) >> depth > leaf:
        depth += 1
    splits = []
    for l in range(depth):
        for k in range(1 << l):
            a, b = k * n >> l, (k + 1) * n >> l
            p = perm[a:b]
            d = int(np.argmax(pos[p].max(0) - pos[p].min(0)))
            perm[a:b] = p[np.argsort(pos[p, d], kind="stable")]
            splits.append((d, pos[perm[(2 * k + 1) * n >> (l + 1)], d]))
    return perm, splits


@pytest.mark.parametrize("n,leaf", [(9, 8), (33, 2), (700, 8), (1023, 8), (1024, 8), (1025, 8),
                                    (2047, 64), (2049, 3), (5000, 8), (40000, 6), (70001, 8)])
@pytest.mark.parametrize("tied", [False, True])
def test_tree_is_the_level_by_level_one(n, leaf, tied):
    rng = np.random.default_rng(n + leaf)
    pos = rng.random((n, 3)) * [1.0, 2.0, 0.5]
    if tied:
        pos = np.round(pos * 16) / 16 + 0.03125
    cloud = vt.vortrace._Cloud()
    box = [-1.0, 3.0, -1.0, 3.0, -1.0, 3.0]
    cloud.loadPoints(pos, np.ones(n), box, np.full(n, 1.0))
    cloud.set_param(L.PARAM_LEAF_SIZE, leaf)
    cloud.buildTree()
    blob = cloud.saveTreeToBytes()
    perm, splits = _numpy_tree(pos, leaf)
    head = len(blob) - 4 * n - 24 * len(splits)
    np.testing.assert_array_equal(np.frombuffer(blob, np.int32, n, head), perm)
    nodes = np.frombuffer(blob, np.float64, 2 * len(splits), head + 4 * n).reshape(-1, 2)
    dims = nodes[:, 0].copy().view(np.uint64) & np.uint64(3)
    np.testing.assert_array_equal(dims, [d for d, _ in splits])
    np.testing.assert_array_equal(nodes[:, 1], [v for _, v in splits])
