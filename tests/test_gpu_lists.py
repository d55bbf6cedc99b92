"""The neighbour lists themselves, read back and compared with brute force, and
the walk on them against the oracle, on clouds whose leaves are far wider than
the radius of a list: compact groups in a sparse field."""
import warnings

import numpy as np
import pytest
from scipy.spatial import cKDTree

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _groups(box, sigma, seed=3):
    """2,000 field points and 60 groups of 70 to 120 points of width sigma."""
    rng = np.random.default_rng(seed)
    centre = rng.uniform(0.1, 0.9, (60, 3)) * box
    pos = [rng.uniform(0, box, (2000, 3))]
    pos += [c + sigma * rng.normal(size=(rng.integers(70, 121), 3)) for c in centre]
    return np.vstack(pos), rng


def _cloud(pos, box, f):
    import vortrace_b200 as vt
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return vt.ProjectionCloud(pos, f, boundbox=[0.0, box] * 3)


def _rays(pos, box, rng, m=1500):
    """Through pairs of points of one group, of a group and the field point nearest
    to it (often in one leaf), and of any two points; past both by some lengths."""
    i = rng.integers(2000, len(pos), m)
    near = cKDTree(pos).query(pos[i], k=40)[1]
    j = near[np.arange(m), rng.integers(1, 40, m)]
    j[: m // 3] = cKDTree(pos[:2000]).query(pos[i[: m // 3]])[1]
    j[-m // 6:] = rng.integers(0, len(pos), m // 6)
    a, b = pos[i], pos[j]
    mid = a + rng.uniform(-0.3, 0.3, (m, 1)) * (b - a)[:, ::-1]
    d = (b - a) * rng.uniform(1, 30, (m, 1))
    return np.clip(mid - d, 0, box), np.clip(mid + d, 0, box)


SHAPES = [(1e2, 1e-3), (1e4, 1e-2), (1e5, 1e-2), (1e5, 1.0)]


@pytest.mark.parametrize("box,sigma", SHAPES)
def test_lists_hold_every_point_inside_their_radius(box, sigma):
    pos, rng = _groups(box, sigma)
    pc = _cloud(pos, box, np.ones(len(pos)))
    s, e = _rays(pos, box, rng)
    pc.projection(s, e)
    lists, head = pc._cloud.neighbour_lists()
    blob = pc._cloud.saveTreeToBytes()
    depth = 0
    while (len(pos) + (1 << depth) - 1) >> depth > 8:
        depth += 1
    perm = np.frombuffer(blob, np.int32, len(pos), len(blob) - 4 * len(pos) - 24 * ((1 << depth) - 1))
    p = pc.pos_orig[pc.orig_ids][perm]
    half = (head & ~np.uint32(1023)).view(np.float32).astype(np.float64)
    assert (head != 0).mean() > 0.5
    tree = cKDTree(p)
    for i in np.flatnonzero(head):
        up, down = (head[i] >> 5) & 31, head[i] & 31
        parts = [lists[i, :up], lists[i, 16 - down:][::-1]]
        ids = np.concatenate([q[:, 3].reshape(-1).view(np.int32) for q in parts])
        rho = np.sqrt(2 * half[i])
        inside = np.setdiff1d(tree.query_ball_point(p[i], rho * (1 - 1e-12)), [i])
        assert np.isin(inside, ids).all(), (i, rho)
        for sign, q in zip((1, -1), parts):
            j = q[:, 3].reshape(-1).view(np.int32)
            ok = j >= 0
            d = p[j[ok]] - p[i]
            v = q[:, :3].transpose(0, 2, 1).reshape(-1, 3)[ok]
            np.testing.assert_array_equal(v, d.astype(np.float32))
            assert np.all(v[:, 2] > 0 if sign > 0 else v[:, 2] <= 0)
            d2 = (d ** 2).sum(1)
            # ascending but for the key's 10 dropped bits (2^-13) and FP32 rounding
            assert np.all(d2[1:] >= d2[:-1] * (1 - 1.3e-4))


@pytest.mark.parametrize("box,sigma", SHAPES)
def test_walk_through_groups_equals_oracle(box, sigma):
    pos, rng = _groups(box, sigma)
    f = rng.uniform(0, 1, len(pos))
    pc = _cloud(pos, box, f)
    s, e = _rays(pos, box, rng, 6000)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        lp = O.load_points(pos, f, [0.0, box] * 3)
    ot = O.OracleTree(lp["pts"], lp["fields"], lp["valid_rgba"])
    out, (cell, s_enter, s_exit, off) = ot.project(s, e, "integrate", segments=True)
    pc.projection(s, e)
    pc._cloud.neighbour_lists()  # they are built
    val, cid, se, ds, offsets = pc.traced_projection(s, e, return_midpoint=False, flatten=True)
    np.testing.assert_array_equal(offsets, off)
    np.testing.assert_array_equal(cid, lp["orig_ids"][cell])
    np.testing.assert_array_equal(se, s_enter)
    np.testing.assert_array_equal(ds, s_exit - s_enter)
    np.testing.assert_array_equal(val, out.reshape(-1))
