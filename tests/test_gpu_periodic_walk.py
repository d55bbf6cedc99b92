"""The periodic walk kernel (every kernel choice but 'plain' on a periodic cloud)
against the one-ray-per-thread periodic walk ('plain'), bit for bit: images,
segments, failures; few and many points, rays along and across the faces, out of
the domain, and with both ends in one cell."""
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(kind):
    import vortrace_b200 as vt
    rng = np.random.default_rng(len(kind))
    n = int(kind[1:]) if kind[0] == "n" else 2000
    pos = rng.uniform(0, 1, (n, 3))
    if kind == "dense corner":  # the densest cells wrap around a corner
        pos[: n // 2] = (0.05 * rng.normal(size=(n // 2, 3))) % 1.0
    if kind == "lattice":
        c = (np.arange(8) + 0.5) / 8
        pos = np.stack(np.meshgrid(c, c, c, indexing="ij"), -1).reshape(-1, 3)
    f = rng.uniform(0, 1, (len(pos), 4))
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return vt.ProjectionCloud(pos, f, boundbox=[0, 1] * 3, periodic=True), rng


def _rays(rng, m=480):
    s, e = rng.uniform(0, 1, (m, 3)), rng.uniform(0, 1, (m, 3))
    k = m // 6
    e[:k, :2] = s[:k, :2]
    s[:k, 2], e[:k, 2] = 0.0, 1.0                    # face to face: one cell at both ends
    s[k:2 * k, 0] = e[k:2 * k, 0] = 1e-4             # along a face
    s[2 * k:3 * k] *= 0.02                            # out of a corner
    e[3 * k:4 * k] = s[3 * k:4 * k] + 0.01 * rng.normal(size=(k, 3))
    e[4 * k:5 * k] = np.clip(1.3 * e[4 * k:5 * k], 0, 1.2)  # past the domain
    return s, e


def _same(pc, call):
    """``call`` with the plain and the other kernel: the same arrays, or the same
    failure (a short ray, for instance, may not find a second cell)."""
    res = []
    for kernel in ("plain", "auto"):
        pc.kernel = kernel
        try:
            out = call()
            res.append(out if isinstance(out, tuple) else (out,))
        except Exception as ex:
            res.append(str(ex))
    assert type(res[0]) is type(res[1]), res
    if isinstance(res[0], str):
        assert res[0] == res[1]
        return
    for a, b in zip(*res):
        np.testing.assert_array_equal(b, a)


@pytest.mark.parametrize("kind", ["n7", "n40", "n500", "n2000", "dense corner", "lattice"])
@pytest.mark.parametrize("reduction", ["integrate", "max", "volume"])
def test_equals_the_plain_walk(kind, reduction):
    pc, rng = _cloud(kind)
    s, e = _rays(rng)
    for i in range(0, len(s), 32):  # a failing ray fails its call
        _same(pc, lambda: pc.projection(s[i:i + 32], e[i:i + 32], reduction=reduction))


@pytest.mark.parametrize("kind", ["n500", "dense corner"])
def test_segments_and_sizes(kind):
    """Segments of batches around the warp and block sizes; lowered limits."""
    from vortrace_b200 import _lib as L
    pc, rng = _cloud(kind)
    s, e = _rays(rng, 4800)
    for i, m in ((0, 1), (0, 31), (900, 33), (1700, 129), (0, 800), (0, 4800)):
        _same(pc, lambda: pc.traced_projection(s[i:i + m], e[i:i + m], flatten=True))
    pc._cloud.set_param(L.PARAM_LOCAL_STACK, 2)
    _same(pc, lambda: pc.projection(s[:800], e[:800]))
    pc._cloud.set_param(L.PARAM_LOCAL_STACK, 1 << 30)
    pc._cloud.set_param(L.PARAM_MAX_ITERATIONS, 3)
    _same(pc, lambda: pc.projection(s[:800], e[:800]))
