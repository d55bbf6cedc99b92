"""The walk on neighbour lists (the 'auto' kernel once the lists are built)
against the CPU oracle: images, segment lists and gradients, bit for bit where
the oracle's arithmetic is the walk's (volume images within 1e-12, CUDA's exp
against glibc's; gradients within the rounding of their sums)."""
import warnings

import numpy as np
import pytest

from oracle import oracle as O
from vortrace_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _plummer(rng, n):
    return W._plummer(rng, n, 2.0, np.full(3, 50.0), 40.0)


def _cloud_points(kind):
    rng = np.random.default_rng(len(kind))
    if kind.startswith("uniform"):  # sizes around the smallest with lists
        return rng.uniform(0, 100, (int(kind[7:]), 3)), [0.0, 100.0] * 3
    if kind == "clustered":
        return np.vstack([_plummer(rng, 5400), rng.uniform(0, 100, (600, 3))]), [0.0, 100.0] * 3
    if kind == "clumps":  # density steps of 1e6 and empty space between
        return np.vstack([50 + 20 * np.array(d) + rng.normal(0, s, (800, 3)) for d, s in
                          (((1, 0, 0), 0.02), ((-1, 0, 0), 0.5), ((0, 1, 1), 3.0))]), \
            [0.0, 100.0] * 3
    if kind == "far":  # rounding of the coordinates far above the tolerance
        return 1.0e6 + rng.uniform(0, 100, (3000, 3)), [1.0e6, 1.0e6 + 100.0] * 3
    if kind == "plane":  # flat tree boxes
        p = rng.uniform(0, 100, (2000, 3))
        p[:, 2] = 50.0
        return p, [0.0, 100.0] * 3
    if kind == "pairs":  # every point twice
        return np.repeat(rng.uniform(0, 100, (700, 3)), 2, axis=0), [0.0, 100.0] * 3
    c = np.arange(9, dtype=np.float64) + 0.5  # lattice
    p = np.stack(np.meshgrid(c, c, c, indexing="ij"), -1).reshape(-1, 3) * (100.0 / 9)
    return p.astype(np.float32).astype(np.float64), [0.0, 100.0] * 3


def _rays(kind, bb, m=600):
    """Random chords, a pixel grid along z, rays from far outside, rays along
    the axes through generators, and short ones."""
    rng = np.random.default_rng(100 + len(kind))
    lo, w = bb[0], bb[1] - bb[0]
    s, e = rng.uniform(0, 1, (m, 3)), rng.uniform(0, 1, (m, 3))
    k = m // 6
    e[k:2 * k, :2] = s[k:2 * k, :2]
    s[k:2 * k, 2], e[k:2 * k, 2] = 0.0, 1.0
    d = rng.normal(size=(k, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    mid = 0.5 + 0.05 * rng.normal(size=(k, 3))
    s[2 * k:3 * k], e[2 * k:3 * k] = mid - 4 * d, mid + 4 * d
    e[3 * k:4 * k] = s[3 * k:4 * k] + 1e-3 * rng.normal(size=(k, 3))
    q = np.floor(9 * rng.uniform(0, 1, (k, 3))) / 9 + 0.5 / 9  # lattice columns
    s[4 * k:5 * k], e[4 * k:5 * k] = q, q
    s[4 * k:5 * k, 0], e[4 * k:5 * k, 0] = 0.0, 1.0
    return lo + w * s, lo + w * e


KINDS = ["uniform64", "uniform65", "uniform300", "uniform4001", "clustered", "clumps", "far",
         "plane", "pairs", "lattice"]


def _setup(kind, fields):
    import vortrace_b200 as vt
    pos, bb = _cloud_points(kind)
    f = fields(len(pos))
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        pc = vt.ProjectionCloud(pos, f, boundbox=bb)
        lp = O.load_points(pos, f, bb)
    return pc, O.OracleTree(lp["pts"], lp["fields"], lp["valid_rgba"]), lp, _rays(kind, bb)


def _has_lists(pc):
    """The lists take more memory than all the rest of the cloud."""
    info = pc._cloud.info()
    return info.device_bytes > 1000 * info.npart


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("nf,reduction", [(1, "integrate"), (3, "integrate"), (2, "max"),
                                          (1, "min"), (4, "volume")])
def test_image_equals_oracle(kind, nf, reduction):
    rng = np.random.default_rng(nf)
    pc, ot, lp, (s, e) = _setup(kind, lambda n: rng.uniform(0, 1, (n, nf)))
    want = ot.project(s, e, reduction)
    got = pc.projection(s, e, reduction=reduction).reshape(want.shape)
    assert _has_lists(pc)
    if reduction == "volume":
        np.testing.assert_allclose(got, want, rtol=1e-12, atol=0)
    else:
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("kind", KINDS)
def test_segments_equal_oracle(kind):
    pc, ot, lp, (s, e) = _setup(kind, lambda n: np.arange(1.0, n + 1.0))
    out, (cell, s_enter, s_exit, off) = ot.project(s, e, "integrate", segments=True)
    val, cid, se, ds, offsets = pc.traced_projection(s, e, return_midpoint=False, flatten=True)
    assert _has_lists(pc)
    np.testing.assert_array_equal(offsets, off)
    np.testing.assert_array_equal(cid, lp["orig_ids"][cell])
    np.testing.assert_array_equal(se, s_enter)
    np.testing.assert_array_equal(ds, s_exit - s_enter)
    np.testing.assert_array_equal(val, out.reshape(-1))


@pytest.mark.parametrize("kind", ["uniform4001", "clustered", "lattice"])
def test_gradient_of_taped_and_rewalked(kind):
    """dL/dfield of 'integrate': the sum of upstream * ds over a cell's
    segments; the first call on a cloud walks the rays again, the second
    scatters the tape."""
    import torch
    from vortrace_b200 import autograd as VA
    rng = np.random.default_rng(5)
    pc, ot, lp, (s, e) = _setup(kind, lambda n: rng.uniform(0, 1, n))
    _, (cell, s_enter, s_exit, off) = ot.project(s, e, "integrate", segments=True)
    up = rng.normal(size=len(s))
    ray = np.repeat(np.arange(len(s)), np.diff(off))
    want = np.zeros(len(pc.pos_orig))
    np.add.at(want, lp["orig_ids"][cell], up[ray] * (s_exit - s_enter))
    f = torch.tensor(pc.fields_orig, device="cuda", requires_grad=True)
    for _ in range(2):
        img = VA.project(pc, f, s, e)
        grad, = torch.autograd.grad(img, f, torch.as_tensor(up, device="cuda"))
        np.testing.assert_allclose(grad.cpu().numpy(), want, rtol=1e-12,
                                   atol=1e-14 * np.abs(want).max())
    assert _has_lists(pc)


def test_limits_and_rebuilt_tree():
    """Lowered limits act as in the other kernels; a rebuilt tree drops the
    lists, and a graph captured before it refuses to launch."""
    import torch
    from vortrace_b200 import _lib as L
    from vortrace_b200.graph import ProjectionGraph
    pc, ot, lp, (s, e) = _setup("uniform4001", lambda n: np.ones(n))
    want = ot.project(s, e, "integrate").reshape(-1)
    np.testing.assert_array_equal(pc.projection(s, e), want)
    pc._cloud.set_param(L.PARAM_LOCAL_STACK, 2)
    np.testing.assert_array_equal(pc.projection(s, e), want)
    assert pc.last_stats["slow_rays"] > 0
    pc._cloud.set_param(L.PARAM_LOCAL_STACK, 1 << 30)
    pc._cloud.set_param(L.PARAM_MAX_ITERATIONS, 3)
    with pytest.raises(L.VortraceError, match="maximum iteration count"):
        pc.projection(s, e)
    pc._cloud.set_param(L.PARAM_MAX_ITERATIONS, 100000)
    bad = s.copy()
    bad[7, 1] = np.nan
    with pytest.raises(ValueError, match="ray 7"):
        pc.projection(bad, e)
    g = ProjectionGraph(pc, torch.as_tensor(s, device="cuda"), torch.as_tensor(e, device="cuda"))
    g.launch()
    g.finish()
    np.testing.assert_array_equal(g.out.cpu().numpy().reshape(-1), want)
    pc._cloud.buildTree()
    assert not _has_lists(pc)
    with pytest.raises(L.VortraceError, match="reallocated"):
        g.launch()
    np.testing.assert_array_equal(pc.projection(s, e), want)
