"""Rays that the list walk leaves to the tree kernels: lattices (a degenerate split
point on every ray), cells near the tolerance, a box of 1e16, against the
one-ray-per-thread FP64 walk bit for bit (gradients within the rounding of their
sums).  Ray counts on both sides of the switch between one ray per warp and one per
thread, with 1 to 32 rays to a warp of the list walk; more than 32 fields."""
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(kind, nf):
    import vortrace_b200 as vt
    rng = np.random.default_rng(len(kind))
    box = {"lattice": 16.0, "mixed": 16.0, "tiny": 2e-3, "huge": 1e16}[kind]
    if kind in ("lattice", "mixed"):
        c = np.arange(16) + 0.5
        pos = np.stack(np.meshgrid(c, c, c, indexing="ij"), -1).reshape(-1, 3)
        if kind == "mixed":  # random points in one half: both kinds of ray in a warp
            move = pos[:, 0] > 8
            pos[move] = rng.uniform(0, 16, (move.sum(), 3)) * [0.5, 1, 1] + [8, 0, 0]
    else:
        pos = rng.uniform(0, box, (4000, 3))
    f = rng.uniform(0, 1, (len(pos), nf))
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return vt.ProjectionCloud(pos, f, boundbox=[0.0, box] * 3), rng, box


def _rays(rng, m, box):
    """Two thirds along z, inside the cells' columns, the others across."""
    s, e = rng.uniform(0, box, (2, m, 3))
    k = 2 * m // 3
    e[:k, :2] = s[:k, :2]
    s[:k, 2], e[:k, 2] = 0.0, box
    return s, e


def _with(pc, kernel, call):
    pc.kernel = kernel
    return call()


@pytest.mark.parametrize("kind", ["lattice", "mixed", "tiny", "huge"])
@pytest.mark.parametrize("m,nf,reduction", [(700, 1, "integrate"), (700, 2, "max"),
                                            (700, 33, "integrate"), (140001, 4, "volume"),
                                            (110001, 1, "integrate")])
def test_image_is_the_plain_one(kind, m, nf, reduction):
    pc, rng, box = _case(kind, nf)
    s, e = _rays(rng, m, box)
    want = _with(pc, "plain", lambda: pc.projection(s, e, reduction=reduction))
    pc.kernel = "auto"
    for _ in range(2):
        np.testing.assert_array_equal(pc.projection(s, e, reduction=reduction), want)
        assert pc.last_stats["rays"] == m
    pc._cloud.neighbour_lists()  # they are built
    # the global-memory stack is for few rays
    assert pc.last_stats["slow_rays"] <= m // 100


@pytest.mark.parametrize("m", [500, 66001])
def test_coordinates_whose_squares_leave_fp32(m):
    """No lists there, and one warp per ray hands its rays over."""
    import vortrace_b200 as vt
    rng = np.random.default_rng(8)
    pos, (s, e) = rng.uniform(0, 1e21, (4000, 3)), _rays(rng, m, 1e21)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        pc = vt.ProjectionCloud(pos, np.ones(4000), boundbox=[0.0, 1e21] * 3)
    want = _with(pc, "plain", lambda: pc.projection(s, e))
    pc.kernel = "auto"
    for _ in range(2):
        np.testing.assert_array_equal(pc.projection(s, e), want)


@pytest.mark.parametrize("kind", ["lattice", "mixed", "tiny"])
@pytest.mark.parametrize("m", [700, 110001])
def test_segments_and_gradients(kind, m):
    import torch
    from vortrace_b200 import _lib as L
    from vortrace_b200 import autograd as VA
    pc, rng, box = _case(kind, 3)
    s, e = _rays(rng, m, box)
    pc.projection(s, e)
    pc._cloud.buildTree()  # (the lists' next walks; AUTO may prefer the tree later)
    a, b = (_with(pc, k, lambda: pc.traced_projection(s, e, return_midpoint=False, flatten=True))
            for k in ("plain", "auto"))
    pc._cloud.neighbour_lists()
    for x, y in zip(a, b):
        np.testing.assert_array_equal(y, x)
    f = torch.tensor(pc.fields_orig, device="cuda", requires_grad=True)
    up = torch.as_tensor(rng.normal(size=(m, 3)), device="cuda")
    want, = torch.autograd.grad(VA.project(pc, f, s, e, kernel="plain"), f, up)
    for _ in range(2):  # from the tape
        pc._cloud.buildTree()
        got, = torch.autograd.grad(VA.project(pc, f, s, e), f, up)
        torch.testing.assert_close(got, want, rtol=1e-11, atol=1e-13 * float(want.abs().max()))
    grad = np.zeros((len(pc.orig_ids), 3))  # walked again
    out = np.ascontiguousarray(pc.projection(s, e))
    pc._cloud.buildTree()
    L.check(pc._cloud._lib.vt_project_adjoint(
        pc._cloud._h, L.dptr(s), L.dptr(e), m, L.REDUCE_SUM, L.dptr(out),
        L.dptr(np.ascontiguousarray(up.cpu().numpy())), L.dptr(grad)))
    np.testing.assert_allclose(grad, want.cpu().numpy(), rtol=1e-11,
                               atol=1e-13 * float(want.abs().max()))


def test_ray_that_goes_round():
    """A ray near a vertex of the mesh at large coordinates, on which the reference's
    walk goes round within its tolerance until its iteration limit: the same error
    from every kernel, also once the reference-order tree is there."""
    import vortrace_b200 as vt
    from vortrace_b200 import _lib as L
    rng = np.random.default_rng(0)
    pos = 1e4 * rng.uniform(0, 1, (rng.integers(70, 3000), 3)) + 1e5
    s = np.array([[106511.39264565839, 103293.52250029893, 108495.26246356587]])
    e = np.array([[106497.31696201646, 103146.07777772452, 108775.09324459988]])
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        pc = vt.ProjectionCloud(pos, np.ones(len(pos)), boundbox=[1e5, 1.1e5] * 3)
    a, b = 1e5 + 1e4 * rng.uniform(0.1, 0.9, (2, 4000, 3))
    pc.projection(a, b)
    pc._cloud.neighbour_lists()  # they are built
    want = pc.projection(a, b)
    pc._cloud.set_param(L.PARAM_MAX_ITERATIONS, 2000)
    for _ in range(2):
        for kernel in ("plain", "auto", "batched"):
            pc.kernel = kernel
            with pytest.raises(L.VortraceError, match="maximum iteration count"):
                pc.projection(s, e)
            with pytest.raises(L.VortraceError, match="maximum iteration count"):
                pc.traced_projection(s, e)
    pc.kernel = "auto"
    np.testing.assert_array_equal(pc.projection(a, b), want)
