"""The periodic walk with many rays to a warp (up to 32) and degenerate split points
on all or on a few of them, against the one-ray-per-thread periodic walk, bit for
bit (gradients within the rounding of their sums)."""
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(kind, m):
    """A 16 x 16 x 100 lattice, random points, or a lattice in one half and random points in
    the other; rays along the lattice's columns and across, none of which starts and
    ends in one cell."""
    import vortrace_b200 as vt
    rng = np.random.default_rng(m)
    a, c = (np.arange(16) + 0.5) / 16, (np.arange(100) + 0.5) / 100
    pos = np.stack(np.meshgrid(a, a, c, indexing="ij"), -1).reshape(-1, 3)
    if kind != "lattice":
        move = np.ones(len(pos), bool) if kind == "random" else pos[:, 0] > 0.5
        pos[move] = rng.uniform(0, 1, (move.sum(), 3)) * [0.5 if kind == "half" else 1, 1, 1] \
            + [0.5 if kind == "half" else 0, 0, 0]
    s, e = rng.uniform(0, 1, (2, m, 3))
    k = 2 * m // 3
    e[:k, :2] = s[:k, :2]
    s[:k, 2], e[:k, 2] = 0.006, 0.986
    e[k:] = np.where(np.abs(e[k:] - s[k:]).max(1, keepdims=True) < 0.2, (s[k:] + 0.4) % 1, e[k:])
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return vt.ProjectionCloud(pos, rng.uniform(0, 1, (len(pos), 3)), boundbox=[0, 1] * 3,
                                  periodic=True), s, e, rng


@pytest.mark.parametrize("kind", ["lattice", "half", "random"])
# rays a warp takes: 1, 3, 32 (148 SMs x 4 blocks x 4 warps)
@pytest.mark.parametrize("m", [901, 7003, 80021])
def test_equals_the_plain_walk(kind, m):
    import torch
    from vortrace_b200 import autograd as VA
    pc, s, e, rng = _case(kind, m)
    f = torch.tensor(pc.fields_orig, device="cuda", requires_grad=True)
    up = torch.as_tensor(rng.normal(size=(m, 3)), device="cuda")
    got = {}
    for kernel in ("plain", "auto"):
        pc.kernel = kernel
        img = [pc.projection(s, e), pc.projection(s, e, reduction="max")]
        if kernel == "auto":
            assert pc.last_stats["rays"] == m and pc.last_stats["slow_rays"] <= m // 100
        img += list(pc.traced_projection(s, e, return_midpoint=False, flatten=True))
        grad, = torch.autograd.grad(VA.project(pc, f, s, e, kernel=kernel), f, up)
        got[kernel] = img, grad
    for a, b in zip(got["plain"][0], got["auto"][0]):
        np.testing.assert_array_equal(b, a)
    want = got["plain"][1]
    torch.testing.assert_close(got["auto"][1], want, rtol=1e-11,
                               atol=1e-13 * float(want.abs().max()))
