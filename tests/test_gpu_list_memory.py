"""Device memory of the list walk: records for the rays in flight only, a limit that
a caller can set, and what becomes of lists above it."""
import warnings

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cloud(n=20000):
    import vortrace_b200 as vt
    rng = np.random.default_rng(n)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        pc = vt.ProjectionCloud(rng.uniform(0, 100, (n, 3)), np.ones(n), boundbox=[0, 100.0] * 3)
    s, e = rng.uniform(0, 100, (2, 16384, 3))
    return pc, s, e


def _has_lists(pc):
    from vortrace_b200 import _lib as L
    try:
        pc._cloud.neighbour_lists()
    except L.VortraceError:
        return False
    return True


def test_records_are_for_the_rays_in_flight():
    """16,384 rays run as 2,960 warps of 6 rays: 73 MB of records, not 388 MB."""
    import torch
    other, a, b = _cloud(3000)
    other.projection(a, b)  # the kernel's code and stacks
    assert _has_lists(other)
    pc, s, e = _cloud()
    pc.kernel = "thread_fp32"
    pc.projection(s, e)  # the other workspaces
    free = torch.cuda.mem_get_info()[0]
    pc.kernel = "auto"
    pc.projection(s, e)
    assert _has_lists(pc)
    lists = 1028 * len(pc.orig_ids)
    assert free - torch.cuda.mem_get_info()[0] < lists + 120e6


def test_limit():
    import torch
    from vortrace_b200 import _lib as L
    from vortrace_b200.graph import ProjectionGraph
    pc, s, e = _cloud()
    lists = 1028 * len(pc.orig_ids)
    pc.kernel = "plain"
    want = pc.projection(s, e)
    pc.kernel = "auto"
    S, E = torch.as_tensor(s, device="cuda"), torch.as_tensor(e, device="cuda")
    for limit, built in ((0, False), (lists // 2, False), (lists + 80_000_000, True), (-1, True),
                         (lists // 2, False), (-1, True)):
        pc.limit_lists(limit)
        np.testing.assert_array_equal(pc.projection(s, e), want)
        assert _has_lists(pc) == built, limit
    g = ProjectionGraph(pc, S, E)
    g.launch()
    g.finish()
    np.testing.assert_array_equal(g.out.cpu().numpy().reshape(want.shape), want)
    pc.limit_lists(0)
    assert not _has_lists(pc)
    with pytest.raises(L.VortraceError, match="reallocated"):
        g.launch()
    g = ProjectionGraph(pc, S, E)  # on the tree: lists may come and go
    pc.limit_lists(-1)
    np.testing.assert_array_equal(pc.projection(s, e), want)
    assert _has_lists(pc)
    pc.limit_lists(0)
    g.launch()
    g.finish()
    np.testing.assert_array_equal(g.out.cpu().numpy().reshape(want.shape), want)
    with pytest.raises(ValueError, match="list bytes"):
        pc.limit_lists(-2)
