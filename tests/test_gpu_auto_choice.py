"""AUTO between the lists and the tree: when the lists are built, and that a cloud
on which they do not pay goes back to the tree.  The walks tell themselves apart by
their queries: two or more per crossing on the tree, two per ray and the asks on
the lists."""
import warnings

import numpy as np
import pytest

from vortrace_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _cloud(kind, n):
    import vortrace_b200 as vt
    rng = np.random.default_rng(n)
    if kind == "uniform":
        pos = rng.uniform(0, 100, (n, 3))
    else:
        pos = np.vstack([W._plummer(rng, 9 * n // 10, 2.0, np.full(3, 50.0), 40.0),
                         rng.uniform(0, 100, (n - 9 * n // 10, 3))])
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return vt.ProjectionCloud(pos, rng.uniform(0, 1, n), boundbox=[0, 100.0] * 3)


def _grid(k, lo, hi):
    x = lo + (np.arange(k) + 0.5) * (hi - lo) / k
    a, b = np.meshgrid(x, x, indexing="ij")
    s = np.stack([a.ravel(), b.ravel(), 0 * a.ravel()], 1)
    e = s.copy()
    e[:, 2] = 100.0
    return s, e


def _walks(pc, s, e, want, calls):
    """Which walk each of the calls ran on."""
    out = []
    for _ in range(calls):
        np.testing.assert_array_equal(pc.projection(s, e), want)
        st = pc.last_stats
        out.append("tree" if st["queries"] > 1.5 * st["crossings"] else "list")
    return out


def test_lists_are_built_when_they_pay():
    s, e = _grid(32, 0, 100)
    pc = _cloud("uniform", 20000)
    pc.kernel = "plain"
    want = pc.projection(s, e)
    pc.kernel = "auto"
    walks = _walks(pc, s, e, want, 6)
    # 1,024 rays of 41 crossings at 10 ns: 0.4 ms a call towards 1.05 ms
    assert walks == ["tree", "tree", "list", "list", "list", "list"]
    s, e = _grid(256, 0, 100)
    pc.kernel = "plain"
    want = pc.projection(s, e)
    pc.kernel = "auto"
    pc._cloud.buildTree()
    assert _walks(pc, s, e, want, 3) == ["list"] * 3


def test_clouds_that_lists_do_not_fit_go_back_to_the_tree():
    """20,000 clustered points ask the tree at half of the crossings: 2 times slower
    on the lists at 1,024 rays."""
    s, e = _grid(32, 40, 60)
    pc = _cloud("clustered", 20000)
    pc.kernel = "plain"
    want = pc.projection(s, e)
    pc.kernel = "auto"
    walks = _walks(pc, s, e, want, 80)
    first = walks.index("list")
    # tried, left after one or two launches, tried again once in 32
    assert walks.count("list") <= 4 and walks[first + 2: first + 20] == ["tree"] * 18
    assert "list" in walks[first + 20:]


@pytest.mark.parametrize("kind,n,k,lists", [("uniform", 360_000, 180, True),
                                            ("clustered", 20_000, 32, False)])
@pytest.mark.parametrize("leaf_size", [False, True])
def test_autotune_takes_the_faster_walk(kind, n, k, lists, leaf_size):
    """360,000 points in leaves of up to 12 (more than 8 of them) can have no lists:
    a leaf size that wins among the tree kernels must not keep them away."""
    s, e = _grid(k, *((0, 100) if kind == "uniform" else (40, 60)))
    pc = _cloud(kind, n)
    pc.kernel = "plain"
    want = pc.projection(s, e)
    pc.kernel = "auto"
    res = pc.autotune(s, e, leaf_size=leaf_size)
    assert res["lists"] == lists and res["kernel"] in ("thread_fp32", "batched_fp64", "batched")
    assert _walks(pc, s, e, want, 4) == ["list" if lists else "tree"] * 4


def _nested():
    import vortrace_b200 as vt
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        pos = W.nested_cloud(20_000, 5)[0]
        return vt.ProjectionCloud(pos, np.ones(len(pos)), boundbox=[0, 100.0] * 3)


def test_clouds_of_compact_groups_start_on_the_tree():
    """The lists of compact groups leave the long sides of the cells around them open,
    which the lists themselves tell: 6 to 8 times slower at 16,384 rays.  A first call
    (a series of snapshots makes no other) and a graph, whose launches are not timed,
    go to the tree; lists are tried once and left."""
    import torch
    from vortrace_b200.graph import ProjectionGraph
    s, e = _grid(128, 0, 100)
    pc = _nested()
    pc.kernel = "plain"
    want = pc.projection(s, e)
    pc = _nested()
    g = ProjectionGraph(pc, torch.as_tensor(s, device="cuda"), torch.as_tensor(e, device="cuda"))
    g.launch()
    st = g.finish()
    assert st["queries"] > 1.5 * st["crossings"]
    np.testing.assert_array_equal(g.out.cpu().numpy().reshape(want.shape), want)
    pc._cloud.neighbour_lists()  # (they were built)
    pc = _nested()
    walks = _walks(pc, s, e, want, 30)
    assert walks[:2] == ["tree"] * 2 and walks.count("list") <= 2
    S, E = _grid(128, 0, 100)
    g = ProjectionGraph(pc, torch.as_tensor(S, device="cuda"), torch.as_tensor(E, device="cuda"))
    g.launch()
    st = g.finish()
    assert st["queries"] > 1.5 * st["crossings"]


def test_graph_on_a_cloud_that_lists_fit():
    import torch
    from vortrace_b200.graph import ProjectionGraph
    s, e = _grid(128, 0, 100)
    pc = _cloud("uniform", 20_000)
    g = ProjectionGraph(pc, torch.as_tensor(s, device="cuda"), torch.as_tensor(e, device="cuda"))
    g.launch()
    st = g.finish()
    assert st["queries"] < 0.5 * st["crossings"]
