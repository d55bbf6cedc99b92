"""Rays that follow a face of the mesh at an angle near the rounding of FP32: the
two cells' distances differ by 1e-8 to 1e-5 over the whole face, and the sign of the
approach is lost in FP32.  Segments against the CPU oracle, bit for bit."""
import warnings

import numpy as np
import pytest
from scipy.spatial import Voronoi

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _walks(ot, s, e):
    """Whether the reference resolves the ray (a face within its tolerance may not)."""
    try:
        ot.project(s, e, "integrate")
    except O.OracleError:
        return False
    return True


@pytest.mark.parametrize("angle", [1e-8, 3e-8, 1.2e-7, 2e-6])
@pytest.mark.parametrize("clustered", [False, True])
def test_rays_along_faces(angle, clustered):
    import vortrace_b200 as vt
    rng = np.random.default_rng(17)
    pos = rng.uniform(0, 100, (4000, 3))
    if clustered:
        pos[1000:] = np.clip(50 + 30 * rng.standard_t(2.0, (3000, 3)) / 4, 0, 100)
    vor = Voronoi(pos)
    s, e = [], []
    for (i, j), verts in zip(vor.ridge_points, vor.ridge_vertices):
        if -1 in verts or len(verts) < 4:
            continue
        y = vor.vertices[verts]
        if y.min() < 5 or y.max() > 95:
            continue
        mid, v = y.mean(0), pos[j] - pos[i]
        v /= np.linalg.norm(v)
        a, b = rng.permutation(len(y))[:2]
        d = y[a] + rng.uniform(0.2, 0.8) * (y[b] - y[a]) - mid  # in the face's plane
        d -= v * (d @ v)
        size = np.linalg.norm(d)
        if size < 0.05:
            continue
        d = d / size + rng.uniform(-angle, angle) * v
        s.append(mid - (size * rng.uniform(1, 6) + 1) * d)
        e.append(mid + (size * rng.uniform(1, 6) + 1) * d)
    s, e = np.array(s), np.array(e)
    assert len(s) > 5000
    f = rng.uniform(0, 1, len(pos))
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        pc = vt.ProjectionCloud(pos, f, boundbox=[0.0, 100.0] * 3)
        lp = O.load_points(pos, f, [0.0, 100.0] * 3)
    ot = O.OracleTree(lp["pts"], lp["fields"], lp["valid_rgba"])
    ok = [_walks(ot, s[k:k + 1], e[k:k + 1]) for k in range(len(s))]
    s, e = s[ok], e[ok]
    assert len(s) > 4000
    out, (cell, s_enter, s_exit, off) = ot.project(s, e, "integrate", segments=True)
    pc.projection(s, e)
    val, cid, se, ds, offsets = pc.traced_projection(s, e, return_midpoint=False, flatten=True)
    info = pc._cloud.info()
    assert info.device_bytes > 1000 * info.npart  # with the lists
    wrong = np.flatnonzero(np.diff(offsets) != np.diff(off))
    assert len(wrong) == 0, (len(wrong), len(s), wrong[:5])
    np.testing.assert_array_equal(cid, lp["orig_ids"][cell])
    np.testing.assert_array_equal(se, s_enter)
    np.testing.assert_array_equal(ds, s_exit - s_enter)
    np.testing.assert_array_equal(val, out.reshape(-1))
