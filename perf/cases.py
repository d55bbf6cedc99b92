"""Performance cases of vortrace_b200: what its users have it do, through its
public entry points, over the range of cloud sizes, ray counts, reductions and
outputs it is used with.

Clouds are drawn like the benchmark workloads (``vortrace_b200/workloads.py``):
``uniform`` (a homogeneous box), ``clustered`` (90% Plummer sphere, 10%
uniform) and ``nested`` (eight Plummer clumps of scale 0.05 to 2, 5% uniform).
A case's ``kind`` says which entry point it goes through:

  rays      ProjectionCloud.projection of arbitrary rays on the host
  traced    ProjectionCloud.traced_projection with per-segment output
  image     ProjectionCloud.grid_projection of an unrotated grid
  snapshot  a new ProjectionCloud from host arrays and its first image
  slice     ProjectionCloud.slice
  fit       autograd.project forward and backward on device rays
  views     rotated views and random rays on the device, a replayed graph
"""
import math
import warnings

import numpy as np
import torch

import vortrace_b200 as vt
from vortrace_b200 import autograd as VA
from vortrace_b200 import grid as GR
from vortrace_b200.graph import ProjectionGraph

BOX = [0.0, 100.0, 0.0, 100.0, 0.0, 100.0]


def listed():
    return [
        # a few hundred absorption sightlines through a small box: a call
        # where launches and latency count
        dict(name="sightlines_300", kind="rays", cloud="uniform", n=100_000, nf=1,
             rays=300, reduction="integrate"),
        # per-segment output (cell ids, positions, lengths) of a bundle of
        # rays, as spectra and light-curve codes read it
        dict(name="traced_5k", kind="traced", cloud="clustered", n=700_000, nf=3,
             rays=5_003, reduction="integrate"),
        # quick look at a small box (the 128 x 128 benchmark grid)
        dict(name="image_128_100k", kind="image", cloud="uniform", n=100_000, nf=1,
             nx=128, ny=128, reduction="integrate", periodic=False),
        # an image of a periodic box, odd sizes
        dict(name="periodic_181x149", kind="image", cloud="uniform", n=150_000, nf=2,
             nx=181, ny=149, reduction="integrate", periodic=True),
        # a time series: every snapshot is loaded and gets one maximum image
        dict(name="snapshot_1m_max", kind="snapshot", cloud="clustered", n=1_000_000, nf=2,
             nx=300, ny=217, reduction="max"),
        # a slice through a large cloud
        dict(name="slice_1024_2m", kind="slice", cloud="clustered", n=2_000_000, nf=3,
             nx=1024, ny=1024),
        # volume rendering at the 512 x 512 benchmark size
        dict(name="volume_512_2m", kind="image", cloud="clustered", n=2_000_000, nf=4,
             nx=512, ny=512, reduction="volume", periodic=False),
        # one step of a fit of the cells' fields to an image: forward, backward
        dict(name="fit_sum_512_2m", kind="fit", cloud="clustered", n=2_000_000, nf=3,
             nx=512, ny=512, reduction="integrate"),
        # one step of a fit of colours and opacities to a rendered image
        dict(name="fit_volume_256_1m", kind="fit", cloud="clustered", n=1_000_000, nf=4,
             nx=256, ny=250, reduction="volume"),
        # the headline image: three fields at 1024 x 1024
        dict(name="image_1024_2m", kind="image", cloud="clustered", n=2_000_000, nf=3,
             nx=1024, ny=1024, reduction="integrate", periodic=False),
        # a fly-around: 64 rotated views and random rays in one launch, device
        # buffers, replayed
        dict(name="views_64_1m", kind="views", cloud="clustered", n=1_000_000, nf=1,
             nviews=64, npix=256, rays=10_000, reduction="integrate"),
        # the largest: a 16M-cell zoom at 2048 x 2048
        dict(name="image_2048_16m", kind="image", cloud="nested", n=16_000_000, nf=1,
             nx=2048, ny=2048, reduction="integrate", periodic=False),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "traced", "image", "image", "image", "periodic", "snapshot",
                       "slice", "fit", "fit", "views"])
    cloud = rng.choice(["uniform", "clustered", "clustered", "nested"])
    n = _logint(rng, 20_000, 4_000_000)
    red = rng.choice(["integrate", "integrate", "volume", "max", "min"])
    nf = 4 if red == "volume" else rng.choice([1, 1, 2, 3, 5])
    if kind == "rays":
        return dict(kind=kind, cloud=cloud, n=n, nf=nf, rays=_logint(rng, 100, 300_000),
                    reduction=red)
    if kind == "traced":
        return dict(kind=kind, cloud=cloud, n=n, nf=nf, rays=_logint(rng, 50, 20_000),
                    reduction=red)
    if kind == "periodic":
        n = _logint(rng, 20_000, 400_000)
        return dict(kind="image", cloud="uniform", n=n, nf=nf, nx=_logint(rng, 40, 250),
                    ny=_logint(rng, 40, 250), reduction=red, periodic=True)
    if kind == "image":
        return dict(kind=kind, cloud=cloud, n=n, nf=nf, nx=_logint(rng, 64, 1500),
                    ny=_logint(rng, 64, 1500), reduction=red, periodic=False)
    if kind == "snapshot":
        return dict(kind=kind, cloud=cloud, n=n, nf=nf, nx=_logint(rng, 50, 700),
                    ny=_logint(rng, 50, 700), reduction=red)
    if kind == "slice":
        return dict(kind=kind, cloud=cloud, n=n, nf=nf, nx=_logint(rng, 100, 2000),
                    ny=_logint(rng, 100, 2000))
    if kind == "fit":
        red = rng.choice(["integrate", "volume"])
        return dict(kind=kind, cloud=cloud, n=n, nf=4 if red == "volume" else nf,
                    nx=_logint(rng, 64, 600), ny=_logint(rng, 64, 600), reduction=red)
    return dict(kind="views", cloud=cloud, n=n, nf=nf, nviews=_logint(rng, 4, 48),
                npix=_logint(rng, 64, 256), rays=_logint(rng, 100, 20_000), reduction=red)


# ------------------------------------------------------------------ inputs
def _dev():
    return torch.device("cuda", 0)


def _uniform(g, shape, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(shape, generator=g, dtype=torch.float64, device=_dev())


def _normal(g, shape):
    return torch.randn(shape, generator=g, dtype=torch.float64, device=_dev())


def _plummer(g, n, a, centre, rmax):
    """n points of a Plummer sphere of scale a, truncated at rmax."""
    mmax = rmax ** 3 / (rmax ** 2 + a ** 2) ** 1.5
    m = _uniform(g, n).clamp_min(1e-12) * mmax
    r = a / torch.sqrt(m ** (-2.0 / 3.0) - 1.0)
    v = _normal(g, (n, 3))
    v /= v.norm(dim=1, keepdim=True)
    return centre + r[:, None] * v


def _cloud(case, seed):
    """A generator for the rays, positions (n, 3) and density (n,) on the
    device.  The number of segments of a traced bundle follows from its
    geometry, so that kind has one mesh and one bundle of rays, and other
    fields for each seed."""
    g = torch.Generator(device=_dev()).manual_seed(
        11 if case["kind"] == "traced" else seed * 7919 + 17)
    n, c = case["n"], torch.full((3,), 50.0, dtype=torch.float64, device=_dev())
    if case["cloud"] == "uniform":
        return g, _uniform(g, (n, 3), 0.0, 100.0), torch.exp(_normal(g, n))
    if case["cloud"] == "clustered":
        a, nc = 2.0, int(round(0.9 * n))
        pos = torch.cat([_plummer(g, nc, a, c, 40.0), _uniform(g, (n - nc, 3), 0.0, 100.0)])
        r2 = ((pos - c) ** 2).sum(1)
        return g, pos, (1.0 + r2 / a ** 2) ** -2.5 * torch.exp(0.3 * _normal(g, n))
    nc, k = int(round(0.95 * n)), 8
    a = torch.exp(_uniform(g, k, math.log(0.05), math.log(2.0))).tolist()
    cs = 50.0 + 4.0 * _normal(g, (k, 3))
    cnt = [nc // k + (1 if i < nc % k else 0) for i in range(k)]
    pos = torch.cat([_plummer(g, cnt[i], a[i], cs[i], 20.0 * a[i]) for i in range(k)]
                    + [_uniform(g, (n - nc, 3), 0.0, 100.0)])
    rho = torch.zeros(n, dtype=torch.float64, device=_dev())
    for i in range(k):
        rho += a[i] ** -3 * (1.0 + ((pos - cs[i]) ** 2).sum(1) / a[i] ** 2) ** -2.5
    return g, pos, rho / rho.max() * torch.exp(0.3 * _normal(g, n))


def _fields(case, seed, rho):
    n, nf = rho.shape[0], case["nf"]
    g = torch.Generator(device=_dev()).manual_seed(seed * 7919 + 4001)
    rho = rho * torch.exp(0.1 * _normal(g, n))
    if case.get("reduction") == "volume":
        # three colour bands in log density, as in the volume benchmark
        lr = torch.log10(rho.clamp_min(1e-300))
        cen = torch.tensor([-1.0, 0.5, 2.0], dtype=torch.float64, device=rho.device)
        col = torch.tensor([[0.25, 0.45, 1.0], [0.3, 1.0, 0.35], [1.0, 0.35, 0.2]],
                           dtype=torch.float64, device=rho.device)
        b = torch.exp(-0.5 * ((lr[:, None] - cen) / 0.25) ** 2)
        return torch.cat([(b @ col).clamp(0.0, 1.0), (0.05 * b.sum(1)).clamp(0.0, 1.0)[:, None]],
                         1).contiguous()
    cols = [rho] + [rho * torch.exp(0.5 * _normal(g, n)) for _ in range(nf - 1)]
    return rho if nf == 1 else torch.stack(cols, 1).contiguous()


def _extent(case):
    """The square the images cover: the box, or the clustered part's centre."""
    return [0.0, 100.0] if case["cloud"] == "uniform" else [40.0, 60.0]


def _rays(case, g):
    """Arbitrary rays: uniform end points in the box, and for clustered clouds
    half of them through the central region."""
    m = case["rays"]
    s, e = _uniform(g, (m, 3), 0.0, 100.0), _uniform(g, (m, 3), 0.0, 100.0)
    if case["cloud"] != "uniform":
        h = m // 2
        mid = 50.0 + 4.0 * _normal(g, (h, 3))
        d = _normal(g, (h, 3))
        d /= d.norm(dim=1, keepdim=True)
        s[:h], e[:h] = mid - 30.0 * d, mid + 30.0 * d
    return s, e


def _rotations(g, k):
    q = _normal(g, (k, 4))
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).T
    return torch.stack([
        torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)], 1),
        torch.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], 1),
        torch.stack([2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1)], 1)


def _inputs(case, seed):
    g, pos, rho = _cloud(case, seed)
    return g, pos, _fields(case, seed, rho)


def _view_rays(case, g):
    """nviews rotated pixel grids (30 x 30 about the centre, bounds past the
    box's corners), then the random rays."""
    p, half = case["npix"], 50.0 * math.sqrt(3.0)
    x = 35.0 + (torch.arange(p, dtype=torch.float64, device=_dev()) + 0.5) * (30.0 / p)
    gx, gy = torch.meshgrid(x - 50.0, x - 50.0, indexing="ij")
    base = torch.stack([gx.reshape(-1), gy.reshape(-1), torch.zeros(p * p, dtype=torch.float64,
                                                                    device=_dev())], 1)
    off = torch.tensor([0.0, 0.0, half], dtype=torch.float64, device=_dev())
    s, e = [], []
    for r in _rotations(g, case["nviews"]):
        s.append((base - off) @ r.T + 50.0)
        e.append((base + off) @ r.T + 50.0)
    rs, re = _rays(case, g)
    return torch.cat(s + [rs]).contiguous(), torch.cat(e + [re]).contiguous()


def _make(pos, fields, **kw):
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return vt.ProjectionCloud(pos, fields, boundbox=BOX, **kw)


def prepare(case, seed):
    g, pos, fields = _inputs(case, seed)
    st = dict(case=case)
    hp, hf = pos.cpu().numpy(), fields.cpu().numpy()
    if case["kind"] == "snapshot":
        st.update(pos=hp, fields=hf, vol=np.full(case["n"], 1e6 / case["n"]))
        return st
    st["pc"] = _make(hp, hf, periodic=case.get("periodic", False))
    if case["kind"] in ("rays", "traced"):
        s, e = _rays(case, g)
        st.update(starts=s.cpu().numpy(), ends=e.cpu().numpy())
    elif case["kind"] == "fit":
        s, e = GR.generate_projection_grid(_extent(case), (case["nx"], case["ny"]),
                                           [0.0, 100.0], None)
        st.update(starts=torch.as_tensor(s.reshape(-1, 3)).to(_dev()),
                  ends=torch.as_tensor(e.reshape(-1, 3)).to(_dev()),
                  fields=fields.clone().requires_grad_(True))
        nout = 3 if case["reduction"] == "volume" else case["nf"]
        shape = (case["nx"] * case["ny"],) + ((nout,) if fields.dim() > 1 else ())
        st["upstream"] = _normal(g, shape)  # dL/dimage of the fit's loss
    elif case["kind"] == "views":
        s, e = _view_rays(case, g)
        st["graph"] = ProjectionGraph(st["pc"], s, e, reduction=case["reduction"])
    return st


# --------------------------------------------------------------- one pass
def run(state):
    case, pc = state["case"], state.get("pc")
    kind = case["kind"]
    if kind == "rays":
        return pc.projection(state["starts"], state["ends"], reduction=case["reduction"])
    if kind == "traced":
        return pc.traced_projection(state["starts"], state["ends"], reduction=case["reduction"],
                                    flatten=True)
    if kind == "image":
        return pc.grid_projection(_extent(case), (case["nx"], case["ny"]), [0.0, 100.0], None,
                                  reduction=case["reduction"])
    if kind == "snapshot":
        pc = _make(state["pos"], state["fields"], vol=state["vol"])
        img = pc.grid_projection(_extent(case), (case["nx"], case["ny"]), [0.0, 100.0], None,
                                 reduction=case["reduction"])
        return img, pc.orig_ids
    if kind == "slice":
        lo, hi = _extent(case)
        return pc.slice([lo, hi, lo, hi], (case["nx"], case["ny"]), 50.0)
    if kind == "fit":
        img = VA.project(pc, state["fields"], state["starts"], state["ends"],
                         reduction=case["reduction"])
        grad, = torch.autograd.grad(img, state["fields"], state["upstream"])
        return img.detach(), grad
    state["graph"].launch()
    state["graph"].finish()
    return state["graph"].out


# ------------------------------------------------------------- least work
def _nrays(case):
    if case["kind"] in ("rays", "traced"):
        return case["rays"]
    if case["kind"] == "views":
        return case["nviews"] * case["npix"] ** 2 + case["rays"]
    return case["nx"] * case["ny"]


def work(case):
    n, nf, m = case["n"], case["nf"], _nrays(case)
    nout = 3 if case.get("reduction") == "volume" else nf
    if case["kind"] == "slice":
        # positions and fields once, the image once; one distance per pixel
        return {"bytes": n * (24 + 8 * nf) + m * 8 * nf, "flops": m * 8}
    # cells a ray crosses: about 1.5 cube roots of the cloud's size
    cross = m * 1.5 * n ** (1.0 / 3.0)
    ray_in = 0 if case["kind"] in ("image", "snapshot") else 48 * m  # grids: made in the call
    b = n * (24 + 8 * nf) + ray_in + m * 8 * nout
    f = cross * (20 + 2 * nout)  # a bisector and the reduction per crossing
    if case["kind"] == "traced":
        b += cross * 24 + 8 * m
    if case["kind"] == "fit":
        b += m * 8 * nout + n * 8 * nf
        f += cross * 4 * nout
    if case["kind"] == "snapshot":
        b += n * 8 * 2 + n * 8  # the volumes and the kept ids
    return {"bytes": b, "flops": f}


# ------------------------------------------------------- 64-bit references
def _envelope(pos, s, e, periodic):
    """For a block of rays, step by step: (cell, length) of the Voronoi cells
    they cross.  Along a ray the squared distance to a generator is t^2 - 2 a t
    + b, so the cells are the lower envelope of the lines b - 2 a t."""
    d = e - s
    length = d.norm(dim=1)
    d = d / length[:, None]
    a = d @ pos.T - (s * d).sum(1)[:, None]
    b = torch.zeros_like(a)
    for j in range(3):
        b += (pos[None, :, j] - s[:, j, None]) ** 2
    rows = torch.arange(s.shape[0], device=s.device)
    cur = b.argmin(1)
    t = torch.zeros_like(length)
    while True:
        ac, bc = a[rows, cur], b[rows, cur]
        den = a - ac[:, None]
        x = torch.where(den > 1e-12, 0.5 * (b - bc[:, None]) / den, math.inf)
        nxt_t, nxt = x.min(1)
        end = torch.minimum(torch.maximum(nxt_t, t), length)
        yield cur, end - t
        t = end
        if bool((nxt_t >= length).all()):
            return
        cur = torch.where(nxt_t < length, nxt, cur)


def _reduce(case, pos, fields, s, e):
    F = fields if fields.dim() > 1 else fields[:, None]
    red = case["reduction"]
    out = []
    block = max(1, min(2048, int(1.2e9 // pos.shape[0])))
    for i in range(0, s.shape[0], block):
        acc, T = None, None
        for cell, ds in _envelope(pos, s[i:i + block], e[i:i + block], False):
            f, on = F[cell], (ds > 0)[:, None]
            if red == "volume":
                acc = torch.zeros_like(f[:, :3]) if acc is None else acc
                T = torch.ones_like(ds) if T is None else T
                o = 1.0 - torch.exp(-f[:, 3] * ds)
                acc = acc + (T * o)[:, None] * f[:, :3]
                T = T * (1.0 - o)
            elif red == "integrate":
                acc = ds[:, None] * f + (0.0 if acc is None else acc)
            else:
                pick = torch.maximum if red == "max" else torch.minimum
                acc = f.clone() if acc is None else torch.where(on, pick(acc, f), acc)
        out.append(acc)
    return torch.cat(out)


def exact(case, seed):
    kind, m = case["kind"], _nrays(case)
    if kind == "slice":
        if m * case["n"] > 3e11:
            return None  # too long without a search structure
    elif (kind not in ("rays", "image") or case.get("periodic")
          or m * case["n"] * 1.5 * case["n"] ** (1.0 / 3.0) > 2.5e11):
        return None
    g, pos, fields = _inputs(case, seed)
    F = fields if fields.dim() > 1 else fields[:, None]
    lo, hi = _extent(case)
    if kind == "slice":
        x = lo + (hi - lo) / (case["nx"] - 1) * torch.arange(case["nx"], dtype=torch.float64,
                                                             device=_dev())
        y = lo + (hi - lo) / (case["ny"] - 1) * torch.arange(case["ny"], dtype=torch.float64,
                                                             device=_dev())
        q = torch.stack([v.reshape(-1) for v in torch.meshgrid(x, y, indexing="ij")], 1)
        near = []
        block = max(1, int(1.2e9 // case["n"]))
        for i in range(0, q.shape[0], block):
            r2 = ((q[i:i + block, None, 0] - pos[None, :, 0]) ** 2
                  + (q[i:i + block, None, 1] - pos[None, :, 1]) ** 2 + (50.0 - pos[:, 2]) ** 2)
            near.append(r2.argmin(1))
        out = F[torch.cat(near)].reshape(case["nx"], case["ny"], -1)
    else:
        if kind == "rays":
            s, e = _rays(case, g)
        else:
            hs, he = GR.generate_projection_grid([lo, hi], (case["nx"], case["ny"]),
                                                 [0.0, 100.0], None)
            s, e = (torch.as_tensor(v.reshape(-1, 3)).to(_dev()) for v in (hs, he))
        out = _reduce(case, pos, fields, s, e)
        if kind == "image":
            out = out.reshape(case["nx"], case["ny"], -1)
    return (out[..., 0] if out.shape[-1] == 1 else out).cpu().numpy()
