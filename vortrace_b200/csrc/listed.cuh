// listed.cuh -- walk kernel on neighbour lists (nbrlist.cu): one ray per
// thread, no tree search per crossing.
//
// Along a ray the squared distance to a generator is t^2 plus a linear
// function of t, so the cells a ray crosses are the lower envelope of lines,
// and the exit from a cell is the nearest of the bisectors with the cell's
// neighbours.  A ray is walked in three passes:
//
//   march   steps from cell to cell, each exit from the cell's neighbour list
//           in FP32 coordinates relative to the cell, and records for every
//           cell its line (the FP64 foot of its generator on the ray and the FP32
//           squared offset, from which any two cells' boundary follows) and whether
//           the boundary into it is certified.  Where the list cannot tell, a
//           tree query at the boundary point does;
//   replay  the reference's insertions (src/ray.cpp:187-430: the nearest cell of
//           the split point of two pending cells) on the records alone: when
//           every split point falls on one recorded cell, clear of its
//           neighbours, the reference's walk is the marched sequence, and the
//           ray is reduced from it with the reference's FP64 split points;
//   walk    for the other rays (0.1% on clustered_2m) the reference's own loop
//           with FP64 queries on the tree, except where certified boundaries
//           give the answer.  A ray with many split points that the 3-NN does not
//           decide, or with more than two queries per cell, is left to the tree
//           kernels, launched next over what is left: clouds that the lists do not
//           fit (lattices, cells near the tolerance) cost little more than without
//           lists.
//
// The march is only a hint: results are the reference's bit for bit.  A boundary
// is certified when every generator other than its two cells is farther from the
// boundary point, in squared distance, by more than 4e-9 plus a bound of the FP64
// rounding (kTol is 1e-9):
//   * generators outside the list are farther than rho >= 2 r + slack from
//     the cell, r the boundary point's distance to it;
//   * listed ones ahead of the ray: their bisector is crossed later than the
//     chosen one by more than both error bounds (below);
//   * those behind the ray have receded since the entry point, so they are as far
//     as the certified entry made them; only the cell the ray came from has to
//     be looked at again.  Without a certified entry all listed ones are tested
//     at the exit point;
//   * or a bounded FP64 query at the boundary point finds its two cells only.
// The FP32 error of half the difference of squared distances to cell P and a
// listed point at v, num - tau den, in units of u = 2^-24 and with R = rho, |v| <= R,
// entry |w| <= 2 R (tested), tau <= 2.5 R:
//   entry point w     the rounding of d, of the entry before and of the steps from
//                     there, R' the rho of the cell before: (6 R' + 4 R) R;
//   num               v and v^2: 4.5 R^2, three fused steps of up to 2.5 R^2 and
//                     the subtraction of thr: 10 R^2;
//   tau               the approximate reciprocal and a product: 3 tau den: 7.5 R^2;
//   den               d, v and three fused steps: 5 R.  6 R are added, so that a den
//                     that is not positive is truly not: tau times 11 R: 27.5 R^2.
// 53.5 R^2 + 6 R' R in all; thr is 64 R^2 + 6 R' R above 2e-9 and the FP64 term.  The
// sign of den is what the points behind rest on: a ray that follows a face at an
// angle of 1e-8 stays for the whole face within 1e-7 of both cells, far above the
// tolerance, and a cell taken for behind that is not would be missed.
// A point that is not listed keeps 1.25 thr at the computed exit, which is off by up
// to thr / den: one that is crossed slower than the chosen point loses less than
// thr there, and one crossed faster would put the next step's exit before its
// entry, which is not certified.
// At a split point s between certified boundaries t_m < s < t_(m+1) the
// difference to every cell is a linear function that is above the bound at
// both ends, except for the two neighbours in the sequence, whose difference is
// slope * distance: when both exceed the bound the reference's 3-NN query
// finds cell m alone within its tolerance, and pushes it; at a certified
// boundary of adjacent cells it finds one of the two first, and accepts.
//
// The tree search of the other kernels costs 595 warp instructions per crossing;
// this kernel takes 68 (clustered_2m, 512x512), and is bound by the latency of
// dependent loads (7.5 of 12.6 cycles between two instructions of a warp): the
// lists (1 KB per point) and the records outgrow the L2.  Walk launch, tree
// search -> lists: clustered_2m 1024x1024 171.6 -> 31.1 ms (march with its queries
// 20 ms, replay and walk 7, reduction 4.5), uniform_100k 128x128 6.3 -> 0.67 ms,
// batched_1m 569 -> 167 ms (10 queries a ray outside the cloud).
#pragma once

namespace vt {

#ifndef VT_LIST_MINB
#define VT_LIST_MINB 5
#endif
// a warp's queries run when at most this many lanes go on for each that waits
#ifndef VT_LIST_WAIT
#define VT_LIST_WAIT 7
#endif
constexpr int kListBlock = 128;
constexpr int kListTries = 64;
// a ray that needs more than kListAsks + 2 x cells tree queries is left to the
// tree kernels
constexpr int kListAsks = 64;
// degenerate split points of a ray that are resolved here, and the most lanes of a
// warp that may meet one together
constexpr int kListRare = 4;
constexpr int kListRareLanes = 2;

__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Foot parameter of P on the ray's line and its squared offset from it; e: the
// offset.
__device__ __forceinline__ void foot(const RayGeom& g, double4 P, double& a, double& q,
                                     double (&e)[3]) {
  const double px = P.x - g.s[0], py = P.y - g.s[1], pz = P.z - g.s[2];
  a = fma(pz, g.d[2], fma(py, g.d[1], px * g.d[0]));
  e[0] = fma(-a, g.d[0], px);
  e[1] = fma(-a, g.d[1], py);
  e[2] = fma(-a, g.d[2], pz);
  q = fma(e[2], e[2], fma(e[1], e[1], e[0] * e[0]));
}

// March state of one ray.  The FP64 part (records) lags one cell behind the FP32
// part (the choice of the next cell), so that its arithmetic runs while the next
// cell's list is on its way.
struct March {
  double t, a, q;      // of the last settled cell: boundary into it, foot, offset^2
  int c1;              // the ray's last cell
  int i;               // record of the current cell
  int prev;            // cell of record i - 1 when it is not settled yet, else -1
  int nxt;             // candidate for the next cell when a query has to decide
  int tries;           // queries at the current cell
  float wx, wy, wz;    // entry point relative to the current cell's generator
  float px, py, pz;    // the same of `prev`, as it was used
  float den;           // rate of the entry boundary (half differences)
  float rho_in;        // rho of the cell that the entry point was found from (0: FP64)
  float rho_chain;     // smallest rho since the points behind were last tested
  float rho_max;
  bool all;            // every settled boundary is certified
  bool clean;          // the boundary into the current cell is certified
  bool prev_clean;     // the boundary into `prev`
};

// Write the record of cell `cell` (index i) from its FP64 point; w receives the
// entry point relative to it.  False when the march has to end.
__device__ __forceinline__ bool list_settle(const DevCloud& c, const RayGeom& g, WalkRec* rec,
                                            March& m, int cell, int i, bool clean, float (&w)[3]) {
  const double4 P = ldg_pt(&c.pts[cell]);
  double a, q, e[3];
  foot(g, P, a, q, e);
  if (i > 0) {
    const double da = a - m.a;
    m.t = 0.5 * ((a + m.a) + (q - m.q) / da);
    // (bisectors within the parallel tolerance of the ray are not certified)
    clean = clean && da > 5e-11;
    m.all = m.all && clean;
  }
  m.a = a;
  m.q = q;
  const float qf = (float)q;
  rec[i] = WalkRec{a, clean ? qf : -qf, cell};
  const double ta = m.t - a;
  w[0] = (float)fma(ta, g.d[0], -e[0]);
  w[1] = (float)fma(ta, g.d[1], -e[1]);
  w[2] = (float)fma(ta, g.d[2], -e[2]);
  return m.t < g.len;
}

// Take one step of the march from cell cur: settle the cell before, then find
// the next cell from the list.  kMarchOn: `cur` is the next cell; kMarchDone: the
// last record (index m.i) is written; kMarchAsk: a query has to tell whether m.nxt
// is the next cell.
enum { kMarchOn = 0, kMarchDone = 1, kMarchAsk = 2 };
__device__ __forceinline__ int list_step(const DevCloud& c, const RayGeom& g, double qm,
                                         WalkRec* rec, int cap, March& m, int& cur) {
  const float dx = (float)g.d[0], dy = (float)g.d[1], dz = (float)g.d[2];
  const bool up = dz > 0.f;
  const float4* grp = c.nbr + (int64_t)cur * (kNbrGroups * 4);
  const unsigned hdr = __ldg(&c.nbr_hdr[cur]);
  const float4* first = grp + (up ? 0 : 4 * (kNbrGroups - 1));
  float4 X = __ldg(first), Y = __ldg(first + 1), Z = __ldg(first + 2);
  bool go = true;
  if (m.prev >= 0) {
    float w[3];
    go = list_settle(c, g, rec, m, m.prev, m.i - 1, m.prev_clean, w);
    m.prev = -1;
    // the entry point as the FP64 one of the cell before puts it
    m.wx += w[0] - m.px;
    m.wy += w[1] - m.py;
    m.wz += w[2] - m.pz;
  }
  if (cur == m.c1 || !go || m.i >= cap - 2) {
    if (cur != m.c1) m.clean = false;  // c1 ends the sequence all the same
    float w[3];
    list_settle(c, g, rec, m, m.c1, m.i, m.clean, w);
    return kMarchDone;
  }
  const float hrho = __uint_as_float(hdr & ~1023u);  // rho^2 / 2
  const float rho = sqrtf(2.f * hrho);
  const float thr =
      2e-9f + fmaf((float)(2e-14 * qm) + 3.6e-7f * m.rho_in, rho, 7.7e-6f * hrho);
  const float w2 = fmaf(m.wx, m.wx, fmaf(m.wy, m.wy, m.wz * m.wz));
  const float wd = fmaf(m.wx, dx, fmaf(m.wy, dy, m.wz * dz));
  const float kInf = __int_as_float(0x7f800000);
  // candidate n: half the difference of squared distances at ray parameter tau
  // past the entry is num - tau den (positive while the ray is nearer to cur; den
  // rounded up);
  // lo = (num - thr) / den bounds its exit from below, lo + 2 thr / den from
  // above.  The smallest lo with its group slot and 1 / den, and the next one.
  float lo1 = kInf, lo2 = kInf, inv1 = 0.f, r2 = kInf;
  int bi = -1;
  bool ended = false;
  const float eps = 3.6e-7f * rho;
  const float2 half2 = make_float2(0.5f, 0.5f), mthr2 = make_float2(-thr, -thr),
               eps2 = make_float2(eps, eps);
  const float2 wx2 = make_float2(-m.wx, -m.wx), wy2 = make_float2(-m.wy, -m.wy),
               wz2 = make_float2(-m.wz, -m.wz);
  const float2 dx2 = make_float2(dx, dx), dy2 = make_float2(dy, dy), dz2 = make_float2(dz, dz);
  // one part of the list; X, Y, Z hold its first group
  auto scan = [&](const bool part_up) {
    const int n = (int)(part_up ? (hdr >> 5) & 31u : hdr & 31u);
    const int step = part_up ? 1 : -1;
    int k = part_up ? 0 : kNbrGroups - 1;
    const int end = k + step * n;
    ended = ended || n == 0;
#pragma unroll 1
    while (k != end) {
      const float2 vx[2] = {make_float2(X.x, X.y), make_float2(X.z, X.w)};
      const float2 vy[2] = {make_float2(Y.x, Y.y), make_float2(Y.z, Y.w)};
      const float2 vz[2] = {make_float2(Z.x, Z.y), make_float2(Z.z, Z.w)};
      const int at = 4 * k;
      k += step;
      if (k != end) {  // the next group's loads while this one is worked on
        X = __ldg(grp + 4 * k);
        Y = __ldg(grp + 4 * k + 1);
        Z = __ldg(grp + 4 * k + 2);
      } else {
        ended = true;
      }
      float2 vv[2];
#pragma unroll
      for (int p = 0; p < 2; ++p)
        vv[p] = __ffma2_rn(vx[p], vx[p], __ffma2_rn(vy[p], vy[p], __fmul2_rn(vz[p], vz[p])));
      // a point at |v| >= 2 r + slack cannot matter, nor can the later ones
      if (vv[0].x * 0.4999f >= fmaf(2.f, r2, 2.5f * thr)) {
        ended = ended && k != end;
        break;
      }
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const float2 num = __ffma2_rn(
            wx2, vx[p], __ffma2_rn(wy2, vy[p], __ffma2_rn(wz2, vz[p],
                                                          __ffma2_rn(half2, vv[p], mthr2))));
        const float2 den =
            __ffma2_rn(dx2, vx[p], __ffma2_rn(dy2, vy[p], __ffma2_rn(dz2, vz[p], eps2)));
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float dj = j ? den.y : den.x;
          const float inv = rcp_approx(dj);
          const float lo = dj > 0.f ? (j ? num.y : num.x) * inv : kInf;
          const bool less = lo < lo1;
          lo2 = fminf(lo2, fmaxf(lo, lo1));
          inv1 = less ? inv : inv1;
          bi = less ? at + 2 * p + j : bi;
          lo1 = fminf(lo, lo1);
        }
      }
      const float tau = fmaf(thr, inv1, lo1);
      r2 = bi >= 0 ? fmaf(tau, fmaf(2.f, wd, tau), w2) : kInf;
    }
  };
  scan(up);
  if (dx != 0.f || dy != 0.f) {
    // the other part's points are all behind a ray along z
    const float4* other = grp + (up ? 4 * (kNbrGroups - 1) : 0);
    X = __ldg(other);
    Y = __ldg(other + 1);
    Z = __ldg(other + 2);
    scan(!up);
  }
  m.tries = 0;
  m.nxt = m.c1;
  if (bi < 0) return kMarchAsk;
  const float best = fmaf(thr, inv1, lo1);
  const float* f = reinterpret_cast<const float*>(grp + 4 * (bi >> 2)) + (bi & 3);
  const float vx = __ldg(f), vy = __ldg(f + 4), vz = __ldg(f + 8);
  const int nxt = __float_as_int(__ldg(f + 12));
  if (nxt < 0) return kMarchAsk;
  m.nxt = nxt;
  const bool far = hrho >= fmaf(2.f, r2, 2.5f * thr);
  bool ok = (!ended || far) && lo2 > fmaf(2.f * thr, inv1, lo1) && w2 <= 8.f * hrho;
  // the entry vouches for the points behind, at the rounding level of the
  // smallest rho since they were last tested, except for the cell it left
  const bool chained = m.clean && rho <= 8.f * m.rho_chain;
  if (chained) {
    ok = ok && m.den * best > thr * fmaf(m.den, inv1, 1.f);
  } else if (ok) {
    ok = far;
    const float yx = fmaf(best, dx, m.wx), yy = fmaf(best, dy, m.wy), yz = fmaf(best, dz, m.wz);
    const int g_up = (int)((hdr >> 5) & 31u), ng = g_up + (int)(hdr & 31u);
#pragma unroll 1
    for (int k = 0; k < 4 * ng && ok; ++k) {
      const int slot = k < 4 * g_up ? k : 4 * kNbrGroups - 4 * ng + k;
      const float* b = reinterpret_cast<const float*>(grp + 4 * (slot >> 2)) + (slot & 3);
      const float ux = __ldg(b), uy = __ldg(b + 4), uz = __ldg(b + 8);
      const float h = 0.5f * fmaf(ux, ux, fmaf(uy, uy, uz * uz));
      const float G = h - fmaf(yx, ux, fmaf(yy, uy, yz * uz));
      const float den = fabsf(fmaf(dx, ux, fmaf(dy, uy, dz * uz)));
      if (slot != bi && !(G > thr * fmaf(den, inv1, 1.f))) ok = false;
    }
  }
  if (!ok) return kMarchAsk;
  m.rho_chain = chained ? fminf(m.rho_chain, rho) : rho;
  m.rho_max = fmaxf(m.rho_max, rho);
  m.rho_in = rho;
  m.prev = cur;
  m.prev_clean = m.clean;
  m.px = m.wx;
  m.py = m.wy;
  m.pz = m.wz;
  m.wx = fmaf(best, dx, m.wx) - vx;
  m.wy = fmaf(best, dy, m.wy) - vy;
  m.wz = fmaf(best, dz, m.wz) - vz;
  m.den = fmaf(dx, vx, fmaf(dy, vy, dz * vz));
  m.clean = true;
  cur = nxt;
  ++m.i;
  return kMarchOn;
}

// f_(i)(s) - f_(j)(s), f the squared distance from the ray's point s to the cells'
// generators; `err` grows by the rounding of the FP32 offsets.
__device__ __forceinline__ double line_diff(double ai, float qi, double aj, float qj, double s,
                                            float& err) {
  qi = fabsf(qi);
  qj = fabsf(qj);
  err = fmaf(1.3e-7f, qi + qj, err);
  return fma(aj - ai, 2.0 * s - ai - aj, (double)qi - (double)qj);
}

// Where the lines of cells i and j (records) cross.
__device__ __forceinline__ double line_cross(double ai, float qi, double aj, float qj) {
  return 0.5 * ((ai + aj) + ((double)fabsf(qj) - (double)fabsf(qi)) / (aj - ai));
}

// Whether the record arrays A (foot parameters) and Q give one cell m of (i, j) as
// the nearest at the crossing s of cells i and j, clear of its two neighbours in the
// sequence by more than `gap` in squared distance; m receives it.
template <class FA, class FQ>
__device__ __forceinline__ bool list_nearest(const FA& A, const FQ& Q, int i, int j, double s,
                                             double gap, int& m) {
  int lo = i + 1, hi = j - 1;
  while (lo < hi) {  // the last foot up to s, then the lowest line around it
    const int mid = (lo + hi + 1) >> 1;
    if (A(mid) <= s) lo = mid;
    else hi = mid - 1;
  }
  float err = 1.3e-7f * (fabsf(Q(i)) + fabsf(Q(j)));
  float none = 0.f;
  double am = A(lo);
  float qm = Q(lo);
  for (; lo + 1 < j; ++lo) {
    const double an = A(lo + 1);
    const float qn = Q(lo + 1);
    if (line_diff(an, qn, am, qm, s, none) >= 0.0) break;
    am = an;
    qm = qn;
  }
  for (; lo - 1 > i; --lo) {
    const double an = A(lo - 1);
    const float qn = Q(lo - 1);
    if (line_diff(an, qn, am, qm, s, none) >= 0.0) break;
    am = an;
    qm = qn;
  }
  m = lo;
  const double left = line_diff(A(lo - 1), Q(lo - 1), am, qm, s, err);
  const double right = line_diff(A(lo + 1), Q(lo + 1), am, qm, s, err);
  return fmin(left, right) > gap + (double)err;
}

// Whether the ends of the ray are clear of the first and the last boundary.
__device__ __forceinline__ bool list_ends_clear(const WalkRec* rec, int n, double len,
                                                double gap) {
  const WalkRec a = rec[0], b = rec[1], c = rec[n - 1], d = rec[n];
  float e0 = 0.f, e1 = 0.f;
  return line_diff(b.a, b.q, a.a, a.q, 0.0, e0) > gap + (double)e0 &&
         line_diff(c.a, c.q, d.a, d.q, len, e1) > gap + (double)e1;
}

// Whether the reference's walk over the cells rec[0..n], whose boundaries are all
// certified, inserts and accepts exactly them: every split point it visits has to
// fall on one cell clear of its neighbours (see the head of this file).  `gap`
// bounds the difference of squared distances that counts as clear, `room` the
// pending points; `depth` receives the most there were.
__device__ __forceinline__ bool list_replay(const WalkRec* rec, int n, double gap, int room,
                                         int& depth) {
  int stack[kBatchStack];
  int i = 0, j = n, sp = 0;
  depth = 1;
  for (;;) {
    if (j == i + 1) {  // accepted
      if (sp == 0) return true;
      i = j;
      j = stack[--sp];
      continue;
    }
    const double s = line_cross(rec[i].a, rec[i].q, rec[j].a, rec[j].q);
    int m;
    if (!list_nearest([&](int k) { return rec[k].a; }, [&](int k) { return rec[k].q; }, i, j, s,
                      gap, m) ||
        sp + 1 >= room)
      return false;
    stack[sp++] = j;
    depth = max(depth, sp + 1);
    j = m;
  }
}

template <int MODE, int NF, int OUT>
__global__ void __launch_bounds__(kListBlock, VT_LIST_MINB) k_list(DevCloud c, WalkIO io) {
  constexpr bool kImage = OUT == kOutImage || OUT == kOutCount || OUT == kOutTape;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  // (lanes past io.batch have no ray and no records)
  const unsigned warp = blockIdx.x * (kListBlock / 32) + (threadIdx.x >> 5);
  WalkRec* rec = io.rec + (warp * io.batch + lane) * io.rec_cap;
  const Fetch64 f64{nullptr, c.nodes, 0};
  const Fetch32 f32{nullptr, c.nodes32, 0};
  unsigned n_rays = 0, n_cross = 0, n_q = 0, n_res = 0, max_sp = 0;
  unsigned n_visit = 0, n_ver = 0, n_qver = 0;  // (not reported by this kernel)

  for (;;) {
    // ---- the warp's next rays (neighbours in the coherent order)
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&io.stats->next_ray, (unsigned long long)io.batch);
    base = __shfl_sync(FULL, base, 0);
    if ((int64_t)base >= io.nrays) break;
    const int64_t slot = (int64_t)base + lane;
    int64_t ray = -1;
    bool live = lane < io.batch && slot < io.nrays;
    int asks = 0;  // tree queries of this ray but for its ends'
    RayGeom g = {};
    double qm = 0.0;  // bounds the magnitude of all coordinates of the walk
    double q_err = 0.0;  // FP32 error of its queries' coordinates
    if (live) {
      ray = io.order ? (int64_t)io.order[slot] : slot;
      ray_init(g, io.starts + 3 * ray, io.ends + 3 * ray);
      if (!ray_finite(g)) {
        report(io, ray, kErrNonFinite);
        live = false;
      } else {
        ++n_rays;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          qm = fmax(qm, fmax(fabs(g.s[k]), fabs(g.e[k])));
          qm = fmax(qm, fmax(fabs(c.bblo[k]), fabs(c.bbhi[k])));
          q_err = fmax(q_err, fmax(fabs(g.s[k] - c.origin[k]), fabs(g.e[k] - c.origin[k])));
        }
        q_err = q_err * 6.0e-8 + (double)c.coord_err;
      }
    }

    // a ray that degenerate split points, overflow or too many queries keep from the
    // list is walked again by the tree kernels, which skip what is emitted
    auto give_up = [&](unsigned emitted) {
      leave(io, ray, emitted);
      --n_rays;
      live = false;
    };

    // ---- end cells and march.  A lane whose next step follows from its list
    // goes on; the others' queries run together once VT_LIST_WAIT or fewer lanes
    // march for each of them.
    int phase = live ? 1 : 4;  // 1, 2: the ends' queries; 3: march; 4: through
    int c0 = -1;
    March m = {};
    {
      int cur = -1;
      float r_ask = 0.f;
      bool on = false;
      while (__any_sync(FULL, phase < 4)) {
        const bool turn = phase < 4 && !on;
        bool query = turn;
        double x = 0.0, y = 0.0, z = 0.0, R = pinf(), dc = 0.0, dn = 0.0;
        if (turn && phase < 3) {
          x = phase == 1 ? g.s[0] : g.e[0];
          y = phase == 1 ? g.s[1] : g.e[1];
          z = phase == 1 ? g.s[2] : g.e[2];
        } else if (turn) {
          // the boundary point between the march's cell and its candidate; the
          // generators nearer than its two cells' distance plus the gap decide
          const double4 pc = ldg_pt(&c.pts[cur]);
          double ac, qc, an, qn, tb, off[3];
          foot(g, pc, ac, qc, off);
          double4 pn;
          bool in;
          for (int k = 0;; ++k) {
            pn = ldg_pt(&c.pts[m.nxt]);
            foot(g, pn, an, qn, off);
            tb = 0.5 * ((an + ac) + (qn - qc) / (an - ac));
            in = an > ac && tb <= g.len;
            if (in || k || m.nxt == m.c1) break;
            m.nxt = m.c1;  // the list's best lies past the end: towards the last cell
          }
          if (in) {
            ray_point(g, tb, x, y, z);
            dc = metric(x, y, z, pc);
            dn = metric(x, y, z, pn);
            R = fmax(dc, dn);
            r_ask = 2.f * sqrtf((float)R);
            R += 4e-9 + 4e-14 * qm * (double)r_ask;
          } else {  // no such boundary: c1 ends the sequence, not certified
            float w[3];
            list_settle(c, g, rec, m, cur, m.i, m.clean, w);
            ++m.i;
            list_settle(c, g, rec, m, m.c1, m.i, false, w);
            phase = 4;
            query = false;
          }
        }
        // a ray that asks twice a cell is as well off on the tree
        if (query && phase == 3 && ++asks > kListAsks + 2 * m.i) {
          give_up(0u);
          phase = 4;
          query = false;
        }
        __syncwarp();
        KnnList<3> r;
        r.clear();
        if (query) {
          ++n_q;
          if (phase < 3) knn64_fetch(c, f64, x, y, z, R, r, n_visit);
          else
            knn3_guarded(c, f32, x, y, z, cur, m.nxt, dc, dn, R, guard_band(R, q_err), r, n_visit,
                         n_ver, n_qver);
        }
        __syncwarp();
        if (query && r.id[0] < 0) {
          // squared distances overflow: in FP64 an error, in the guarded FP32 of
          // the march not yet one
          if (phase < 3) report(io, ray, kErrNonFiniteDist);
          else give_up(0u);
          live = false;
          phase = 4;
        } else if (query && phase < 3) {
          if (r.id[1] >= 0 && r.r2[1] == r.r2[0]) {
            hand_over(io, ray, 0u);  // exactly tied nearest cells
            live = false;
            phase = 4;
          } else if (phase == 1) {
            cur = c0 = r.id[0];
            phase = 2;
          } else {
            m.c1 = r.id[0];
            m.nxt = m.prev = -1;
            m.all = true;
            const double4 P = ldg_pt(&c.pts[cur]);
            m.wx = (float)(g.s[0] - P.x);
            m.wy = (float)(g.s[1] - P.y);
            m.wz = (float)(g.s[2] - P.z);
            phase = m.c1 == cur ? 4 : 3;
          }
        } else if (query) {
          const double4 pc = ldg_pt(&c.pts[cur]), pn = ldg_pt(&c.pts[m.nxt]);
          const bool own = r.id[0] == cur || r.id[0] == m.nxt;
          if (!own && r.r2[0] < fmin(dc, dn) && ++m.tries < kListTries) {
            m.nxt = r.id[0];  // a nearer cell lies between
          } else {
            float w[3];
            list_settle(c, g, rec, m, cur, m.i, m.clean, w);
            m.prev = -1;
            m.clean = own && (r.id[1] == cur || r.id[1] == m.nxt) && r.id[2] < 0;
            m.rho_chain = r_ask;
            m.rho_in = 0.f;
            m.rho_max = fmaxf(m.rho_max, r_ask);
            m.wx = (float)(x - pn.x);
            m.wy = (float)(y - pn.y);
            m.wz = (float)(z - pn.z);
            m.den = (float)fma(pn.z - pc.z, g.d[2],
                               fma(pn.y - pc.y, g.d[1], (pn.x - pc.x) * g.d[0]));
            cur = m.nxt;
            ++m.i;
            m.nxt = -1;
          }
        }
        if (turn) on = phase == 3 && m.nxt < 0;
        for (;;) {
          const unsigned go = __ballot_sync(FULL, on);
          const unsigned wait = __ballot_sync(FULL, phase < 4 && !on);
          if (__popc(go) <= VT_LIST_WAIT * __popc(wait)) break;
          if (on) {
            const int k = list_step(c, g, qm, rec, io.rec_cap, m, cur);
            on = k == kMarchOn;
            if (k == kMarchDone) phase = 4;
          }
        }
      }
    }

    // ---- reduction.  Rays whose walk is the marched sequence are reduced from it
    const int nrec = m.i;
    const bool one = live && m.c1 == c0;  // both ends in one cell
    const double gap = 4e-9 + 4e-14 * qm * (double)m.rho_max;
    bool whole = one;
    {
      const int room = io.local_cap < kBatchStack ? io.local_cap : kBatchStack;
      const bool may = live && !one && m.all && 2 * (int64_t)nrec <= io.max_iter &&
                       list_ends_clear(rec, nrec, g.len, gap);
      int depth = 0;
      if (may) whole = list_replay(rec, nrec, gap, room, depth);
      __syncwarp();
      if (whole) max_sp = max(max_sp, (unsigned)depth);
    }
    std::conditional_t<OUT == kOutTape, TapeReducer<MODE, NF, true>, Reducer<MODE, NF>> red = {};
    FillSink fill = {};
    AdjSink<MODE, NF> adj = {};
    auto nseg_of = [&]() -> unsigned {
      if (kImage) return red.nseg;
      if (OUT == kOutFill) return fill.nseg;
      return adj.nseg;
    };
    auto emit = [&](int cell, double a, double b) {
      if (kImage) red.seg(cell, a, b);
      else if (OUT == kOutFill) fill.seg(cell, a, b);
      else adj.seg(cell, a, b);
    };
    auto finish_ok = [&]() {
      if (kImage) {
        red.write(io.out + ray * io.nout);
        if (OUT == kOutCount) io.counts[ray] = red.nseg;
      }
      n_cross += nseg_of();
      live = false;
    };
    auto fail = [&](int rc) {
      if (rc == kNeedSlow || rc == kNeedTie) hand_over(io, ray, nseg_of());
      else report(io, ray, rc);
      live = false;
    };
    if (live) {
      if (kImage) red.init(&c, io.out + ray * io.nout);
      if constexpr (OUT == kOutTape) red.set_tape(&io, ray, 0u);
      if constexpr (OUT == kOutFill) fill.init(&c, io, ray);
      if constexpr (OUT == kOutAdj) adj.init(&c, io, ray, 0u);
    }
    {
      int cell = c0, k = one ? 0 : 1;
      double enter = 0.0;
      double4 pc = make_double4(0.0, 0.0, 0.0, 0.0);
      if (whole) pc = ldg_pt(&c.pts[cell]);
      while (__any_sync(FULL, whole)) {
        if (whole) {
          if (!one) {
            const int to = rec[k].cell;
            const double4 pn = ldg_pt(&c.pts[to]);
            const double s = split_analytic(g, pc, pn);
            emit(cell, enter, s);
            cell = to;
            enter = s;
            pc = pn;
          }
          if (one || k == nrec) {
            emit(cell, enter, g.len);
            finish_ok();
            whole = false;
          }
          ++k;
        }
        if constexpr (OUT == kOutTape) red.flush_tape(io);
      }
    }

    // ---- the other rays: the reference's walk, with the records as hints
    if (__any_sync(FULL, live)) {
      LocalStack<kBatchStack> st;
      int st_li[kBatchStack];  // list index of each pending point (-1: not in it)
      st.set_cap(io.local_cap);
      st.clear();
      int cur = c0, nxt = -1, open_cell = c0, ci = 0, ni = 0;
      double cur_s = 0.0, nxt_s = 0.0, entry_s = 0.0, s = 0.0;
      int64_t iter = 0;
      double4 pc = make_double4(0.0, 0.0, 0.0, 0.0), pn = pc;
      if (live) {
        st_li[0] = nrec;
        st.push(m.c1, g.len);
        pc = ldg_pt(&c.pts[cur]);
      }
      auto accept = [&]() {
        emit(open_cell, entry_s, s);
        open_cell = nxt;
        entry_s = s;
        st.pop();
        cur = nxt;
        ci = ni;
        cur_s = nxt_s;
        pc = pn;
        if (st.empty()) {
          emit(open_cell, entry_s, cur_s);
          finish_ok();
        }
      };
      // Degenerate split points (parallel bisectors, more than two cells at one
      // distance) take the functions of the tree kernels, one lane at a time.  A few
      // of the rays through a dense core meet one; where several lanes do, the cloud
      // is a lattice or the like and the rays are left to the tree kernels.
      int rares = 0;
      auto one_by_one = [&](bool want, auto call) {
        const int together = __popc(__ballot_sync(FULL, want));
        if (want && (together > kListRareLanes || ++rares > kListRare)) {
          give_up(nseg_of());
          want = false;
        }
        for (unsigned w = __ballot_sync(FULL, want); w; w &= w - 1) {
          if (lane == __ffs(w) - 1) call();
          __syncwarp();
        }
      };
      auto next_point = [&]() {
        nxt = st.top_id();
        nxt_s = st.top_s();
        ni = st_li[st.sp - 1];
        pn = ldg_pt(&c.pts[nxt]);
      };
      // an iteration without a query; false when it needs one or the ray is done
      auto hinted = [&]() -> bool {
        next_point();
        s = split_analytic(g, pc, pn);
        // parallel bisectors, skips, bounds and clamps go the long way
        if (!(ci >= 0 && ni > ci && iter < io.max_iter && s < DBL_MAX * 0.5 &&
              s >= dadd(cur_s, 1e-15) && s <= dsub(nxt_s, 1e-15)) ||
            dsub(nxt_s, cur_s) < 1e-14)
          return false;
        if (ni == ci + 1) {
          if (signbit(rec[ni].q)) return false;
          ++iter;
          accept();
          return live;
        }
        int k;
        if (!list_nearest([&](int e) { return rec[e].a; }, [&](int e) { return rec[e].q; }, ci, ni,
                          s, gap, k))
          return false;
        const WalkRec a = rec[k];
        if (a.cell == cur || a.cell == nxt || signbit(a.q) || signbit(rec[k + 1].q) ||
            st.room() < 1)
          return false;
        ++iter;
        st_li[st.sp] = k;
        st.push(a.cell, s);
        return true;
      };
      bool on = live;
      while (__any_sync(FULL, live)) {
        // ---- iterations without a query, until half of the lanes need one
        for (;;) {
          const unsigned go = __ballot_sync(FULL, on), wait = __ballot_sync(FULL, live && !on);
          if (__popc(go) <= __popc(wait)) break;
          if (on) on = hinted();
          if constexpr (OUT == kOutTape) red.flush_tape(io);
        }
        // ---- one iteration with a query for each of the waiting lanes
        const bool turn = live && !on;
        bool query = false, rare = false;
        if (turn) {
          next_point();
          if (++iter > io.max_iter) {
            fail(kErrMaxIter);
          } else if (dsub(nxt_s, cur_s) < 1e-14) {  // zero-width skip
            st.pop();
            cur = nxt;
            ci = ni;
            cur_s = nxt_s;
            open_cell = cur;
            pc = pn;
            if (st.empty()) {
              emit(open_cell, entry_s, cur_s);
              finish_ok();
            }
          } else {
            s = split_analytic(g, pc, pn);
            query = ++asks <= kListAsks + 2 * nrec;
            rare = query && !(s < DBL_MAX * 0.5 && s >= cur_s - kTol && s <= nxt_s + kTol);
            if (!query) give_up(nseg_of());
          }
        }
        one_by_one(rare, [&] {  // parallel bisectors
          const RareOut ro = rare_split(c, g, cur, nxt, cur_s, nxt_s);
          n_q += ro.nq;
          s = ro.s;
          if (ro.rc) fail(ro.rc);
          else if (s < dsub(cur_s, kTol) || s > dadd(nxt_s, kTol)) fail(kErrSplitBounds);
        });
        query = query && live;
        double x = 0.0, y = 0.0, z = 0.0, R = 0.0;
        KnnList<3> r;
        r.clear();
        if (query) {
          const double lo = dadd(cur_s, 1e-15), hi = dsub(nxt_s, 1e-15);
          s = (s < lo) ? lo : (hi < s) ? hi : s;
          ray_point(g, s, x, y, z);
          R = dadd(fmax(metric(x, y, z, pc), metric(x, y, z, pn)), 4.0 * kTol);
          ++n_q;
          // the bounded search, and the unbounded one where it cannot decide
          for (int k = 0; k < 2; ++k) {
            knn64_fetch(c, f64, x, y, z, R, r, n_visit);
            if (k || knn3_decision_valid(r, R)) break;
            ++n_res;
            r.clear();
            R = pinf();
          }
        }
        __syncwarp();
        if (query && r.id[0] < 0) fail(kErrNonFiniteDist);
        // ---- what the 3-NN of a split point decides
        bool has_c = false, has_n = false, three_eq = true;
#pragma unroll
        for (int k = 0; k < 3; k++) {
          if (dsub(r.r2[k], r.r2[0]) >= kTol) {
            three_eq = false;
            break;
          }
          if (r.id[k] == cur) has_c = true;
          if (r.id[k] == nxt) has_n = true;
        }
        one_by_one(query && live && three_eq && !has_c && !has_n, [&] {  // 100-NN
          const RareOut ro = rare_expand(c, x, y, z, cur, nxt);
          n_q += ro.nq;
          if (ro.rc) fail(ro.rc);
          has_c = ro.a;
          has_n = ro.b;
        });
        int sc = r.id[0], sn = r.id[0];
        const bool insert = query && live && !has_c && !has_n;
        one_by_one(insert && !(dadd(r.r2[0], kTol) < r.r2[1]), [&] {  // cells on both sides
          const RareOut ro = rare_case1a(c, g, x, y, z, cur, nxt);
          n_q += ro.nq;
          sc = ro.a;
          sn = ro.b;
          if (ro.rc) fail(ro.rc);
        });
        if (query && live) {
          if (has_c || has_n) {
            accept();
          } else if (st.room() < (sc == sn ? 1 : 2)) {
            fail(kNeedSlow);
          } else {
            // back on the list when the pushed cell is the recorded one
            int k0 = 0;
            for (int hi = nrec; k0 < hi;) {  // the last foot up to s
              const int mid = (k0 + hi + 1) >> 1;
              if (rec[mid].a <= s) k0 = mid;
              else hi = mid - 1;
            }
            auto push = [&](int id) {
              int li = -1;
              for (int k = max(k0 - 2, 0); k <= min(k0 + 2, nrec); ++k)
                if (rec[k].cell == id) li = k;
              st_li[st.sp] = li;
              st.push(id, s);
            };
            if (sc != sn) push(sn);
            push(sc);
          }
        }
        if (turn) on = live;
        if constexpr (OUT == kOutTape) red.flush_tape(io);
        if (turn) max_sp = max(max_sp, (unsigned)st.maxsp);
      }
    }
  }
  warp_add(&io.stats->rays, n_rays);
  warp_add(&io.stats->crossings, n_cross);
  warp_add(&io.stats->queries, n_q);
  warp_add(&io.stats->fp64_resolves, n_res);
  warp_max(&io.stats->max_stack, max_sp);
}

// Blocks of a launch over nrays rays on nsms SMs, and the rays that a warp takes at
// a time: few rays are spread over all resident warps.
inline int64_t list_blocks(int64_t nrays, int nsms) {
  const int64_t blocks = (int64_t)nsms * VT_LIST_MINB;
  const int64_t need = (nrays + kListBlock / 32 - 1) / (kListBlock / 32);
  return need < blocks ? (need > 0 ? need : 1) : blocks;
}
inline int list_batch(int64_t nrays, int nsms) {
  const int64_t warps = list_blocks(nrays, nsms) * (kListBlock / 32);
  const int64_t per = (nrays + warps - 1) / warps;
  return (int)(per < 32 ? (per < 1 ? 1 : per) : 32);
}

template <int MODE, int NF, int OUT>
int launch_list(vt_cloud* cl, WalkIO& io, cudaStream_t st) {
  int dev = 0, nsms = 0;
  VT_CUDA(cudaGetDevice(&dev));
  VT_CUDA(cudaDeviceGetAttribute(&nsms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t blocks = list_blocks(io.nrays, nsms);
  k_list<MODE, NF, OUT><<<(unsigned)blocks, kListBlock, 0, st>>>(cl->view, io);
  return VT_OK;
}

}  // namespace vt
