// nbrlist.cu -- neighbour lists of a built cloud, for the list walk
// (listed.cuh).
//
// The list of a point p holds the vectors v = q - p to its nearest points q
// (FP32, rounded from the FP64 difference) in two parts, those with vz > 0 and
// the others, each in order of distance, in groups of four: {vx[4], vy[4],
// vz[4], tree index[4]}, one 64-byte block (two sectors) per group, kNbrGroups
// blocks reserved per point, the first part in the blocks 0, 1, ... and the
// second in the last block, the one before it, ....  (A ray along +z or -z, as of an unrotated pixel
// grid, can only leave towards one of the parts.)  Its header is a float, half
// the squared radius rho inside which the list is complete (every point nearer
// than rho is listed), its low 10 bits replaced by the number of groups of the
// two parts, 5 bits each (0: no list).  A walk that leaves p's cell at distance
// r from p needs the points nearer than 2 r only, so it reads the groups in
// order and stops there: 13 points on average in a homogeneous cloud (the ball
// through a random point of a cell's surface holds 5/3 points, the ball of twice
// the radius eight times as many), and 60 points cover 99.7% of the exits.
//
// One warp per leaf: it gathers the tree's points within a radius of the
// leaf's box (the radius from the density of an ancestor of 32 to 63 points),
// 32 nodes five levels down per step, keeps their coordinates relative to
// the leaf's first point in shared memory as FP32, and each of the leaf's points
// selects its own from them and sorts them by their squared distance from the FP64
// coordinates (128-element bitonic sort, four elements per lane).
//
// Why every point nearer than rho is listed.  u = 2^-24; S is the largest
// gathered coordinate vector relative to the leaf's first point.  The FP32 vector
// from the point to a gathered one differs from the true one by the rounding of
// both (u S each at most) and of their difference (u d): its length is off by 2 u S
// + 3 u d at most, sum of squares included, and the selection's radius re = ri + e
// by 3 u re, so that e = 6 u (S + ri) lets all points at d <= ri in.  Of these,
// 60 are kept in the order of the FP64 distance rounded to FP32 (u) without its 10
// lowest bits (1.3e-4 of d^2), and rho is the first one left out, or ri, less
// 1e-4 of rho^2 for the roundings.  A leaf can be as wide as the gaps between
// compact groups, so that S / ri has no bound: with e in the place of a fixed
// share of rho the radius stays true, and a point whose e is not small against
// the distances selects too many and gets no list.
#include "common.cuh"
#include "internal.h"

namespace vt {

constexpr int kNbrWarps = 2;      // warps per block
constexpr int kNbrCand = 768;     // gathered points per leaf (at most 1024)
constexpr int kNbrKeys = 128;     // points sorted per list
constexpr int kNbrStack = 192;    // pending nodes per warp
constexpr int kNbrSteps = 2048;   // node expansions per leaf (a dozen in practice)
constexpr int kNbrTarget = 80;    // points aimed at inside the gather radius
constexpr unsigned kAll = 0xffffffffu;

struct NbrScratch {
  float x[kNbrCand], y[kNbrCand], z[kNbrCand];
  int id[kNbrCand];
  int stack[kNbrStack];
  unsigned key[kNbrKeys];
};

// Gather into S the points within r of the box [lo, hi] (FP32 frame); -1 when
// they do not fit.
__device__ __forceinline__ int gather_near(const DevCloud& c, NbrScratch& S, int lane, float4 lo,
                                           float4 hi, float r, double px, double py, double pz) {
  const int D = c.depth;
  const int ninternal = (int)(c.nleaves - 1);
  // the FP32 copies are off by at most coord_err per component: every point
  // within r of the leaf's points passes this radius on the copies
  const float rr = r * 1.00002f + 4.f * c.coord_err;
  const float r2 = rr * rr;
  int count = 0, sp = 0;
  int s = D == 0 ? 0 : ((D - 1) % 5) + 1;
  int level = s;
  int first = (1 << s) - 1, gm = 1 << s;
  for (int steps = 0; steps < kNbrSteps; ++steps) {
    const int node = first + lane;
    bool in = false;
    if (lane < gm) {
      const float4 l = __ldg(&c.boxlo[node]), h = __ldg(&c.boxhi[node]);
      const float gx = fmaxf(0.f, fmaxf(l.x - hi.x, lo.x - h.x));
      const float gy = fmaxf(0.f, fmaxf(l.y - hi.y, lo.y - h.y));
      const float gz = fmaxf(0.f, fmaxf(l.z - hi.z, lo.z - h.z));
      in = gx * gx + gy * gy + gz * gz <= r2;
    }
    const unsigned mask = __ballot_sync(kAll, in);
    if (level == D) {
      // four leaves at a time: eight lanes look at the points of one leaf
      for (unsigned m = mask; m;) {
        int leaf = -1;
        for (int k = 0; k < 4; ++k) {
          const int b = m ? __ffs(m) - 1 : -1;
          if (m) m &= m - 1;
          if ((lane >> 3) == k && b >= 0) leaf = first + b - ninternal;
        }
        bool ok = false;
        int p = 0;
        if (leaf >= 0) {
          int64_t a, b;
          leaf_range(c, leaf, a, b);
          p = (int)a + (lane & 7);
          if (p < (int)b) {
            const float4 q = __ldg(&c.pts32[p]);
            const float gx = fmaxf(0.f, fmaxf(q.x - hi.x, lo.x - q.x));
            const float gy = fmaxf(0.f, fmaxf(q.y - hi.y, lo.y - q.y));
            const float gz = fmaxf(0.f, fmaxf(q.z - hi.z, lo.z - q.z));
            ok = gx * gx + gy * gy + gz * gz <= r2;
          }
        }
        const unsigned om = __ballot_sync(kAll, ok);
        if (count + __popc(om) > kNbrCand) return -1;
        if (ok) {
          const int at = count + __popc(om & ((1u << lane) - 1u));
          const double4 P = ldg_pt(&c.pts[p]);
          S.x[at] = __double2float_rn(P.x - px);
          S.y[at] = __double2float_rn(P.y - py);
          S.z[at] = __double2float_rn(P.z - pz);
          S.id[at] = p;
        }
        count += __popc(om);
      }
    } else {
      if (sp + __popc(mask) > kNbrStack) return -1;
      if (in) S.stack[sp + __popc(mask & ((1u << lane) - 1u))] = node;
      sp += __popc(mask);
      __syncwarp();
    }
    if (sp == 0) {
      __syncwarp();
      return count;
    }
    const int v = S.stack[--sp];
    __syncwarp();
    const int k = 31 - __clz(v + 1);
    s = min(5, D - k);
    level = k + s;
    first = ((v + 1) << s) - 1;
    gm = 1 << s;
  }
  return -1;
}

// Ascending bitonic sort of 128 keys, element lane + 32 h in v[h].
__device__ __forceinline__ void sort128(unsigned (&v)[4], int lane) {
#pragma unroll
  for (int k = 2; k <= 128; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int p = h ^ (j >> 5);
          if (p > h) {
            const bool up = ((32 * h) & k) == 0;
            const unsigned a = min(v[h], v[p]), b = max(v[h], v[p]);
            v[h] = up ? a : b;
            v[p] = up ? b : a;
          }
        }
      } else {
        const bool low = (lane & j) == 0;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const unsigned p = __shfl_xor_sync(kAll, v[h], j);
          const bool up = ((lane + 32 * h) & k) == 0;
          v[h] = low == up ? min(v[h], p) : max(v[h], p);
        }
      }
    }
  }
}

__global__ void __launch_bounds__(kNbrWarps * 32)
    k_nbr_lists(DevCloud c, float* __restrict__ nbr, uint32_t* __restrict__ hdr) {
  __shared__ NbrScratch s_all[kNbrWarps];
  const int lane = threadIdx.x & 31;
  NbrScratch& S = s_all[threadIdx.x >> 5];
  const int64_t leaf = (int64_t)blockIdx.x * kNbrWarps + (threadIdx.x >> 5);
  if (leaf >= c.nleaves) return;
  int64_t a, b;
  leaf_range(c, leaf, a, b);
  const int ninternal = (int)(c.nleaves - 1);
  const float4 lo = __ldg(&c.boxlo[ninternal + leaf]), hi = __ldg(&c.boxhi[ninternal + leaf]);
  // radius that holds about kNbrTarget points at the density of the smallest
  // ancestor of at least 32 points
  int up = 0;
  while (up < c.depth && (c.n >> (c.depth - up)) < 32) ++up;
  const int anc = (int)((ninternal + leaf + 1) >> up) - 1;
  const float cnt = (float)(c.n >> (c.depth - up));
  const float4 al = __ldg(&c.boxlo[anc]), ah = __ldg(&c.boxhi[anc]);
  const float ex = ah.x - al.x, ey = ah.y - al.y, ez = ah.z - al.z;
  float r = cbrtf(ex) * cbrtf(ey) * cbrtf(ez) * cbrtf((float)kNbrTarget / 4.18879f / cnt);
  if (!(r > 0.02f * fmaxf(ex, fmaxf(ey, ez)))) r = 0.5f * fmaxf(ex, fmaxf(ey, ez));
  const double4 P0 = ldg_pt(&c.pts[a]);
  float s_max = 0.f;  // largest gathered coordinate vector
  int m = -1;
  if (r > 0.f && r < 1e15f) {
    for (int t = 0; t < 12 && m < 0; ++t) {
      m = gather_near(c, S, lane, lo, hi, r, P0.x, P0.y, P0.z);
      __syncwarp();
      if (m < 0) r *= 0.75f;
    }
    for (int j = lane; j < m; j += 32)
      s_max = fmaxf(s_max, S.x[j] * S.x[j] + S.y[j] * S.y[j] + S.z[j] * S.z[j]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s_max = fmaxf(s_max, __shfl_xor_sync(kAll, s_max, o));
    s_max = sqrtf(s_max);
  }
  for (int64_t i = a; i < b; ++i) {
    const double4 P = ldg_pt(&c.pts[i]);
    const float x = __double2float_rn(P.x - P0.x), y = __double2float_rn(P.y - P0.y),
                z = __double2float_rn(P.z - P0.z);
    // the points nearer than ri (at most kNbrKeys: a smaller ri when there are
    // more), by their FP32 distance, which is off by less than e
    float ri2 = r * r;
    int k = 0;
    bool fits = false;
    for (int t = 0; t < 8 && m > 0 && !fits; ++t) {
      k = 0;
      const float ri = sqrtf(ri2), re = ri + 3.6e-7f * (s_max + ri);
      for (int j0 = 0; j0 < m; j0 += 32) {
        const int j = j0 + lane;
        bool in = false;
        if (j < m && S.id[j] != (int)i) {
          const float dx = S.x[j] - x, dy = S.y[j] - y, dz = S.z[j] - z;
          in = dx * dx + dy * dy + dz * dz <= re * re;
        }
        const unsigned im = __ballot_sync(kAll, in);
        const int at = k + __popc(im & ((1u << lane) - 1u));
        if (in && at < kNbrKeys) S.key[at] = (unsigned)j;
        k += __popc(im);
      }
      __syncwarp();
      fits = k <= kNbrKeys;
      if (!fits) ri2 *= fminf(0.9f, powf((float)kNbrTarget / (float)k, 0.6666667f));
    }
    int g_up = 0, g_down = 0;
    float half_rho2 = 0.f;
    if (fits && k > 0) {
      unsigned v[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        // key: the squared distance with its 10 lowest mantissa bits replaced
        // by the gathered slot
        v[h] = kAll;
        if (lane + 32 * h < k) {
          const unsigned j = S.key[lane + 32 * h];
          const double4 Q = ldg_pt(&c.pts[S.id[j]]);
          const double dx = dsub(Q.x, P.x), dy = dsub(Q.y, P.y), dz = dsub(Q.z, P.z);
          v[h] = (__float_as_uint(__double2float_rn(dx * dx + dy * dy + dz * dz)) & ~1023u) | j;
        }
      }
      sort128(v, lane);
      const int kept = min(k, kNbrMax);
      // complete up to the first point left out, or up to ri
      const unsigned next = __shfl_sync(kAll, v[kNbrMax >> 5], kNbrMax & 31);
      const float rho2 = k > kNbrMax ? fminf(__uint_as_float(next & ~1023u), ri2) : ri2;
      half_rho2 = 0.5f * rho2 * 0.9999f;
      // the two parts: ranks of this lane's points in theirs
      float vx[2], vy[2], vz[2];
      int id[2], at[2], n_up = 0, n_down = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const bool in = lane + 32 * h < kept;
        id[h] = -1;
        vx[h] = vy[h] = vz[h] = 0.f;
        if (in) {
          id[h] = S.id[v[h] & 1023u];
          const double4 Q = ldg_pt(&c.pts[id[h]]);
          vx[h] = __double2float_rn(dsub(Q.x, P.x));
          vy[h] = __double2float_rn(dsub(Q.y, P.y));
          vz[h] = __double2float_rn(dsub(Q.z, P.z));
        }
        const unsigned um = __ballot_sync(kAll, in && vz[h] > 0.f);
        const unsigned dm = __ballot_sync(kAll, in && !(vz[h] > 0.f));
        const unsigned below = (1u << lane) - 1u;
        at[h] = vz[h] > 0.f ? n_up + __popc(um & below) : n_down + __popc(dm & below);
        n_up += __popc(um);
        n_down += __popc(dm);
      }
      g_up = (n_up + 3) >> 2;
      g_down = (n_down + 3) >> 2;
      float* out = nbr + (int64_t)i * (kNbrGroups * 16);
      auto put = [&](bool up, int e, float x, float y, float z, int p) {
        const int grp = up ? e >> 2 : kNbrGroups - 1 - (e >> 2);
        float* o = out + grp * 16 + (e & 3);
        o[0] = x;
        o[4] = y;
        o[8] = z;
        o[12] = __int_as_float(p);
      };
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (id[h] >= 0) put(vz[h] > 0.f, at[h], vx[h], vy[h], vz[h], id[h]);
      // past a part's end: a point too far away to matter
      if (lane < 4 * g_up - n_up) put(true, n_up + lane, 1e17f, 1e17f, 1e17f, -1);
      if (lane < 4 * g_down - n_down) put(false, n_down + lane, 1e17f, 1e17f, -1e17f, -1);
    }
    if (lane == 0)
      hdr[i] = g_up + g_down ? (__float_as_uint(half_rho2) & ~1023u) |
                                   (unsigned)(g_up << 5) | (unsigned)g_down
                             : 0u;
    __syncwarp();
  }
}

// Sums over every `step`-th point and 32 directions u: sum[0] of s^2, s the extent of
// the point's cell along u as its list has it (no farther than the cloud's box), the
// weight with which rays meet this part of the cell; sum[1] of the s^2 whose end the
// list does not vouch for (2 s > rho).  One warp per point, a direction per lane.
__global__ void __launch_bounds__(128)
    k_nbr_open(DevCloud c, int64_t step, double* __restrict__ sum) {
  const int lane = threadIdx.x & 31;
  const int64_t i = ((int64_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * step;
  if (i >= c.n) return;
  const unsigned hdr = __ldg(&c.nbr_hdr[i]);
  if (hdr == 0) return;
  // a spiral of directions: equal steps in z, the golden angle around it
  const float uz = 1.f - (float)(2 * lane + 1) / 32.f, ur = sqrtf(1.f - uz * uz);
  float ux, uy;
  sincosf(2.39996323f * (float)lane, &uy, &ux);
  ux *= ur;
  uy *= ur;
  const double4 P = ldg_pt(&c.pts[i]);
  auto side = [&](int d, double p, float u) {
    return u == 0.f ? __int_as_float(0x7f800000)
                    : (float)(((u > 0.f ? c.bbhi[d] : c.bblo[d]) - p) / (double)u);
  };
  float s = fminf(side(0, P.x, ux), fminf(side(1, P.y, uy), side(2, P.z, uz)));
  const float* list = reinterpret_cast<const float*>(c.nbr) + i * (kNbrGroups * 16);
  const int n_up = 4 * (int)((hdr >> 5) & 31u), n = n_up + 4 * (int)(hdr & 31u);
  for (int k = 0; k < n; ++k) {
    const int slot = k < n_up ? k : 4 * kNbrGroups - n + k;
    const float* v = list + 16 * (slot >> 2) + (slot & 3);
    const float x = __ldg(v), y = __ldg(v + 4), z = __ldg(v + 8);
    const float den = x * ux + y * uy + z * uz;
    if (den > 0.f) s = fminf(s, 0.5f * (x * x + y * y + z * z) / den);
  }
  const double w = (double)s * (double)s;
  // hdr: rho^2 / 2
  double all = w, open = 2.0 * w > (double)__uint_as_float(hdr & ~1023u) ? w : 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    all += __shfl_xor_sync(kAll, all, o);
    open += __shfl_xor_sync(kAll, open, o);
  }
  if (lane == 0) {
    atomicAdd(&sum[0], all);
    atomicAdd(&sum[1], open);
  }
}

// The share of the cells' surface, as rays meet it, at which the lists cannot tell the
// next cell: AUTO's measure of whether the list walk fits the cloud.  At most
// kNbrOpenPoints of the points are looked at.
constexpr int64_t kNbrOpenPoints = 65536;
static int nbr_open_share(vt_cloud* cl, double& share) {
  DevBuf<double> sum;
  double h[2] = {0.0, 0.0};
  if (sum.alloc(2)) return VT_ERR_NOMEM;
  VT_CUDA(cudaMemsetAsync(sum.p, 0, 2 * sizeof(double), cl->stream));
  const int64_t n = cl->view.n, step = (n + kNbrOpenPoints - 1) / kNbrOpenPoints;
  const int64_t points = (n + step - 1) / step;
  k_nbr_open<<<(unsigned)((points + 3) / 4), 128, 0, cl->stream>>>(cl->view, step, sum.p);
  VT_CUDA(cudaGetLastError());
  VT_CUDA(cudaMemcpyAsync(h, sum.p, sizeof(h), cudaMemcpyDeviceToHost, cl->stream));
  VT_CUDA(cudaStreamSynchronize(cl->stream));
  share = h[0] > 0.0 ? h[1] / h[0] : 1.0;
  return VT_OK;
}

void drop_nbr_lists(vt_cloud* cl) {
  cl->nbr_d.reset();
  cl->nbr_hdr_d.reset();
  cl->view.nbr = nullptr;
  cl->view.nbr_hdr = nullptr;
  ++cl->list_gen;
}

size_t nbr_list_bytes(const vt_cloud* cl) {
  return (size_t)cl->npart * (kNbrGroups * 4 * sizeof(float4) + sizeof(uint32_t));
}

// Build the lists of a built, non-periodic cloud (no-op when built).  Without
// the memory for them and for `records` bytes of walk records the cloud simply has
// none.
int build_nbr_lists(vt_cloud* cl, size_t records) {
  if (cl->view.nbr) return VT_OK;
  const size_t n = (size_t)cl->npart, count = n * kNbrGroups * 4;
  size_t most = (size_t)cl->list_bytes;
  if (cl->list_bytes < 0) {
    // a quarter of the free memory: a caller that shares the device keeps the rest
    size_t total = 0;
    VT_CUDA(cudaMemGetInfo(&most, &total));
    most /= 4;
  }
  if (nbr_list_bytes(cl) + records > most) return VT_OK;
  if (cl->nbr_d.alloc(count) || cl->nbr_hdr_d.alloc(n)) {
    cudaGetLastError();  // not enough memory after all
    drop_nbr_lists(cl);
    return VT_OK;
  }
  const unsigned blocks = (unsigned)((cl->view.nleaves + kNbrWarps - 1) / kNbrWarps);
  k_nbr_lists<<<blocks, kNbrWarps * 32, 0, cl->stream>>>(cl->view, (float*)cl->nbr_d.p,
                                                         cl->nbr_hdr_d.p);
  VT_CUDA(cudaGetLastError());
  cl->view.nbr = cl->nbr_d.p;
  cl->view.nbr_hdr = cl->nbr_hdr_d.p;
  const int rc = nbr_open_share(cl, cl->list_open_share);
  if (rc) drop_nbr_lists(cl);
  if (rc != VT_ERR_NOMEM) return rc;
  cudaGetLastError();
  return VT_OK;
}

}  // namespace vt
