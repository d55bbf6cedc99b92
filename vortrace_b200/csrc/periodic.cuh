// periodic.cuh -- walk kernel for periodic clouds: the exact FP64 walk of walk_ray()
// (src/ray.cpp:187-430) with one query per lane and loop trip.
//
// The per-ray code of k_plain never brings the lanes of a warp together again
// once their rays took different branches (the same-cell sampling at the start of
// every periodic ray): 138 ms for 27,000 rays through 150,000 cells against 20 ms of
// the same rays in the same cloud without periodicity.  Here every kind of query (end cells, same-cell sampling, bisection,
// split points) is a phase of one loop: a trip prepares each lane's query, all lanes
// search the tree together, then the lanes whose query has a periodic image within
// reach search the images, again together, and each lane applies its answer.  Rays
// run in the coherent order, up to 32 neighbours to a warp: 14 ms for the same rays.
// What is left is the FP64 tree search, two per crossing, from the root: 2,900 warp
// instructions per crossing at 3.6 lanes (16,384 rays, 7 to a warp).
#pragma once

namespace vt {

#ifndef VT_PERIODIC_MINB
#define VT_PERIODIC_MINB 4
#endif

// degenerate split points of a ray that are resolved here, and the most lanes of a
// warp that may meet one together (k_plain's own time is that of its longest ray, so
// that a few rays are better kept)
constexpr int kPeriodicRare = 64;
constexpr int kPeriodicRareLanes = 8;

// 100-NN classification and Case 1a on a periodic cloud, not inlined
static __device__ __noinline__ RareOut rare_expand_periodic(const DevCloud& c, double x, double y,
                                                            double z, int cur, int nxt) {
  bool has_c = false, has_n = false;
  unsigned v = 0;
  RareOut o{0.0, 0, 0, 0, 1u};
  o.rc = expand_classify<true>(c, x, y, z, cur, nxt, has_c, has_n, v);
  o.a = has_c;
  o.b = has_n;
  return o;
}
static __device__ __noinline__ RareOut rare_case1a_periodic(const DevCloud& c, RayGeom g, double x,
                                                            double y, double z, int cur,
                                                            int nxt) {
  Search64T<true> S(c);
  return case1a(g, S, x, y, z, cur, nxt);
}

// The minimum image of p about the point `ref` (src/ray.cpp:71-86).
__device__ __forceinline__ double4 min_image(const DevCloud& c, double4 p, const double (&ref)[3]) {
  double v[3] = {p.x, p.y, p.z};
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const double half = dmul(c.box[d], 0.5), diff = dsub(v[d], ref[d]);
    if (diff > half) v[d] = dsub(v[d], c.box[d]);
    else if (diff < -half) v[d] = dadd(v[d], c.box[d]);
  }
  return make_double4(v[0], v[1], v[2], 0.0);
}

// Merge the results `g` of an image into the list `r` (queryTreeK,
// src/pointcloud.cpp:313-367): one entry per particle with its smallest distance,
// sorted ascending (equal distances in the order they came), truncated.
__device__ __forceinline__ void merge_image(KnnList<3>& r, const KnnList<3>& g) {
  double md[6];
  int mi[6];
  int n = 0;
  for (int i = 0; i < 3; ++i)
    if (r.id[i] >= 0) {
      md[n] = r.r2[i];
      mi[n++] = r.id[i];
    }
  for (int i = 0; i < 3; ++i) {
    if (g.id[i] < 0) continue;
    bool found = false;
    for (int k = 0; k < n && !found; ++k)
      if (mi[k] == g.id[i]) {
        md[k] = fmin(md[k], g.r2[i]);
        found = true;
      }
    if (!found) {
      md[n] = g.r2[i];
      mi[n++] = g.id[i];
    }
  }
  for (int a = 1; a < n; a++) {
    const double d = md[a];
    const int id = mi[a];
    int b = a;
    for (; b > 0 && md[b - 1] > d; --b) {
      md[b] = md[b - 1];
      mi[b] = mi[b - 1];
    }
    md[b] = d;
    mi[b] = id;
  }
  r.clear();
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (i < n) {
      r.r2[i] = md[i];
      r.id[i] = mi[i];
    }
}

template <int MODE, int NF, int OUT>
__global__ void __launch_bounds__(128, VT_PERIODIC_MINB) k_periodic(DevCloud c, WalkIO io) {
  constexpr bool kImage = OUT == kOutImage || OUT == kOutCount || OUT == kOutTape;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const Fetch64 f64{nullptr, c.nodes, 0};
  enum { kIdle, kStart, kEnd, kSample, kBisect, kNext, kSplit };
  unsigned n_rays = 0, n_cross = 0, n_q = 0, max_sp = 0, n_visit = 0;

  for (;;) {
    // ---- the warp's next rays (neighbours in the coherent order)
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&io.stats->next_ray, (unsigned long long)io.batch);
    base = __shfl_sync(FULL, base, 0);
    if ((int64_t)base >= io.nrays) break;
    const int64_t slot = (int64_t)base + lane;
    int64_t ray = -1;
    int phase = kIdle;
    RayGeom g = {};
    std::conditional_t<OUT == kOutTape, TapeReducer<MODE, NF, true>, Reducer<MODE, NF>> red = {};
    FillSink fill = {};
    AdjSink<MODE, NF> adj = {};
    LocalStack<kBatchStack> st;
    st.set_cap(io.local_cap);
    st.clear();
    if (lane < io.batch && slot < io.nrays) {
      ray = io.order ? (int64_t)io.order[slot] : slot;
      ray_init(g, io.starts + 3 * ray, io.ends + 3 * ray);
      if (!ray_finite(g)) {
        report(io, ray, kErrNonFinite);
      } else {
        phase = kStart;
        ++n_rays;
        if (kImage) red.init(&c, io.out + ray * io.nout);
        if constexpr (OUT == kOutTape) red.set_tape(&io, ray, 0u);
        if constexpr (OUT == kOutFill) fill.init(&c, io, ray);
        if constexpr (OUT == kOutAdj) adj.init(&c, io, ray, 0u);
      }
    }
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
    int cur = -1, nxt = -1, open_cell = -1, c0 = -1, level = 1, at = 1, tries = 0;
    double cur_s = 0.0, nxt_s = 0.0, entry_s = 0.0, s = 0.0, lo = 0.0, hi = 0.0;
    int64_t iter = 0;
    auto finish_ok = [&]() {
      emit(open_cell, entry_s, cur_s);
      if (kImage) {
        red.write(io.out + ray * io.nout);
        if (OUT == kOutCount) io.counts[ray] = red.nseg;
      }
      n_cross += nseg_of();
      phase = kIdle;
    };
    auto fail = [&](int rc) {
      if (rc == kNeedSlow || rc == kNeedTie) hand_over(io, ray, nseg_of());
      else report(io, ray, rc);
      phase = kIdle;
    };
    // the rare functions search for themselves, one lane at a time; where several lanes
    // want one together (a lattice) or a ray wants many, the rays are walked again by
    // k_plain (30,000 rays along the columns of a 32^3 lattice: 24.6 ms one lane at a
    // time, 7.6 by k_plain alone).  A caller without scratch for the queue
    // (vt_project_device_noalloc) has them done here.
    int rares = 0;
    auto one_by_one = [&](bool want, auto call) {
      const int together = __popc(__ballot_sync(FULL, want));
      if (want && io.redo_q && (together > kPeriodicRareLanes || ++rares > kPeriodicRare)) {
        leave(io, ray, nseg_of());
        --n_rays;
        phase = kIdle;
        want = false;
      }
      for (unsigned w = __ballot_sync(FULL, want); w; w &= w - 1) {
        if (lane == __ffs(w) - 1) call();
        __syncwarp();
      }
    };
    auto use_split = [&]() {  // the split point s is known: clamp it and query there
      if (s < dsub(cur_s, kTol) || s > dadd(nxt_s, kTol)) {
        fail(kErrSplitBounds);
        return;
      }
      const double a = dadd(cur_s, 1e-15), b = dsub(nxt_s, 1e-15);
      s = (s < a) ? a : (b < s) ? b : s;
      phase = kSplit;
    };

    while (__any_sync(FULL, phase != kIdle)) {
      // ---- prepare this lane's query
      if (phase == kNext) {
        for (;;) {
          if (++iter > io.max_iter) {
            fail(kErrMaxIter);
            break;
          }
          nxt = st.top_id();
          nxt_s = st.top_s();
          if (!(dsub(nxt_s, cur_s) < 1e-14)) {
            const double s_ref = dmul(0.5, dadd(cur_s, nxt_s));
            double ref[3];
            ray_point(g, s_ref, ref[0], ref[1], ref[2]);
            s = split_analytic(g, min_image(c, ldg_pt(&c.pts[cur]), ref),
                               min_image(c, ldg_pt(&c.pts[nxt]), ref));
            if (s < DBL_MAX * 0.5 && s >= cur_s - kTol && s <= nxt_s + kTol) {
              use_split();
            } else {
              phase = kBisect;
              lo = cur_s;
              hi = nxt_s;
              tries = 0;
            }
            break;
          }
          st.pop();  // zero-width skip
          cur = nxt;
          cur_s = nxt_s;
          open_cell = cur;
          if (st.empty()) {
            finish_ok();
            break;
          }
        }
      }
      double x = 0.0, y = 0.0, z = 0.0, q_s = 0.0;
      const bool query = phase != kIdle;
      const bool one = phase != kSplit;
      if (phase == kStart) {
        x = g.s[0]; y = g.s[1]; z = g.s[2];
      } else if (phase == kEnd) {
        x = g.e[0]; y = g.e[1]; z = g.e[2];
      } else if (query) {
        if (phase == kSample) q_s = ddiv(dmul(g.len, (double)at), (double)(1 << level));
        else if (phase == kBisect) q_s = dmul(0.5, dadd(lo, hi));
        else q_s = s;
        ray_point(g, q_s, x, y, z);
      }
      __syncwarp();
      // ---- the searches of the warp, together: the query itself, then its images
      // in the reference's order while they are within reach
      KnnList<3> r;
      r.clear();
      if (query) {
        ++n_q;
        knn64_fetch(c, f64, x, y, z, pinf(), r, n_visit);
      }
      __syncwarp();
      bool tie = one && r.id[1] >= 0 && r.r2[1] == r.r2[0];
      const ImageDist dist(c, x, y, z);
      int im = 27;
      if (query && r.id[0] >= 0 && !dist.none(dadd(one ? r.r2[0] : r.r2[2], kTol))) im = 0;
      for (;;) {
        const double bound = one ? r.r2[0] : r.r2[2];
        while (im < 27 && (im == 13 || dist(im / 9 - 1, im / 3 % 3 - 1, im % 3 - 1) >
                                           dadd(bound, kTol)))
          ++im;
        if (!__any_sync(FULL, im < 27)) break;
        if (im < 27) {
          // (only entries nearer than the bound can change the list)
          KnnList<3> f;
          f.clear();
          knn64_fetch(c, f64, dadd(x, dmul((double)(im / 9 - 1), c.box[0])),
                      dadd(y, dmul((double)(im / 3 % 3 - 1), c.box[1])),
                      dadd(z, dmul((double)(im % 3 - 1), c.box[2])), bound, f, n_visit);
          if (!one) {
            merge_image(r, f);
          } else if (f.id[0] >= 0) {
            tie = tie || (f.id[1] >= 0 && f.r2[1] == f.r2[0]);
            r.id[0] = f.id[0];
            r.r2[0] = f.r2[0];
          }
          ++im;
        }
        __syncwarp();
      }
      // ---- apply
      bool split = false;
      if (!query) {
      } else if (r.id[0] < 0) {
        fail(kErrNonFiniteDist);  // squared distances overflowed
      } else if (tie) {
        fail(kNeedTie);  // exactly tied nearest cells: resolved in k_slow
      } else if (phase == kStart) {
        c0 = r.id[0];
        phase = kEnd;
      } else if (phase == kEnd) {
        st.push(r.id[0], g.len);
        cur = open_cell = c0;
        phase = r.id[0] == c0 ? kSample : kNext;
      } else if (phase == kSample) {
        // a second cell on the ray, at 1/2, 1/4, 3/4, 1/8, ... (src/ray.cpp:220-246)
        if (r.id[0] != c0) {
          st.push(r.id[0], q_s);
          phase = kNext;
        } else if ((at += 2) >= 1 << level) {
          at = 1;
          if (++level > 10) fail(kErrPeriodicBisect);
        }
      } else if (phase == kBisect) {
        const int mc = r.id[0];
        if (mc != cur && mc != nxt) {
          s = q_s;
          use_split();
        } else {
          if (mc == cur) lo = q_s;
          else hi = q_s;
          if (dsub(hi, lo) < 1e-12) {
            s = dmul(0.5, dadd(lo, hi));
            use_split();
          } else if (++tries >= 64) {
            fail(kErrBinSearch);
          }
        }
      } else {
        split = true;
      }
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
      one_by_one(split && three_eq && !has_c && !has_n, [&] {
        const RareOut ro = rare_expand_periodic(c, x, y, z, cur, nxt);
        n_q += ro.nq;
        if (ro.rc) fail(ro.rc);
        has_c = ro.a;
        has_n = ro.b;
      });
      int sc = r.id[0], sn = r.id[0];
      one_by_one(split && phase != kIdle && !has_c && !has_n &&
                     !(dadd(r.r2[0], kTol) < r.r2[1]),
                 [&] {
                   const RareOut ro = rare_case1a_periodic(c, g, x, y, z, cur, nxt);
                   n_q += ro.nq;
                   sc = ro.a;
                   sn = ro.b;
                   if (ro.rc) fail(ro.rc);
                 });
      if (split && phase != kIdle) {
        phase = kNext;
        if (has_c || has_n) {
          emit(open_cell, entry_s, s);
          open_cell = nxt;
          entry_s = s;
          st.pop();
          cur = nxt;
          cur_s = nxt_s;
          if (st.empty()) finish_ok();
        } else if (st.room() < (sc == sn ? 1 : 2)) {
          fail(kNeedSlow);
        } else {
          if (sc != sn) st.push(sn, s);
          st.push(sc, s);
        }
      }
      if constexpr (OUT == kOutTape) red.flush_tape(io);
    }
    max_sp = max(max_sp, (unsigned)st.maxsp);
  }
  warp_add(&io.stats->rays, n_rays);
  warp_add(&io.stats->crossings, n_cross);
  warp_add(&io.stats->queries, n_q);
  warp_max(&io.stats->max_stack, max_sp);
}

template <int MODE, int NF, int OUT>
int launch_periodic(vt_cloud* cl, WalkIO& io, cudaStream_t st) {
  int dev = 0, nsms = 0;
  VT_CUDA(cudaGetDevice(&dev));
  VT_CUDA(cudaDeviceGetAttribute(&nsms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t most = (int64_t)nsms * VT_PERIODIC_MINB, need = (io.nrays + 3) / 4;
  const int64_t blocks = need < most ? need : most, warps = 4 * blocks;
  const int64_t per = (io.nrays + warps - 1) / warps;
  io.batch = (int)(per < 1 ? 1 : (per < 32 ? per : 32));
  k_periodic<MODE, NF, OUT><<<(unsigned)blocks, 128, 0, st>>>(cl->view, io);
  return VT_OK;
}

}  // namespace vt
