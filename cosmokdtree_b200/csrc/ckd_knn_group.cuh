// ckd_knn_group.cuh -- exact kNN with G = 32, 16 or 8 lanes of a warp per query
// (sorted rows, k <= 128).
//
// The per-lane kernel (ckd_knn_lane.cuh) needs hundreds of thousands of queries to
// fill the GPU and keeps k heap entries per lane in shared memory.  Here the lanes of
// a group share one query, and the 32 / G queries of a warp go in step:
//
//   * the k best are a sorted list in registers (R per lane, G R >= k entries), so
//     no heap and no final sort; candidates that pass the bound are collected in
//     shared memory and merged G at a time by a bitonic network, for all queries of
//     the warp when one of them has G waiting;
//   * a descent along the query's side of the split planes (a 32-byte record a level)
//     to a subtree of at most max(2 G, 4 k) points, whose whole leaf-ordered range is
//     scanned (lanes over points, FP64 records), gives the first bound; the
//     siblings' boxes are tested later, by the lanes together;
//   * after that up to G pending subtrees are taken from the stack at once, a lane
//     each: their children are tested in parallel, subtrees of at most kUnit points
//     are scanned as ranges, the ranges flattened over the lanes.
//
// Bound by instruction issue (70-76 % of slots at G = 8 and 16) and, for small batches,
// by dependent loads.  Measured (us a call, before -> now): one query of 2^20 points,
// k = 16: 54 -> 16 (a lane before; part of it the shorter way through the host); 30k queries
// of 10^6 clustered points, k = 100: 9470 -> 549 (heaps in the output rows before); 200k
// queries of 2^22 6-D points, k = 64: 16060 -> 6370; 100k queries of 2^22 clustered points,
// k = 32: 1199 -> 847.  The whole warp for each of the last ones takes 947: fewer lanes a
// query waste less on short ranges and few pending nodes, at the price of waiting for
// three neighbours.
// Dropped: following single children inside a lane (10 to 30 % slower), an FP32
// screen of the points before the FP64 records (no gain).
//
// Ranking is by (FP64 squared distance, id) throughout, the same separately
// rounded arithmetic as every other kernel, so rows equal the per-lane kernel's.
#pragma once
#include <algorithm>

#include "ckd_common.cuh"
#include "ckd_knn.cuh"
#include "ckd_traverse.cuh"

namespace ckd {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr unsigned kUntested = 0xffffffffu;  // stack entry whose box has not been tested
constexpr int32_t kUnit = 16;     // subtrees of at most this many points are scanned as a range

// (d, id) lexicographic order
__device__ __forceinline__ bool rank_lt(double d1, int32_t i1, double d2, int32_t i2) {
  return d1 < d2 || (d1 == d2 && i1 < i2);
}

// one compare-exchange of a bitonic network across lanes: keep the smaller of
// (own, partner's) iff keep_min
__device__ __forceinline__ void cas_lane(double& d, int32_t& i, int mask, bool keep_min) {
  const double od = __shfl_xor_sync(FULL, d, mask);
  const int32_t oi = __shfl_xor_sync(FULL, i, mask);
  if (rank_lt(od, oi, d, i) == keep_min) {
    d = od;
    i = oi;
  }
}

// The sorted list of a query's best G R candidates: entry s in register s / G of
// the query's lane s % G.
template <int G, int R>
struct GroupList {
  double d[R];
  int32_t i[R];

  // merge one candidate per lane (cd = +inf, ci = INT32_MAX: none)
  __device__ __forceinline__ void merge(double cd, int32_t ci, int gl) {
#pragma unroll
    for (int size = 2; size <= G; size <<= 1)
#pragma unroll
      for (int m = size >> 1; m > 0; m >>= 1)  // descending over the group
        cas_lane(cd, ci, m, ((gl & m) == 0) != ((gl & size) == 0));
    // the last G entries against the descending candidates: the smaller of each
    // pair leaves a bitonic sequence holding the best G R of all
    if (rank_lt(cd, ci, d[R - 1], i[R - 1])) {
      d[R - 1] = cd;
      i[R - 1] = ci;
    }
#pragma unroll
    for (int m = R >> 1; m > 0; m >>= 1)
#pragma unroll
      for (int r = 0; r < R; ++r)
        if ((r & m) == 0 && rank_lt(d[r + m], i[r + m], d[r], i[r])) {
          const double td = d[r];
          const int32_t ti = i[r];
          d[r] = d[r + m];
          i[r] = i[r + m];
          d[r + m] = td;
          i[r + m] = ti;
        }
#pragma unroll
    for (int m = G >> 1; m > 0; m >>= 1)
#pragma unroll
      for (int r = 0; r < R; ++r) cas_lane(d[r], i[r], m, (gl & m) == 0);
  }
};

// Shared memory of a query: stack of pending subtrees (node, bound bits), ranges
// waiting for a scan (first point, count; bound), candidates waiting for a merge.
template <int G>
struct GroupShape {
  static constexpr int kQ = 32 / G;                   // queries per warp
  static constexpr int U = 2;                         // points per lane and pass of a scan
  static constexpr int kRun = G / 2;                  // ranges that wait before they are scanned
  static constexpr int kList = kRun + 2 * G;          // a round adds at most 2 G
  static constexpr int kBuf = G * (U + 1);
};
// stack entries: a round's growth above the room for one-at-a-time descents
__host__ __device__ constexpr int group_stack(int g, int depth) { return 2 * depth + 4 + 2 * g; }
template <int G>
size_t group_smem(int depth) {  // per block of 4 warps
  using S = GroupShape<G>;
  return (size_t)4 * S::kQ *
         (group_stack(G, depth) * 8 + S::kBuf * 12 + S::kList * 12);
}

// What a bounded search gets besides: every query's squared bound and leaf, and the
// list of the queries that hold fewer than k points within their bound.
struct GroupBound {
  const double* r2;
  const int32_t* qleaf;
  int32_t* miss;
  unsigned* nmiss;
};

// BOUND: every list starts full of sentinels (r2, INT32_MAX) instead of HUGE, so
// pruning starts at once, at the lowest ancestor of the query's leaf whose cell strictly
// contains the ball, from where the same descent gives the nearest range first (a loose
// bound alone, as in voids, prunes little until k are found: 500k queries of 2^22 points
// of one cluster, half of them outside it, k = 64: 39.4 -> 30.9 ms, of 2^22 clustered points
// 5.8 -> 5.2, 6-D 10 % less); every point with d2 <= r2 is still accepted, so a list that ends
// without a sentinel among its first k is exact.  The others are listed for a rerun and
// their rows are not written.
template <int D, bool PER, int G, int R, bool BOUND = false>
__global__ void __launch_bounds__(128) k_knn_group(TreeView tv, const double* __restrict__ Q,
                                                   const int32_t* __restrict__ order, int64_t nq,
                                                   int k, int depth, double* __restrict__ dist,
                                                   int64_t* __restrict__ idx,
                                                   const int32_t* __restrict__ qroot,
                                                   GroupBound gb = GroupBound{}) {
  using S = GroupShape<G>;
  constexpr int NV = (D + 3) / 4, PF = pair_f4(D), U = S::U, NG = 4 * S::kQ;
  extern __shared__ __align__(16) unsigned char gsm[];
  const int scap = group_stack(G, depth);
  const int lane = threadIdx.x & 31;
  const int gl = lane & (G - 1), grp = threadIdx.x / G;  // lane of the query, query of the block
  const int gsh = lane & ~(G - 1);                       // first lane of the query
  const unsigned gm = G == 32 ? FULL : ((1u << (G & 31)) - 1u);
  const unsigned lt = (1u << gl) - 1u;
  // bits of the query's lanes in a ballot of the warp
  auto ballot = [&](bool p) -> unsigned { return (__ballot_sync(FULL, p) >> gsh) & gm; };
  double* bufd = reinterpret_cast<double*>(gsm) + (size_t)grp * S::kBuf;
  uint2* stk = reinterpret_cast<uint2*>(gsm + (size_t)NG * S::kBuf * 8) + (size_t)grp * scap;
  int2* ur = reinterpret_cast<int2*>(gsm + (size_t)NG * (S::kBuf + scap) * 8) + grp * S::kList;
  float* ul = reinterpret_cast<float*>(gsm + (size_t)NG * (S::kBuf + scap + S::kList) * 8) +
              grp * S::kList;
  int32_t* bufi = reinterpret_cast<int32_t*>(
                      gsm + (size_t)NG * ((S::kBuf + scap + S::kList) * 8 + S::kList * 4)) +
                  grp * S::kBuf;
  const int64_t slot = (int64_t)blockIdx.x * NG + grp;
  if (slot - grp % S::kQ >= nq) return;  // a warp without queries leaves together
  const bool valid = slot < nq;
  const int64_t qi = valid ? (order ? (int64_t)order[slot] : slot) : 0;

  double q[D];
  QueryScreen<D, PER> qs;
  float xl[D], xh[D];
#pragma unroll
  for (int j = 0; j < D; ++j) {
    q[j] = valid ? Q[qi * D + j] : 0.0;
    qs.q32[j] = __double2float_rn(q[j]);
    qs.dlt[j] = kTwoM21 * (fabsf(qs.q32[j]) + tv.slack[j]) * 1.0001f;
    xl[j] = __fadd_ru(qs.q32[j], qs.dlt[j]);
    xh[j] = __fsub_rd(qs.q32[j], qs.dlt[j]);
  }
  bool wf = !PER;  // the ball cannot reach the periodic faces: direct gaps bound it
  GroupList<G, R> L;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    L.d[r] = CKD_HUGE;
    L.i[r] = -1;
  }
  double bd = CKD_HUGE;  // the k-th best (d2, id) so far
  int32_t bid = -1;
  float wd32 = FLT_MAX;  // FP32 upper bound of bd
  int nb = 0;            // candidates waiting

  auto box_lb = [&](const float (&lo)[4 * NV], const float (&hi)[4 * NV]) -> float {
    if (!PER || wf) {
      float s2 = 0.0f;
#pragma unroll
      for (int j = 0; j < D; ++j) {
        const float g = fmaxf(fmaxf(lo[j] - xl[j], xh[j] - hi[j]), 0.0f);
        s2 = fmaf(g, g, s2);
      }
      return s2 * kShrink;
    }
    return box_mind_lb<D, PER>(tv, qs, lo, hi);
  };
  auto node_lb = [&](int32_t nd) -> float {
    float lo[4 * NV], hi[4 * NV];
    const float2* b = reinterpret_cast<const float2*>(tv.box32 + (int64_t)nd * 2 * D);
#pragma unroll
    for (int j = 0; j < D; ++j) {
      const float2 lh = CKD_LDT(b + j);
      lo[j] = lh.x;
      hi[j] = lh.y;
    }
    return box_lb(lo, hi);
  };
  // both children of an internal node: bounds, ids (~id when scanned as a range)
  // and ranges
  auto expand = [&](int32_t node, float& ml, float& mr, int4& info, int4& range) {
    const float4* rec = tv.pair + (int64_t)node * PF;
    float v[4][4 * NV];
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int h = 0; h < NV; ++h) {
        const float4 f = CKD_LDT(rec + b * NV + h);
        v[b][4 * h] = f.x;
        v[b][4 * h + 1] = f.y;
        v[b][4 * h + 2] = f.z;
        v[b][4 * h + 3] = f.w;
      }
    info = CKD_LDT(reinterpret_cast<const int4*>(rec + 4 * NV));
    range = CKD_LDT(reinterpret_cast<const int4*>(rec + 4 * NV + 1));
    ml = box_lb(v[0], v[1]);
    mr = box_lb(v[2], v[3]);
  };
  // merge up to G waiting candidates of every query of the warp
  auto flush = [&]() {
    const bool have = gl < nb;
    const double cd = have ? bufd[gl] : CUDART_INF;
    const int32_t ci = have ? bufi[gl] : 0x7fffffff;
    __syncwarp();
#pragma unroll
    for (int o = G; o < S::kBuf; o += G) {  // move the rest down
      const bool more = o + gl < nb;
      const double md = more ? bufd[o + gl] : 0.0;
      const int32_t mi = more ? bufi[o + gl] : 0;
      if (more) {
        bufd[o - G + gl] = md;
        bufi[o - G + gl] = mi;
      }
      __syncwarp();
    }
    nb = nb > G ? nb - G : 0;
    L.merge(cd, ci, gl);
    const int kr = (k - 1) / G, kl = (k - 1) & (G - 1);
    double sd = L.d[0];
    int32_t si = L.i[0];
#pragma unroll
    for (int r = 1; r < R; ++r)
      if (r == kr) {
        sd = L.d[r];
        si = L.i[r];
      }
    bd = __shfl_sync(FULL, sd, kl, G);
    bid = __shfl_sync(FULL, si, kl, G);
    wd32 = __double2float_ru(bd);
    if (PER && !wf) {
      const float r32 = sqrt_up(wd32);
      bool inside = true;
#pragma unroll
      for (int j = 0; j < D; ++j)
        inside = inside &&
                 __fadd_ru(__fadd_ru(fabsf(qs.q32[j]), r32), qs.dlt[j]) < 0.5f * (float)tv.L[j];
      wf = inside;
    }
  };
  // Whether the query is further than HUGE from every point, by the largest coordinate of
  // each axis, or not finite: it finds nothing, and would read the whole tree for it (64
  // such of 2^20 points, k = 100: 16 ms).  Asked for only when the first range has
  // left fewer than k, off the path that every query takes, of values that the walk holds.
  // Not on periodic trees, whose queries lie in the box.
  auto beyond = [&]() -> bool {
    float s2 = 0.0f;
#pragma unroll
    for (int j = 0; j < D; ++j) {
      const float b = tv.slack[j], g = 0.5f * fmaxf(fmaxf(-b - xl[j], xh[j] - b), 0.0f);
      s2 = xl[j] - xh[j] <= FLT_MAX ? fmaf(g, g, s2) : CUDART_INF_F;
    }
    return !(s2 * kShrink <= 0.25f * FLT_MAX);
  };
  const int32_t seed = max(2 * G, 4 * k);
  int nu = 0;  // ranges waiting to be scanned
  int top = 0;
  int32_t next = valid ? (qroot ? qroot[qi] : 0) : -1;  // next seed descent's subtree, -1: none
  if (BOUND && valid) {
    const double b = gb.r2[qi];
    if (b < CKD_HUGE) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        L.d[r] = b;
        L.i[r] = 0x7fffffff;
      }
      bd = b;
      bid = 0x7fffffff;
      wd32 = __double2float_ru(b);
      const float r32 = __fsqrt_ru(wd32);
      int32_t a = gb.qleaf[qi];
      while (a >= 0) {
        const float2* c = reinterpret_cast<const float2*>(tv.cell32 + (int64_t)a * 2 * D);
        bool inside = true;
#pragma unroll
        for (int j = 0; j < D; ++j) {
          const float2 lh = CKD_LDT(c + j);
          inside = inside && __fsub_rd(__fsub_rd(qs.q32[j], r32), qs.dlt[j]) > lh.x &&
                   __fadd_ru(__fadd_ru(qs.q32[j], r32), qs.dlt[j]) < lh.y;
        }
        if (inside) break;
        a = load_meta(tv.meta, a).parent;
      }
      if (a >= 0) next = a;  // the descent starts there
    }
  }
  __syncwarp();
  while (__any_sync(FULL, next >= 0 || top > 0)) {
    const bool act = next >= 0 || top > 0;
    if (next < 0 && top > 0 && bd == CKD_HUGE) {
      next = (int32_t)stk[--top].x;
      if (!PER && beyond()) {
        next = -1;
        top = 0;
      }
    }
    __syncwarp();
    int32_t c0 = -1, c1 = -1, st0 = 0, ct0 = 0, st1 = 0, ct1 = 0;
    float l0 = 0.0f, l1 = 0.0f;
    const bool seeded = next >= 0;
    if (seeded) {
      // fewer than k found yet: descent from the nearest waiting subtree (at first
      // the root) along the query's side of the splits to a range
      NodeMeta m = load_meta(tv.meta, next);
      while (m.left >= 0 && m.count > seed) {
        double qa = 0.0;
#pragma unroll
        for (int j = 0; j < D; ++j)
          if (j == m.axis) qa = q[j];
        const bool left = qa < m.split;
        if (gl == 0)  // the sibling waits
           stk[top] = make_uint2((unsigned)(left ? m.left + 1 : m.left), kUntested);
        ++top;
        m = load_meta(tv.meta, left ? m.left : m.left + 1);
      }
      next = -1;
      if (gl == 0) {
        st0 = m.start;
        ct0 = m.count;
      }
    } else if (act) {
      // up to G waiting subtrees at once, a lane each
      const int n = min(min(top, G), max(1, depth + 2 * G - top));
      int32_t c = -1;
      if (gl < n) {
        const uint2 e = stk[top - 1 - gl];
        c = (int32_t)e.x;
        l0 = __uint_as_float(e.y);
        if (e.y == kUntested) {  // a sibling of the descent: its box is tested here
          const NodeMeta m = load_meta(tv.meta, c);
          l0 = node_lb(c);
          if (m.left < 0 || m.count <= kUnit) {
            if (l0 <= wd32) {
              st0 = m.start;
              ct0 = m.count;
            }
            c = -1;
          }
        }
      }
      top -= n;
      if (c >= 0 && l0 <= wd32) {
        int4 info, range;
        expand(c, l0, l1, info, range);
        const bool nl = l0 <= wd32, nr = l1 <= wd32;
        const bool rl = info.z || range.y <= kUnit, rr = info.w || range.w <= kUnit;
        if (nl && rl) {
          st0 = range.x;
          ct0 = range.y;
        }
        if (nr && rr) {
          st1 = range.z;
          ct1 = range.w;
        }
        if (nl && !rl) c0 = info.x;
        if (nr && !rr) c1 = info.y;
      }
    }
    __syncwarp();
    // push the internal children
    const unsigned b0 = ballot(c0 >= 0), b1 = ballot(c1 >= 0);
    const int o = top + __popc(b0 & lt) + __popc(b1 & lt);
    if (c0 >= 0) stk[o] = make_uint2((unsigned)c0, __float_as_uint(l0));
    if (c1 >= 0) stk[o + (c0 >= 0 ? 1 : 0)] = make_uint2((unsigned)c1, __float_as_uint(l1));
    top += __popc(b0) + __popc(b1);
    // list the ranges
    const unsigned u0 = ballot(ct0 > 0), u1 = ballot(ct1 > 0);
    const int u = nu + __popc(u0 & lt) + __popc(u1 & lt);
    if (ct0 > 0) {
      ur[u] = make_int2(st0, ct0);
      ul[u] = l0;
    }
    if (ct1 > 0) {
      ur[u + (ct0 > 0 ? 1 : 0)] = make_int2(st1, ct1);
      ul[u + (ct0 > 0 ? 1 : 0)] = l1;
    }
    nu += __popc(u0) + __popc(u1);
    __syncwarp();
    // Scan the listed ranges, flattened over the query's lanes, when enough wait,
    // while fewer than k are known, and at the end; what then waits for a merge is
    // merged too in the last two cases.
    const bool force = seeded || bd == CKD_HUGE || top == 0;
    const bool run = force || nu >= S::kRun;
    if (!__any_sync(FULL, run && (nu > 0 || nb > 0))) continue;
    const int nus = run ? nu : 0;
#pragma unroll 1
    for (int ub = 0; __any_sync(FULL, ub < nus || (force && nb > 0)); ub += G) {
      int32_t st = 0, ct = 0;
      if (ub + gl < nus) {
        const int2 r = ur[ub + gl];
        st = r.x;
        ct = ul[ub + gl] <= wd32 ? r.y : 0;
      }
      int32_t inc = ct;
#pragma unroll
      for (int x = 1; x < G; x <<= 1) {
        const int32_t v = __shfl_up_sync(FULL, inc, x, G);
        if (gl >= x) inc += v;
      }
      const int32_t total = __shfl_sync(FULL, inc, G - 1, G);
      const int32_t delta = st - (inc - ct);  // position = delta + flattened index
      const bool last = force && ub + G >= nus;
#pragma unroll 1
      for (int32_t b = 0; __any_sync(FULL, b < total || (last && nb > 0)); b += G * U) {
        double d2[U];
        int32_t id[U];
        bool pass[U];
#pragma unroll
        for (int x = 0; x < U; ++x) {
          const int32_t t = b + G * x + gl;
          int j = 0;  // the range holding t: the first with inc > t
#pragma unroll
          for (int y = G / 2; y > 0; y >>= 1) {
            const int32_t v = __shfl_sync(FULL, inc, j + y - 1, G);
            if (v <= t) j += y;
          }
          const int32_t p = __shfl_sync(FULL, delta, j, G) + t;
          pass[x] = t < total;
          id[x] = 0;
          d2[x] = 0.0;
          if (pass[x]) {
            d2[x] = point_d2_rec<D, PER>(tv, q, p);
            id[x] = CKD_LDT(&tv.ids[p]);
          }
        }
#pragma unroll
        for (int x = 0; x < U; ++x) {
          pass[x] = pass[x] && rank_lt(d2[x], id[x], bd, bid);
          const unsigned pm = ballot(pass[x]);
          if (pass[x]) {
            const int z = nb + __popc(pm & lt);
            bufd[z] = d2[x];
            bufi[z] = id[x];
          }
          nb += __popc(pm);
        }
        __syncwarp();
        while (__any_sync(FULL, nb >= G || (nb > 0 && last && b + G * U >= total))) flush();
      }
    }
    if (run) nu = 0;
    __syncwarp();
  }
  if (BOUND) {  // a sentinel among the first k: fewer than k points within the bound
    bool left = false;
#pragma unroll
    for (int r = 0; r < R; ++r) left = left || (r * G + gl < k && L.i[r] == 0x7fffffff);
    const bool missed = ballot(left) != 0;
    if (missed && gl == 0) gb.miss[atomicAdd(gb.nmiss, 1u)] = (int32_t)qi;
    if (missed) return;
  }
  if (!valid) return;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int s = r * G + gl;
    if (s < k) {
      dist[qi * k + s] = sqrt(L.d[r]);
      idx[qi * k + s] = L.i[r] < 0 ? -2 : (int64_t)L.i[r];
    }
  }
}

template <int D, bool PER, int G, int R>
ckd_status group_launch(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq, int k,
                        double* dist, int64_t* idx, const int32_t* qroot, cudaStream_t s) {
  k_knn_group<D, PER, G, R><<<(unsigned)cdiv(nq, 4 * GroupShape<G>::kQ), 128,
                              group_smem<G>(t->depth), s>>>(t->view(), q, order, nq, k, t->depth,
                                                            dist, idx, qroot);
  CKD_LAUNCH_CHECK();
  return CKD_OK;
}

// Lanes per query: fewer leave more queries in flight per instruction but split a
// query's work less, so the line moves with the batch and with k (2^20 uniform points,
// us at G = 32 / 16 / 8: 3000 queries, k = 16: 31 / 43 / 64; 25k, k = 8: 112 / 99 / 93;
// 100k, k = 16: 454 / 383 / 375; 50k, k = 32: 286 / 267 / 327).  In 6-D and for k > 32
// a query alone fills a warp's lanes (200k 6-D queries, k = 32: 4627 / 4847 / 6194).
template <int D, bool PER>
ckd_status group_pick(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq, int k,
                      double* dist, int64_t* idx, const int32_t* qroot, cudaStream_t s) {
  if constexpr (D <= 4) {
    if (k <= 32 && nq > 4000) {
      const bool eight = (k <= 8 && nq > 9000) || (k <= 16 && nq > 75000);
      if (eight && k <= 8) return group_launch<D, PER, 8, 1>(t, q, order, nq, k, dist, idx, qroot, s);
      if (eight) return group_launch<D, PER, 8, 2>(t, q, order, nq, k, dist, idx, qroot, s);
      if (k <= 16) return group_launch<D, PER, 16, 1>(t, q, order, nq, k, dist, idx, qroot, s);
      return group_launch<D, PER, 16, 2>(t, q, order, nq, k, dist, idx, qroot, s);
    }
  }
  if (k <= 32) return group_launch<D, PER, 32, 1>(t, q, order, nq, k, dist, idx, qroot, s);
  if (k <= 64) return group_launch<D, PER, 32, 2>(t, q, order, nq, k, dist, idx, qroot, s);
  return group_launch<D, PER, 32, 4>(t, q, order, nq, k, dist, idx, qroot, s);
}

template <int D, bool PER, int G, int R>
ckd_status group_bound_launch(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq,
                              int k, double* dist, int64_t* idx, const GroupBound& gb,
                              cudaStream_t s) {
  k_knn_group<D, PER, G, R, true><<<(unsigned)cdiv(nq, 4 * GroupShape<G>::kQ), 128,
                                    group_smem<G>(t->depth), s>>>(
      t->view(), q, order, nq, k, t->depth, dist, idx, nullptr, gb);
  CKD_LAUNCH_CHECK();
  return CKD_OK;
}

// the bounded search, k <= 64
template <int D, bool PER>
ckd_status group_bound_pick(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq,
                            int k, double* dist, int64_t* idx, const GroupBound& gb,
                            cudaStream_t s) {
  if constexpr (D <= 4) {
    if (k <= 16) return group_bound_launch<D, PER, 16, 1>(t, q, order, nq, k, dist, idx, gb, s);
    if (k <= 32) return group_bound_launch<D, PER, 16, 2>(t, q, order, nq, k, dist, idx, gb, s);
  } else {
    if (k <= 32) return group_bound_launch<D, PER, 32, 1>(t, q, order, nq, k, dist, idx, gb, s);
  }
  return group_bound_launch<D, PER, 32, 2>(t, q, order, nq, k, dist, idx, gb, s);
}

}  // namespace

// one translation unit instantiates each dimension (knn_group_*.cu)
#define CKD_KNN_GROUP(DD)                                                                        \
  ckd_status knn_group_d##DD(const ckd_tree* t, const double* q, const int32_t* order,           \
                             int64_t nq, int k, double* dist, int64_t* idx,                      \
                             const int32_t* qroot, cudaStream_t s) {                             \
    return t->periodic ? group_pick<DD, true>(t, q, order, nq, k, dist, idx, qroot, s)           \
                       : group_pick<DD, false>(t, q, order, nq, k, dist, idx, qroot, s);         \
  }                                                                                              \
  ckd_status knn_group_bound_d##DD(const ckd_tree* t, const double* q, const int32_t* order,     \
                                   int64_t nq, int k, double* dist, int64_t* idx,                \
                                   const double* r2, const int32_t* qleaf, int32_t* miss,        \
                                   unsigned* nmiss, cudaStream_t s) {                            \
    const GroupBound gb{r2, qleaf, miss, nmiss};                                                 \
    return t->periodic ? group_bound_pick<DD, true>(t, q, order, nq, k, dist, idx, gb, s)        \
                       : group_bound_pick<DD, false>(t, q, order, nq, k, dist, idx, gb, s);      \
  }

}  // namespace ckd
