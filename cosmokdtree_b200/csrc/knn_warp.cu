// knn_warp.cu -- exact kNN with a warp per query (sorted rows, k <= 128).
//
// The per-lane kernel (ckd_knn_lane.cuh) needs tens of thousands of queries to
// fill the GPU and keeps k heap entries per lane in shared memory.  Here the 32
// lanes of a warp share one query:
//
//   * the k best are a sorted list in registers (R per lane, 32 R >= k entries),
//     so no heap and no final sort; candidates that pass the bound are collected
//     in shared memory and merged 32 at a time by a bitonic network;
//   * the descent follows the nearer child down to a subtree of at most
//     max(32, 2 k) points, whose whole leaf-ordered range is scanned (lanes over
//     points, coalesced FP64 records) and gives the first bound;
//   * after that up to 32 pending subtrees are taken from the stack at once, a
//     lane each: their children are tested in parallel, subtrees of at most
//     kUnit points are scanned as ranges, the ranges flattened over the lanes.
//
// Bound by instruction issue and dependent loads: 2^20 uniform points, k = 16,
// 100k queries issue about 4000 warp instructions a query.  Measured (us a call,
// before -> with this kernel): one query of 2^20 points, k = 16: 54 -> 24; 30k
// queries of 10^6 clustered points, k = 100: 9470 -> 660 (heaps in the output rows
// before); 200k queries of 2^22 6-D points, k = 64: 16060 -> 6830 (per-lane
// before).  The seed's descent follows the split planes alone (a 32-byte record a
// level) and leaves the siblings' boxes to be tested by the lanes together: 568 ->
// 514 us on the 100k queries above.  Two points a lane and pass of a scan: 6-D,
// k = 16, 2335 -> 2073 us.  An FP32 screen of the points before the FP64 records
// gained nothing (6-D, k = 64: 4020 without, 4190 with).
//
// Ranking is by (FP64 squared distance, id) throughout, the same separately
// rounded arithmetic as every other kernel, so rows equal the per-lane kernel's.
#include "ckd_common.cuh"
#include "ckd_knn.cuh"
#include "ckd_traverse.cuh"

namespace ckd {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int kWarpStack = 320;    // pending subtrees per warp
constexpr int kWarpReserve = 130;  // stack room kept for one-at-a-time descents (tree depth < 127)
constexpr unsigned kUntested = 0xffffffffu;  // stack entry whose box has not been tested
constexpr int32_t kUnit = 16;     // subtrees of at most this many points are scanned as a range
constexpr int kUnitRun = 16;      // ranges that wait before they are scanned
constexpr int U = 2;  // points per lane and pass of a scan
constexpr int kUnitList = 128;     // ranges waiting for a scan, per warp

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

// The sorted list of the best 32 R candidates: entry s in register s / 32 of lane
// s % 32.
template <int R>
struct WarpList {
  double d[R];
  int32_t i[R];

  // merge one candidate per lane (cd = +inf, ci = INT32_MAX: none)
  __device__ __forceinline__ void merge(double cd, int32_t ci, int lane) {
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
      for (int m = size >> 1; m > 0; m >>= 1)  // descending over the warp
        cas_lane(cd, ci, m, ((lane & m) == 0) != ((lane & size) == 0));
    // the last 32 entries against the descending candidates: the smaller of each
    // pair leaves a bitonic sequence holding the best 32 R of all
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
    for (int m = 16; m > 0; m >>= 1)
#pragma unroll
      for (int r = 0; r < R; ++r) cas_lane(d[r], i[r], m, (lane & m) == 0);
  }
};

template <int D, bool PER, int R>
__global__ void __launch_bounds__(128) k_knn_warp(TreeView tv, const double* __restrict__ Q,
                                                  const int32_t* __restrict__ order, int64_t nq,
                                                  int k, double* __restrict__ dist,
                                                  int64_t* __restrict__ idx,
                                                  const int32_t* __restrict__ qroot) {
  constexpr int NV = (D + 3) / 4;
  constexpr int PF = pair_f4(D);
  __shared__ uint2 s_stk[4][kWarpStack];  // (node, or ~node to scan; bound bits)
  __shared__ double s_bd[4][32 * (U + 1)];          // candidates waiting for a merge
  __shared__ int32_t s_bi[4][32 * (U + 1)];
  __shared__ int2 s_ur[4][kUnitList];     // ranges waiting for a scan: first point, count
  __shared__ float s_ul[4][kUnitList];    // and their bounds
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int64_t slot = (int64_t)blockIdx.x * 4 + w;
  if (slot >= nq) return;  // the whole warp leaves together
  uint2* stk = s_stk[w];
  double* bufd = s_bd[w];
  int32_t* bufi = s_bi[w];
  int2* ur = s_ur[w];
  float* ul = s_ul[w];
  const int64_t qi = order ? (int64_t)order[slot] : slot;

  double q[D];
  QueryScreen<D, PER> qs;
  float xl[D], xh[D];
#pragma unroll
  for (int j = 0; j < D; ++j) {
    q[j] = Q[qi * D + j];
    qs.q32[j] = __double2float_rn(q[j]);
    qs.dlt[j] = kTwoM21 * (fabsf(qs.q32[j]) + tv.slack[j]) * 1.0001f;
    xl[j] = __fadd_ru(qs.q32[j], qs.dlt[j]);
    xh[j] = __fsub_rd(qs.q32[j], qs.dlt[j]);
  }
  bool wf = !PER;  // the ball cannot reach the periodic faces: direct gaps bound it
  WarpList<R> L;
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
  // merge the oldest 32 waiting candidates (fewer at the end)
  auto flush = [&]() {
    const bool have = lane < nb;
    const double cd = have ? bufd[lane] : CUDART_INF;
    const int32_t ci = have ? bufi[lane] : 0x7fffffff;
    __syncwarp();
    for (int o = 32; o < nb; o += 32) {  // move the rest down
      const bool more = o + lane < nb;
      const double md = more ? bufd[o + lane] : 0.0;
      const int32_t mi = more ? bufi[o + lane] : 0;
      __syncwarp();
      if (more) {
        bufd[o - 32 + lane] = md;
        bufi[o - 32 + lane] = mi;
      }
      __syncwarp();
    }
    nb = nb > 32 ? nb - 32 : 0;
    L.merge(cd, ci, lane);
    const int kr = (k - 1) >> 5, kl = (k - 1) & 31;
    double sd = L.d[0];
    int32_t si = L.i[0];
#pragma unroll
    for (int r = 1; r < R; ++r)
      if (r == kr) {
        sd = L.d[r];
        si = L.i[r];
      }
    bd = __shfl_sync(FULL, sd, kl);
    bid = __shfl_sync(FULL, si, kl);
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
  const int32_t seed = max(64, 4 * k);
  int nu = 0;  // ranges waiting to be scanned
  int top = 0;
  int32_t next = qroot ? qroot[qi] : 0;  // subtree of the next seed descent, -1: none
  while (next >= 0 || top > 0) {
    if (bd == CKD_HUGE) {
      // fewer than k found yet: nearer-first descent from the nearest waiting
      // subtree (at first the root) to a range
      if (next < 0) {
        --top;
        next = (int32_t)stk[top].x;
        __syncwarp();
      }
      NodeMeta m = load_meta(tv.meta, next);
      while (m.left >= 0 && m.count > seed) {
        double qa = 0.0;
#pragma unroll
        for (int j = 0; j < D; ++j)
          if (j == m.axis) qa = q[j];
        const bool left = qa < m.split;
        if (lane == 0)
          stk[top] = make_uint2((unsigned)(left ? m.left + 1 : m.left), kUntested);
        ++top;
        m = load_meta(tv.meta, left ? m.left : m.left + 1);
      }
      const int32_t st = m.start, ct = m.count;
      if (lane == 0) {
        ur[nu] = make_int2(st, ct);
        ul[nu] = 0.0f;
      }
      ++nu;
      __syncwarp();
      next = -1;
    } else {
      // up to 32 waiting subtrees at once, a lane each
      const int n = min(min(top, 32), max(1, kWarpStack - kWarpReserve - top));
      int32_t c = -1, c0 = -1, c1 = -1, st0 = 0, ct0 = 0, st1 = 0, ct1 = 0;
      float l0 = 0.0f, l1 = 0.0f;
      if (lane < n) {
        const uint2 e = stk[top - 1 - lane];
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
      __syncwarp();
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
      // push the internal children
      const unsigned b0 = __ballot_sync(FULL, c0 >= 0), b1 = __ballot_sync(FULL, c1 >= 0);
      const int o = top + __popc(b0 & lt) + __popc(b1 & lt);
      if (c0 >= 0) stk[o] = make_uint2((unsigned)c0, __float_as_uint(l0));
      if (c1 >= 0) stk[o + (c0 >= 0 ? 1 : 0)] = make_uint2((unsigned)c1, __float_as_uint(l1));
      top += __popc(b0) + __popc(b1);
      // list the ranges
      const unsigned u0 = __ballot_sync(FULL, ct0 > 0), u1 = __ballot_sync(FULL, ct1 > 0);
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
    }
    // Scan the listed ranges, flattened over the warp, when enough wait (the list
    // holds another round's 64 at any time), while fewer than k are known, and at
    // the end; what then waits for a merge is merged too in the last two cases.
    const bool force = bd == CKD_HUGE || top == 0;
    if (nu < kUnitRun && !force) continue;
#pragma unroll 1
    for (int u0 = 0; u0 < nu || (force && nb > 0); u0 += 32) {
      int32_t st = 0, ct = 0;
      float lb = 0.0f;
      if (u0 + lane < nu) {
        const int2 r = ur[u0 + lane];
        lb = ul[u0 + lane];
        st = r.x;
        ct = lb <= wd32 ? r.y : 0;
      }
      int32_t inc = ct;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t v = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += v;
      }
      const int32_t total = __shfl_sync(FULL, inc, 31);
      const int32_t delta = st - (inc - ct);  // position = delta + flattened index
      const bool last = force && u0 + 32 >= nu;
#pragma unroll 1
      for (int32_t b = 0; b < total || (last && nb > 0); b += 32 * U) {
        if (b < total) {
          double d2[U];
          int32_t id[U];
          bool pass[U];
#pragma unroll
          for (int c = 0; c < U; ++c) {
            const int32_t t = b + 32 * c + lane;
            int j = 0;  // the range holding t: the first with inc > t
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
              const int32_t v = __shfl_sync(FULL, inc, j + o - 1);
              if (v <= t) j += o;
            }
            const int32_t p = __shfl_sync(FULL, delta, j) + t;
            pass[c] = t < total;
            id[c] = 0;
            d2[c] = 0.0;
            if (pass[c]) {
              d2[c] = point_d2_rec<D, PER>(tv, q, p);
              id[c] = CKD_LDT(&tv.ids[p]);
            }
          }
#pragma unroll
          for (int c = 0; c < U; ++c) {
            pass[c] = pass[c] && rank_lt(d2[c], id[c], bd, bid);
            const unsigned pm = __ballot_sync(FULL, pass[c]);
            if (pass[c]) {
              const int o = nb + __popc(pm & lt);
              bufd[o] = d2[c];
              bufi[o] = id[c];
            }
            nb += __popc(pm);
          }
          __syncwarp();
        }
        while (nb >= 32 || (nb > 0 && last && b + 32 * U >= total)) flush();
      }
    }
    nu = 0;
    __syncwarp();
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int s = r * 32 + lane;
    if (s < k) {
      dist[qi * k + s] = sqrt(L.d[r]);
      idx[qi * k + s] = L.i[r] < 0 ? -2 : (int64_t)L.i[r];
    }
  }
}

template <int D, bool PER>
ckd_status warp_launch(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq, int k,
                       double* dist, int64_t* idx, const int32_t* qroot, cudaStream_t s) {
  const unsigned g = (unsigned)cdiv(nq, 4);
  const TreeView tv = t->view();
  if (k <= 32)
    k_knn_warp<D, PER, 1><<<g, 128, 0, s>>>(tv, q, order, nq, k, dist, idx, qroot);
  else if (k <= 64)
    k_knn_warp<D, PER, 2><<<g, 128, 0, s>>>(tv, q, order, nq, k, dist, idx, qroot);
  else
    k_knn_warp<D, PER, 4><<<g, 128, 0, s>>>(tv, q, order, nq, k, dist, idx, qroot);
  CKD_LAUNCH_CHECK();
  return CKD_OK;
}

}  // namespace

ckd_status knn_warp(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq, int k,
                    double* dist, int64_t* idx, const int32_t* qroot, cudaStream_t s) {
  switch (t->d * 2 + (t->periodic ? 1 : 0)) {
#define CKD_KW(DD)                                                                         \
  case 2 * DD: return warp_launch<DD, false>(t, q, order, nq, k, dist, idx, qroot, s);     \
  case 2 * DD + 1: return warp_launch<DD, true>(t, q, order, nq, k, dist, idx, qroot, s);
    CKD_KW(1) CKD_KW(2) CKD_KW(3) CKD_KW(4) CKD_KW(5) CKD_KW(6) CKD_KW(7) CKD_KW(8)
#undef CKD_KW
  }
  return fail(CKD_ERR_BAD_DIM, "dimensionality must be 1..8");
}

}  // namespace ckd
