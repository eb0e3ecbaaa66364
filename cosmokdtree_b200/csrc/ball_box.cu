// ball_box.cu -- ball (radius) and axis-aligned box searches, two-phase CSR.
//
// Ball (cosmokdtree.f90:1015-1212): a point is a result iff its FP64 squared
// distance (reference arithmetic) is <= radius^2 (inclusive, :1126, :1175).  The
// reference's "fully inside" shortcut (:1116-1118, :1332-1366) selects exactly
// the same points, because a node's max-distance bound is never below the
// computed distance of a point inside it; the searches use it with the tight box
// to skip distance work, on periodic trees too when the box lies within half a box
// side of the query on every axis.  An unsorted row is in leaf order, which is the
// reference's non-periodic order (left-first depth-first walk).  sorted=1 orders each
// row by (d2, id).
//
// Box (cosmokdtree.f90:1220-1328): descend left iff box_lo[axis] < split, right
// iff box_hi[axis] > split (strict), leaf test lo <= x <= hi on every axis
// (inclusive), no periodic wrap.  Rows are in leaf order, the reference's.
//
// Kernels: k_range_warp (balls and boxes, a warp per query), k_range_group (small
// balls, eight lanes per query), k_ball (packets of 32 queries: the first pass of very
// large batches, and trees too deep or coordinates too large for the FP32 tests),
// k_ball_fill_warp (heavy rows of those trees), k_box_lane (very large batches of
// boxes), k_box (boxes on trees deeper than its stack).
#include <algorithm>

#include "ckd_common.cuh"
#include "ckd_knn.cuh"
#include "ckd_traverse.cuh"

namespace ckd {

namespace {

constexpr int kStack = 96;

template <int D, bool PER, bool FILL, bool ROOTS = false>
__global__ void __launch_bounds__(128) k_ball(TreeView tv, const double* __restrict__ Q,
                                              const int32_t* __restrict__ order, int64_t nq_max,
                                              const unsigned* __restrict__ nq_dev,
                                              double r2, int32_t* __restrict__ gstack,
                                              int stack_len, int64_t* __restrict__ counts,
                                              const int64_t* __restrict__ offsets,
                                              int64_t* __restrict__ oidx,
                                              double* __restrict__ odist, int want_d2,
                                              const int32_t* __restrict__ qroot,
                                              int32_t* __restrict__ heavy = nullptr,
                                              unsigned* __restrict__ n_heavy = nullptr,
                                              int budget = 0) {
  // packet stack entries; with ROOTS (forests) each entry also carries the lanes
  // whose balls reached its parent, and the search starts one entry per distinct
  // root among the warp's queries
  __shared__ int32_t sstk[4][kStack];
  __shared__ unsigned smsk[4][ROOTS ? kStack : 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int64_t gw = (int64_t)blockIdx.x * nw + w;
  int32_t* stk = gstack ? gstack + gw * 2 * stack_len : sstk[w];
  unsigned* msk = gstack && ROOTS
                      ? reinterpret_cast<unsigned*>(gstack + gw * 2 * stack_len + stack_len)
                      : smsk[w];
  const int64_t nq = nq_dev ? (int64_t)*nq_dev : nq_max;
  if (gw * 32 >= nq) return;  // whole warp past the (device-side) query count
  int64_t slot = gw * 32 + lane;
  bool valid = slot < nq;
  int64_t qi = valid ? (order ? (int64_t)order[slot] : slot) : 0;
  double q[D];
#pragma unroll
  for (int j = 0; j < D; ++j) q[j] = valid ? Q[qi * D + j] : 0.0;
  double rr = valid ? r2 : -1.0;
  int64_t cnt = 0;
  int64_t cur = (FILL && valid) ? offsets[qi] : 0;
  const int64_t cur_end = (FILL && valid) ? offsets[qi + 1] : 0;
  int32_t cov_lo = 0, cov_hi = 0;  // point range already counted whole (count pass)
  int visited = 0;
  int top = 0;
  if (ROOTS) {
    const int32_t root = valid ? qroot[qi] : -1;
    const unsigned grp = __match_any_sync(0xffffffffu, root);
    const bool leader = valid && lane == __ffs(grp) - 1;
    const unsigned leaders = __ballot_sync(0xffffffffu, leader);
    if (leader) {
      const int e = __popc(leaders & ((1u << lane) - 1u));
      stk[e] = root;
      msk[e] = grp;
    }
    top = __popc(leaders) - 1;
  } else if (lane == 0) {
    stk[0] = 0;
  }
  __syncwarp();
  while (top >= 0) {
    int32_t node = stk[top];
    const unsigned em = ROOTS ? msk[top] : 0xffffffffu;
    --top;
    __syncwarp();
    if (heavy && ++visited > budget) {  // left to the warp kernel, which starts again
      const unsigned vm = __ballot_sync(0xffffffffu, valid);
      unsigned base = 0;
      if (lane == 0) base = atomicAdd(n_heavy, (unsigned)__popc(vm));
      base = __shfl_sync(0xffffffffu, base, 0);
      if (valid) heavy[base + __popc(vm & ((1u << lane) - 1u))] = (int32_t)qi;
      return;
    }
    NodeMeta m = load_meta(tv.meta, node);
    bool need = ((em >> lane) & 1u) && box_mind2<D, PER>(tv, q, node) <= rr;
    if (!FILL && need && m.start >= cov_lo && m.start < cov_hi) need = false;
    if (!FILL && need && m.left >= 0 &&
        (PER ? box_maxd2_near<D>(tv, q, node) : box_maxd2<D>(tv, q, node)) <= rr) {
      cnt += m.count;  // whole subtree inside the ball
      cov_lo = m.start;
      cov_hi = m.start + m.count;
      need = false;
    }
    unsigned nm = __ballot_sync(0xffffffffu, need);
    if (nm == 0) continue;
    if (m.left < 0) {
      for (int i = 0; i < m.count; ++i) {
        int32_t p = m.start + i;
        double d2 = point_d2<D, PER>(tv, q, p);
        if (need && d2 <= rr) {
          if (FILL) {
            if (cur >= cur_end) continue;  // the row is full (count and fill always agree)
            oidx[cur] = __ldg(&tv.ids[p]);
            odist[cur] = want_d2 ? d2 : sqrt(d2);
            ++cur;
          } else {
            ++cnt;
          }
        }
      }
    } else {
      if (lane == 0) {
        stk[top + 1] = m.left + 1;
        stk[top + 2] = m.left;
        if (ROOTS) {
          msk[top + 1] = nm;
          msk[top + 2] = nm;
        }
      }
      top += 2;
      __syncwarp();
    }
  }
  if (!FILL && valid) counts[qi] = cnt;
}

__device__ __forceinline__ bool key_lt(double d1, int64_t i1, double d2, int64_t i2) {
  return d1 < d2 || (d1 == d2 && i1 < i2);
}

// Per-row sort by (d2, id) of the fill output (d2 stored in dist), then sqrt.
// Rows of at most 32 results: insertion sort by their own thread.  Longer rows
// are listed for k_sort_big (a block per row), with a scratch range for the
// rows longer than one shared-memory tile.
constexpr int kSortTile = 2048;
__global__ void k_sort_rows(const int64_t* __restrict__ offsets, int64_t nq,
                            int64_t* __restrict__ idx, double* __restrict__ dist,
                            int32_t* __restrict__ big, unsigned long long* __restrict__ sel,
                            int64_t* __restrict__ tmp_off) {
  int64_t qi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (qi >= nq) return;
  int64_t b = offsets[qi], e = offsets[qi + 1], n = e - b;
  if (n > 32) {
    const unsigned long long slot = atomicAdd(&sel[0], 1ull);
    big[slot] = (int32_t)qi;
    tmp_off[slot] = n > kSortTile ? (int64_t)atomicAdd(&sel[1], (unsigned long long)n) : 0;
    return;
  }
  double* D2 = dist + b;
  int64_t* I = idx + b;
  for (int64_t i = 1; i < n; ++i) {
    double d = D2[i];
    int64_t x = I[i];
    int64_t j = i - 1;
    while (j >= 0 && key_lt(d, x, D2[j], I[j])) {
      D2[j + 1] = D2[j];
      I[j + 1] = I[j];
      --j;
    }
    D2[j + 1] = d;
    I[j + 1] = x;
  }
  for (int64_t i = 0; i < n; ++i) D2[i] = sqrt(D2[i]);
}

// A block per listed row: tiles of kSortTile sorted in shared memory (bitonic),
// then merge passes of doubling width between the row and its scratch range
// (merge path: each thread finds where its 8 outputs start by binary search).
// Keys (d2, id) are distinct within a row, so the order is total.
__global__ void __launch_bounds__(256) k_sort_big(const int64_t* __restrict__ offsets,
                                                  const int32_t* __restrict__ big,
                                                  const unsigned long long* __restrict__ sel,
                                                  const int64_t* __restrict__ tmp_off,
                                                  int64_t* __restrict__ idx,
                                                  double* __restrict__ dist,
                                                  int64_t* __restrict__ tidx,
                                                  double* __restrict__ tdist) {
  __shared__ double sk[kSortTile];
  __shared__ int64_t si[kSortTile];
  const int tid = threadIdx.x, nt = blockDim.x;
  const int64_t nbig = (int64_t)sel[0];
  for (int64_t r = blockIdx.x; r < nbig; r += gridDim.x) {
    const int32_t qi = big[r];
    const int64_t b = offsets[qi], n = offsets[qi + 1] - b;
    double* D2 = dist + b;
    int64_t* I = idx + b;
    for (int64_t t0 = 0; t0 < n; t0 += kSortTile) {
      const int m = (int)min((int64_t)kSortTile, n - t0);
      int P = 1;
      while (P < m) P <<= 1;
      for (int i = tid; i < P; i += nt) {
        sk[i] = i < m ? D2[t0 + i] : INFINITY;
        si[i] = i < m ? I[t0 + i] : INT64_MAX;
      }
      __syncthreads();
      for (int k = 2; k <= P; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
          for (int i = tid; i < P; i += nt) {
            const int ixj = i ^ j;
            if (ixj > i) {
              const bool up = (i & k) == 0;
              if (key_lt(sk[ixj], si[ixj], sk[i], si[i]) == up) {
                const double td = sk[i];
                const int64_t ti = si[i];
                sk[i] = sk[ixj];
                si[i] = si[ixj];
                sk[ixj] = td;
                si[ixj] = ti;
              }
            }
          }
          __syncthreads();
        }
      for (int i = tid; i < m; i += nt) {
        D2[t0 + i] = sk[i];
        I[t0 + i] = si[i];
      }
      __syncthreads();
    }
    if (n > kSortTile) {
      double* sD = D2;
      int64_t* sI = I;
      double* dD = tdist + tmp_off[r];
      int64_t* dI = tidx + tmp_off[r];
      for (int64_t w = kSortTile; w < n; w <<= 1) {
        for (int64_t s0 = 0; s0 < n; s0 += 2 * w) {
          const int64_t na = min(w, n - s0);
          const int64_t nb = max((int64_t)0, min(w, n - s0 - w));
          const double* AD = sD + s0;
          const int64_t* AI = sI + s0;
          const double* BD = AD + na;
          const int64_t* BI = AI + na;
          const int64_t mt = na + nb;
          for (int64_t k0 = (int64_t)tid * 8; k0 < mt; k0 += (int64_t)nt * 8) {
            int64_t lo = max((int64_t)0, k0 - nb), hi = min(k0, na);
            while (lo < hi) {
              const int64_t mid = (lo + hi) >> 1;
              if (key_lt(AD[mid], AI[mid], BD[k0 - 1 - mid], BI[k0 - 1 - mid])) lo = mid + 1;
              else hi = mid;
            }
            int64_t i = lo, j = k0 - lo;
            const int64_t kend = min(k0 + 8, mt);
            for (int64_t k = k0; k < kend; ++k) {
              const bool ta = j >= nb || (i < na && key_lt(AD[i], AI[i], BD[j], BI[j]));
              if (ta) {
                dD[s0 + k] = AD[i];
                dI[s0 + k] = AI[i];
                ++i;
              } else {
                dD[s0 + k] = BD[j];
                dI[s0 + k] = BI[j];
                ++j;
              }
            }
          }
        }
        __syncthreads();
        double* tD = sD;
        sD = dD;
        dD = tD;
        int64_t* tI = sI;
        sI = dI;
        dI = tI;
      }
      if (sD != D2)
        for (int64_t i = tid; i < n; i += nt) {
          D2[i] = sD[i];
          I[i] = sI[i];
        }
      __syncthreads();
    }
    for (int64_t i = tid; i < n; i += nt) D2[i] = sqrt(D2[i]);
    __syncthreads();
  }
}

// ---------------------------------------------------------- heavy ball rows
// Rows with at least kHeavyRow results are filled by a whole warp per query:
// one warp-uniform left-first DFS (stack in shared memory), leaves scanned with
// the lanes over the points (FP64 distances, results compacted in point order by
// ballot prefix), and subtrees whose tight box lies entirely inside the ball
// (box_maxd2 / box_maxd2_near <= r^2) emitted in one coalesced pass over their
// contiguous positions.  The order of a row is the per-lane kernel's: left-first
// DFS, leaf order.
constexpr int64_t kHeavyRow = 256;
constexpr int kHeavyStack = 128;

// A whole subtree of at least kTaskMin points inside a heavy row's ball is not
// copied by the warp that found it but recorded as emission tasks of at most
// kTaskChunk points, which k_ball_emit spreads over the whole GPU: a row of
// millions of points no longer serialises on one warp.  When the task buffer is
// full the warp copies the subtree itself (same output).
constexpr int32_t kTaskMin = 1024;
constexpr int32_t kTaskChunk = 4096;
constexpr unsigned kTaskCap = 1u << 20;  // at most: 64 a query, at least 2^16
struct EmitTask {
  int64_t out;  // first output slot
  int32_t start, count, qi, pad;
};

template <int D, bool PER>
__global__ void __launch_bounds__(128) k_ball_fill_warp(TreeView tv, const double* __restrict__ Q,
                                                        const int32_t* __restrict__ rows,
                                                        const unsigned* __restrict__ n_rows,
                                                        double r2, int32_t* __restrict__ gstack,
                                                        int stack_len,
                                                        const int64_t* __restrict__ offsets,
                                                        int64_t* __restrict__ oidx,
                                                        double* __restrict__ odist, int want_d2,
                                                        EmitTask* __restrict__ tasks,
                                                        unsigned* __restrict__ n_tasks,
                                                        unsigned task_cap,
                                                        const int32_t* __restrict__ qroot) {
  __shared__ int32_t sstk[4][kHeavyStack];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  const int64_t nrows = (int64_t)*n_rows;
  for (int64_t r = (int64_t)blockIdx.x * nw + w; r < nrows; r += (int64_t)gridDim.x * nw) {
    int32_t* stk = gstack ? gstack + ((int64_t)blockIdx.x * nw + w) * stack_len : sstk[w];
    const int64_t qi = rows[r];
    double q[D];
#pragma unroll
    for (int j = 0; j < D; ++j) q[j] = Q[qi * D + j];
    int64_t cur = offsets[qi];
    const int64_t cur_end = offsets[qi + 1];
    int top = 0;
    if (lane == 0) stk[0] = qroot ? qroot[qi] : 0;
    __syncwarp();
    while (top >= 0) {
      const int32_t node = stk[top];
      --top;
      __syncwarp();
      const NodeMeta m = load_meta(tv.meta, node);
      if (!(box_mind2<D, PER>(tv, q, node) <= r2)) continue;
      const bool inside =
          m.left >= 0 && (PER ? box_maxd2_near<D>(tv, q, node) : box_maxd2<D>(tv, q, node)) <= r2;
      if (inside && tasks && m.count >= kTaskMin && cur < cur_end) {
        const int64_t len = min((int64_t)m.count, cur_end - cur);
        const unsigned nt = (unsigned)((len + kTaskChunk - 1) / kTaskChunk);
        unsigned tb = 0;
        if (lane == 0) tb = atomicAdd(n_tasks, nt);
        tb = __shfl_sync(0xffffffffu, tb, 0);
        if (tb + nt <= task_cap) {
          for (unsigned c = lane; c < nt; c += 32) {
            EmitTask e;
            e.out = cur + (int64_t)c * kTaskChunk;
            e.start = m.start + (int32_t)c * kTaskChunk;
            e.count = (int32_t)min((int64_t)kTaskChunk, len - (int64_t)c * kTaskChunk);
            e.qi = (int32_t)qi;
            e.pad = 0;
            tasks[tb + c] = e;
          }
          cur += m.count;
          continue;
        }
        // the buffer is full: the slots left in it hold no work
        for (unsigned c = lane; c < nt && tb + c < task_cap; c += 32) tasks[tb + c] = EmitTask{};
      }
      if (inside) {  // whole subtree: positions m.start .. m.start + count - 1 in order
        for (int32_t i = lane; i < m.count; i += 32) {
          const int32_t p = m.start + i;
          const int64_t o = cur + i;
          if (o < cur_end) {
            const double d2 = point_d2<D, PER>(tv, q, p);
            oidx[o] = __ldg(&tv.ids[p]);
            odist[o] = want_d2 ? d2 : sqrt(d2);
          }
        }
        cur += m.count;
      } else if (m.left < 0) {
        for (int32_t base = 0; base < m.count; base += 32) {
          const int32_t i = base + lane;
          bool hit = false;
          double d2 = 0.0;
          if (i < m.count) {
            d2 = point_d2<D, PER>(tv, q, m.start + i);
            hit = d2 <= r2;
          }
          const unsigned hm = __ballot_sync(0xffffffffu, hit);
          if (hit) {
            const int64_t o = cur + __popc(hm & lt_mask);
            if (o < cur_end) {
              oidx[o] = __ldg(&tv.ids[m.start + i]);
              odist[o] = want_d2 ? d2 : sqrt(d2);
            }
          }
          cur += __popc(hm);
        }
      } else {
        if (lane == 0) {
          stk[top + 1] = m.left + 1;
          stk[top + 2] = m.left;
        }
        top += 2;
        __syncwarp();
      }
    }
    __syncwarp();
  }
}

// Copies of the recorded whole-subtree chunks, a warp per chunk.
template <int D, bool PER>
__global__ void __launch_bounds__(128) k_ball_emit(TreeView tv, const double* __restrict__ Q,
                                                   const EmitTask* __restrict__ tasks,
                                                   const unsigned* __restrict__ n_tasks,
                                                   unsigned task_cap,
                                                   int64_t* __restrict__ oidx,
                                                   double* __restrict__ odist, int want_d2) {
  const int lane = threadIdx.x & 31;
  const int64_t nt = min((int64_t)*n_tasks, (int64_t)task_cap);
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < nt;
       t += nwarps) {
    const EmitTask e = tasks[t];
    double q[D];
#pragma unroll
    for (int j = 0; j < D; ++j) q[j] = Q[(int64_t)e.qi * D + j];
#pragma unroll 4
    for (int32_t i = lane; i < e.count; i += 32) {
      const int32_t p = e.start + i;
      const double d2 = point_d2<D, PER>(tv, q, p);
      oidx[e.out + i] = __ldg(&tv.ids[p]);
      odist[e.out + i] = want_d2 ? d2 : sqrt(d2);
    }
  }
}

// ------------------------------------------------------- ball, FP32 node tests
// One query's ball against FP32 boxes.  The tests only decide what is surely
// outside (pruned) or surely inside (taken whole); every other point is tested in FP64 with the reference arithmetic, so results are exact.  Query
// coordinates beyond the FP32 range are clamped: the gaps of the clamped query
// never exceed the true ones (tree coordinates are below 1e18 here), and such a
// query takes nothing whole.
template <int D, bool PER>
struct BallQuery {
  static constexpr int kD = D;
  static constexpr int NV = (D + 3) / 4;
  static constexpr bool kDist = true;
  const TreeView& tv;
  double q[D];
  double rr;
  QueryScreen<D, PER> qs;
  float xl[D], xh[D];
  float r2u, r2d;  // r^2 rounded up / down
  bool wf;              // the ball cannot reach the periodic faces
  bool whole_ok;

  __device__ __forceinline__ BallQuery(const TreeView& t, const double* __restrict__ Q, int64_t qi,
                                       double r2)
      : tv(t), rr(r2) {
    whole_ok = true;
    r2u = __double2float_ru(r2);
    r2d = __double2float_rd(r2);
    const float r32 = sqrt_up(r2u);
    wf = true;
#pragma unroll
    for (int j = 0; j < D; ++j) {
      q[j] = Q[qi * D + j];
      const float x = __double2float_rn(q[j]);
      whole_ok = whole_ok && fabsf(x) < 1e18f;
      qs.q32[j] = fminf(fmaxf(x, -2e18f), 2e18f);
      qs.dlt[j] = kTwoM21 * (fabsf(qs.q32[j]) + tv.slack[j]) * 1.0001f;
      xl[j] = __fadd_ru(qs.q32[j], qs.dlt[j]);
      xh[j] = __fsub_rd(qs.q32[j], qs.dlt[j]);
      if (PER)
        wf = wf && __fadd_ru(__fadd_ru(fabsf(qs.q32[j]), r32), qs.dlt[j]) < 0.5f * (float)tv.L[j];
    }
  }
  // lower bound of the squared distance to any point of the box
  __device__ __forceinline__ float lb(const float (&lo)[4 * NV], const float (&hi)[4 * NV]) const {
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
  }
  // whether every point of the box is surely within r: the direct differences,
  // rounded up, bound every point's (the minimum image is the direct difference
  // when that is at most half a side)
  __device__ __forceinline__ bool holds(const float (&lo)[4 * NV], const float (&hi)[4 * NV]) const {
    float s2 = 0.0f;
    bool ok = whole_ok;
#pragma unroll
    for (int j = 0; j < D; ++j) {
      const float g = fmaxf(__fsub_ru(xl[j], lo[j]), __fsub_ru(hi[j], xh[j]));
      if (PER) ok = ok && g <= 0.4999999f * (float)tv.L[j];
      s2 = __fmaf_ru(g, g, s2);
    }
    return ok && __fmul_ru(s2, 1.000002f) <= r2d;
  }
  __device__ __forceinline__ bool reaches(const float (&lo)[4 * NV],
                                          const float (&hi)[4 * NV]) const {
    return lb(lo, hi) <= r2u;
  }
  __device__ __forceinline__ bool hit(int32_t p, bool whole, double& d2) const {
    d2 = point_d2_rec<D, PER>(tv, q, p);
    return whole || d2 <= rr;
  }
  __device__ __forceinline__ void resume(int32_t) {}
  // The subtree that holds the ball, from a root: while the split plane is further
  // than r from the query, only its side of it can hold results.  The points left
  // of a split lie at or below it, those on the right at or above it, and rounding
  // is monotone, so a point on the far side has a computed squared distance of at
  // least (split - q)^2, computed the same way.  Not for balls that may reach a
  // periodic face.
  __device__ __forceinline__ int2 root(int32_t node, int32_t unit) {
    NodeMeta m = load_meta(tv.meta, node);
    while (m.left >= 0 && m.count > unit && (!PER || wf)) {
      double qa = 0.0;
#pragma unroll
      for (int j = 0; j < D; ++j)
        if (j == m.axis) qa = q[j];
      const double g = dsub(m.split, qa);
      if (!(dmul(g, g) > rr)) break;
      node = g > 0.0 ? m.left : m.left + 1;
      m = load_meta(tv.meta, node);
    }
    return m.left < 0 || m.count <= unit ? make_int2(m.start, m.count) : make_int2(node, 0);
  }
};

// -------------------------------------------------------- box, FP32 node tests
// One query box against the tree.  What the reference returns is the points of the
// closed box that its strict descent reaches (left iff lo < split, right iff
// hi > split, :1296-1300).  The points left of a split lie at or below it and those
// on the right at or above it, so a point strictly inside the box is reached at
// every split above it: subtrees whose tight box lies strictly inside are taken
// whole, subtrees whose tight box misses the closed box hold nothing, and only a
// point on a face of the box needs its path checked (also what a NaN bound leaves).
template <int D>
struct BoxQuery {
  static constexpr int kD = D;
  static constexpr int NV = (D + 3) / 4;
  static constexpr bool kDist = false;
  const TreeView& tv;
  double lo[D], hi[D];
  float lod[D], lou[D], hid[D], hiu[D];  // the bounds rounded down / up
  int32_t top;                           // node that the root descent reached

  __device__ __forceinline__ BoxQuery(const TreeView& t, const double* __restrict__ boxes,
                                      int64_t bi, double)
      : tv(t) {
#pragma unroll
    for (int j = 0; j < D; ++j) {
      lo[j] = boxes[bi * 2 * D + 2 * j];
      hi[j] = boxes[bi * 2 * D + 2 * j + 1];
      lod[j] = __double2float_rd(lo[j]);
      lou[j] = __double2float_ru(lo[j]);
      hid[j] = __double2float_rd(hi[j]);
      hiu[j] = __double2float_ru(hi[j]);
    }
  }
  __device__ __forceinline__ bool reaches(const float (&blo)[4 * NV],
                                          const float (&bhi)[4 * NV]) const {
    bool out = false;
#pragma unroll
    for (int j = 0; j < D; ++j) out = out || bhi[j] < lod[j] || blo[j] > hiu[j];
    return !out;
  }
  __device__ __forceinline__ bool holds(const float (&blo)[4 * NV],
                                        const float (&bhi)[4 * NV]) const {
    bool in = true;
#pragma unroll
    for (int j = 0; j < D; ++j) in = in && lou[j] < blo[j] && bhi[j] < hid[j];
    return in;
  }
  // which sides of a node's split the strict descent visits (:1296, :1300)
  __device__ __forceinline__ void sides(const NodeMeta& m, bool& gl, bool& gr) const {
    double bl = 0.0, bh = 0.0;
#pragma unroll
    for (int j = 0; j < D; ++j)
      if (j == m.axis) {
        bl = lo[j];
        bh = hi[j];
      }
    gl = bl < m.split;
    gr = bh > m.split;
  }
  // for entries of an earlier walk: paths are checked from the root
  __device__ __forceinline__ void resume(int32_t node) { top = node; }
  __device__ __forceinline__ int2 root(int32_t node, int32_t unit) {
    NodeMeta m = load_meta(tv.meta, node);
    while (m.left >= 0 && m.count > unit) {
      bool gl, gr;
      sides(m, gl, gr);
      if (!gl && !gr) return make_int2(0, INT32_MIN);
      if (gl && gr) break;
      node = gl ? m.left : m.left + 1;
      m = load_meta(tv.meta, node);
    }
    top = node;
    return m.left < 0 || m.count <= unit ? make_int2(m.start, m.count) : make_int2(node, 0);
  }
  __device__ __forceinline__ bool hit(int32_t p, bool whole, double&) const {
    if (whole) return true;
    double v[4 * NV];
#pragma unroll
    for (int h = 0; h < NV; ++h) {
      const double2* r = reinterpret_cast<const double2*>(tv.pts64 + (int64_t)p * NV + h);
      const double2 a = CKD_LDT(r), b = CKD_LDT(r + 1);
      v[4 * h] = a.x;
      v[4 * h + 1] = a.y;
      v[4 * h + 2] = b.x;
      v[4 * h + 3] = b.y;
    }
    bool in = true, inner = true;
#pragma unroll
    for (int j = 0; j < D; ++j) {
      in = in && !(v[j] < lo[j] || v[j] > hi[j]);  // :1319
      inner = inner && lo[j] < v[j] && v[j] < hi[j];
    }
    if (!in || inner) return in;
    // on a face: reached iff every split on its path is passed on its side
    NodeMeta m = load_meta(tv.meta, top);
    while (m.left >= 0) {
      bool gl, gr;
      sides(m, gl, gr);
      const NodeMeta l = load_meta(tv.meta, m.left);
      if (p < l.start + l.count) {
        if (!gl) return false;
        m = l;
      } else {
        if (!gr) return false;
        m = load_meta(tv.meta, m.left + 1);
      }
    }
    return true;
  }
};

// Children of an internal node that the query reaches, as entries {node, 0},
// {start, count} (to be tested point by point) or {start, -count} (whole);
// y == kNone: not reached.  Subtrees of at most `unit` points come as ranges.
constexpr int32_t kNone = INT32_MIN;
template <class QT>
__device__ __forceinline__ void expand(const QT& qt, int32_t node, int32_t unit, int2& a, int2& b) {
  constexpr int NV = QT::NV;
  const float4* rec = qt.tv.pair + (int64_t)node * pair_f4(QT::kD);
  float v[4][4 * NV];
#pragma unroll
  for (int s = 0; s < 4; ++s)
#pragma unroll
    for (int h = 0; h < NV; ++h) {
      const float4 f = CKD_LDT(rec + s * NV + h);
      v[s][4 * h] = f.x;
      v[s][4 * h + 1] = f.y;
      v[s][4 * h + 2] = f.z;
      v[s][4 * h + 3] = f.w;
    }
  const int4 info = CKD_LDT(reinterpret_cast<const int4*>(rec + 4 * NV));
  const int4 range = CKD_LDT(reinterpret_cast<const int4*>(rec + 4 * NV + 1));
  const bool ra = info.z || range.y <= unit, rb = info.w || range.w <= unit;
  a = make_int2(ra ? range.x : info.x, ra ? range.y : 0);
  b = make_int2(rb ? range.z : info.y, rb ? range.w : 0);
  if (!qt.reaches(v[0], v[1])) a.y = kNone;
  else if (qt.holds(v[0], v[1])) a = make_int2(range.x, -range.y);
  if (!qt.reaches(v[2], v[3])) b.y = kNone;
  else if (qt.holds(v[2], v[3])) b = make_int2(range.z, -range.w);
}

// ------------------------------------------------- ball and box, warp per query
// The warp keeps a stack of entries (expand) in depth-first order, the
// next one on top.  Up to 32 entries are taken at once, a lane each: nodes are
// replaced by their reached children (left on top), so the children of many nodes
// are tested in parallel.
//   count: ranges never enter the stack; whole ones are added up, the others listed
//     and scanned over the lanes when enough wait;
//   fill: the ranges above the topmost node are next in the row: they are emitted
//     in order, flattened over the lanes, the others stay where they are.  A whole
//     range of kTaskMin points on becomes emission tasks, which k_ball_emit spreads
//     over the GPU.
// A row is in leaf order, the order of the packet kernel and of k_ball_fill_warp.
// The packet kernel walks the union of 32 balls with FP64 box tests, which is what
// it was bound by; 4001 scattered queries on 2^22 clustered points, 20000 results
// each: count 32.2 -> 0.45 ms, fill 8.8 -> 1.85 ms; 10^5 on 2^20 uniform points, 5
// results each: 0.39 -> 0.26 and 0.44 -> 0.28 ms.  Now bound by issue: about 3000
// warp instructions a query of the latter.  A lane per query (tried for small
// balls, 100k queries) was no faster, waiting on its dependent loads.
constexpr int kBallStack = 384;
constexpr int kBallReserve = 130;  // room for one-at-a-time descents (tree depth < 127)
constexpr int kBallWide = 190;     // entries up to which several are expanded at once
constexpr int kBallList = 128;
constexpr int kBallListRun = 16;   // ranges that wait before they are scanned (count)
constexpr int32_t kBallUnit = 32;  // subtrees of at most this many points are scanned as a range
constexpr int32_t kBallRoot = 64;  // and of this many where the descent from the root ends

// What the fill's walk leaves of a long row: its pending entries, in order and refined
// by breadth-first levels, as parts. A second launch counts their results, a third
// writes each part behind those before it, a warp per part.  One warp walked the row
// alone before, and the longest rows were all that ran at the end of a pass (10 % of
// the warps active): 4001 balls of 20000 results on 2^22 clustered points, fill 0.93 ->
// 0.67 ms with the recount; 12800 boxes on 200 trees 2.26 -> 0.99.  A budget of 32 or 128
// steps and 64 entries are within 10 %.  The count pass, which has nothing to tell long
// rows by, walks them whole; parts shared by the warps of a block only were up to 1.5
// times slower than whole rows.
struct Part {
  int64_t base;    // where the row's first part begins
  int32_t head;    // the row's first part
  int32_t qi;      // -1: none
  int32_t x, y;    // the entry
  int32_t count;   // its results
  int32_t pad;
};
constexpr int kPartMin = 128;     // entries that a row is refined to, at least, where it can be
// A level at most doubles the entries, and a row that finds no room for its parts is
// walked on from what it was refined to: one-at-a-time descents still have their room.
// (96 entries and a stack of 320: 4001 clustered balls 1249 -> 1293 us a call.)
static_assert(kBallWide + kBallReserve <= kBallStack &&
              2 * (kPartMin - 1) + kBallReserve <= kBallStack, "walks and refined rows fit");
constexpr int kPartBudget = 64;   // steps (32 lanes' work each) before a row is cut
struct Parts {
  Part* list;       // null: rows are not cut
  unsigned* n;
  unsigned cap;
  bool run;         // the rows of this launch are parts
};

// The row's pending entries made parts; false when they do not fit.
template <class QT>
__device__ __forceinline__ bool cut_row(const QT& bq, const Parts& parts, int64_t qi, int64_t cur,
                                       int2*& stk, int2* tmp, int& top) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  if (!parts.list || parts.run) return false;
  // read by one lane: other warps add to it, and the warp has to agree
  unsigned used = 0;
  if (lane == 0) used = *(volatile unsigned*)parts.n;
  if (__shfl_sync(FULL, used, 0) >= parts.cap) return false;
  bool more = true;
  while (more && top < kPartMin) {
    int m = 0;
    more = false;
#pragma unroll 1
    for (int u0 = 0; u0 < top; u0 += 32) {
      int2 a = make_int2(0, kNone), b = make_int2(0, kNone);
      const int2 e = u0 + lane < top ? stk[u0 + lane] : make_int2(0, kNone);
      if (e.y == 0) expand(bq, e.x, kBallUnit, a, b);
      else a = e;
      const unsigned ma = __ballot_sync(FULL, a.y != kNone);
      const unsigned mb = __ballot_sync(FULL, b.y != kNone);
      const int o = m + __popc(ma & lt) + __popc(mb & lt);  // right below left
      if (b.y != kNone) tmp[o] = b;
      if (a.y != kNone) tmp[o + (b.y != kNone ? 1 : 0)] = a;
      m += __popc(ma) + __popc(mb);
      more = more || __any_sync(FULL, a.y == 0 || b.y == 0);
    }
    __syncwarp();
    int2* const t = stk;
    stk = tmp;
    tmp = t;
    top = m;
  }
  if (top == 0) return true;
  unsigned pb = 0;
  if (lane == 0) pb = atomicAdd(parts.n, (unsigned)top);
  pb = __shfl_sync(FULL, pb, 0);
  const bool fits = pb + (unsigned)top <= parts.cap;
  for (int i = lane; i < top && pb + i < parts.cap; i += 32) {
    Part p;
    p.base = cur;
    p.head = (int32_t)pb;
    p.qi = fits ? (int32_t)qi : -1;
    p.x = stk[top - 1 - i].x;
    p.y = stk[top - 1 - i].y;
    p.count = 0;
    p.pad = 0;
    parts.list[pb + i] = p;
  }
  __syncwarp();
  return fits;
}

template <class QT, bool FILL>
__global__ void __launch_bounds__(128) k_range_warp(
    TreeView tv, const double* __restrict__ Q, const int32_t* __restrict__ order, int64_t nq,
    double r2, int64_t* __restrict__ counts,
    const int64_t* __restrict__ offsets, int64_t* __restrict__ oidx, double* __restrict__ odist,
    int want_d2, EmitTask* __restrict__ tasks, unsigned* __restrict__ n_tasks, unsigned task_cap,
    const int32_t* __restrict__ qroot, const unsigned* __restrict__ n_rows = nullptr,
    const Parts parts = Parts{}) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ int2 s_stk[4][FILL ? 2 : 1][kBallStack];
  __shared__ int2 s_list[4][FILL ? 1 : kBallList];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  int2* stk = s_stk[w][0];
  int2* list = s_list[w];
  const int64_t nr = parts.run ? (int64_t)min(*parts.n, parts.cap) : n_rows ? (int64_t)*n_rows : nq;
  for (int64_t r = (int64_t)blockIdx.x * 4 + w; r < nr; r += (int64_t)gridDim.x * 4) {
    int64_t qi, cur = 0, cur_end = 0;
    int2 first;
    if (parts.run) {
      const Part p = parts.list[r];
      qi = p.qi;
      if (qi < 0) continue;
      first = make_int2(p.x, p.y);
      if (FILL) {
        for (int64_t i = p.head + lane; i < r; i += 32) cur += parts.list[i].count;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) cur += __shfl_xor_sync(FULL, cur, o);
        cur += p.base;
        // no further than the row, whose length is the caller's
        cur_end = min(cur + p.count, offsets[qi + 1]);
      }
    } else {
      qi = order ? (int64_t)order[r] : r;
      if (FILL) {
        cur = offsets[qi];
        cur_end = offsets[qi + 1];
      }
    }
    if (FILL && cur >= cur_end) continue;
    QT bq(tv, Q, qi, r2);
    int64_t cnt = 0;  // per lane
    int top = 1, nl = 0, work = 0;
    if (parts.run) bq.resume(qroot ? qroot[qi] : 0);
    else first = bq.root(qroot ? qroot[qi] : 0, kBallRoot);
    if (first.y == kNone) top = 0;
    if (lane == 0) stk[0] = first;
    __syncwarp();
    while (top > 0) {
      if (FILL && cur >= cur_end) break;  // all of the row's results are found
      if (FILL && ++work > kPartBudget) {
        work = 0;
        if (cut_row(bq, parts, qi, cur, stk, s_stk[w][stk == s_stk[w][0] ? 1 : 0], top)) break;
      }
      const int n = min(min(top, 32), max(1, kBallWide - top));
      int2 e = make_int2(0, kNone);
      if (lane < n) e = stk[top - 1 - lane];
      __syncwarp();
      top -= n;
      // lanes below `lead` hold the ranges that come next (fill)
      int lead = 0;
      if (FILL) {
        const unsigned nm = __ballot_sync(FULL, lane >= n || e.y == 0);
        lead = nm ? __ffs(nm) - 1 : 32;
        const unsigned big = __ballot_sync(FULL, lane < lead && e.y <= -kTaskMin);
        if (big & 1u) lead = 1;
        else if (big) lead = __ffs(big) - 1;
      }
      int2 a = make_int2(0, kNone), b = make_int2(0, kNone);
      if (lane < n && lane >= lead) {
        if (e.y == 0) expand(bq, e.x, kBallUnit, a, b);
        else a = e;
      }
      if (!FILL) {
        if (a.y < 0 && a.y != kNone) {
          cnt -= a.y;
          a.y = kNone;
        }
        if (b.y < 0 && b.y != kNone) {
          cnt -= b.y;
          b.y = kNone;
        }
        const unsigned ga = __ballot_sync(FULL, a.y > 0), gb = __ballot_sync(FULL, b.y > 0);
        const int o = nl + __popc(ga & lt) + __popc(gb & lt);
        if (a.y > 0) list[o] = a;
        if (b.y > 0) list[o + (a.y > 0 ? 1 : 0)] = b;
        nl += __popc(ga) + __popc(gb);
        if (a.y > 0) a.y = kNone;
        if (b.y > 0) b.y = kNone;
      }
      // back onto the stack, the first lane's entries on top, left above right
      const unsigned ma = __ballot_sync(FULL, a.y != kNone);
      const unsigned mb = __ballot_sync(FULL, b.y != kNone);
      const int total = __popc(ma) + __popc(mb);
      const int above = __popc(ma & lt) + __popc(mb & lt);
      if (a.y != kNone) stk[top + total - 1 - above] = a;
      if (b.y != kNone) stk[top + total - 1 - above - (a.y != kNone ? 1 : 0)] = b;
      top += total;
      __syncwarp();
      if (!FILL) {
        if (nl < kBallListRun && top > 0) continue;
#pragma unroll 1
        for (int u0 = 0; u0 < nl; u0 += 32) {
          const int2 x = u0 + lane < nl ? list[u0 + lane] : make_int2(0, 0);
          int32_t inc = x.y;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int32_t v = __shfl_up_sync(FULL, inc, o);
            if (lane >= o) inc += v;
          }
          const int32_t tot = __shfl_sync(FULL, inc, 31);
          const int32_t delta = x.x - (inc - x.y);
#pragma unroll 2
          for (int32_t t = lane; t - lane < tot; t += 32) {
            int j = 0;  // the range holding t: the first with inc > t
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
              const int32_t v = __shfl_sync(FULL, inc, j + o - 1);
              if (v <= t) j += o;
            }
            const int32_t p = __shfl_sync(FULL, delta, j) + t;
            double d2;
            if (t < tot && bq.hit(p, false, d2)) ++cnt;
          }
        }
        nl = 0;
        __syncwarp();
      } else if (lead > 0) {
        if (lead == 1) {  // a large whole range: tasks, unless their buffer is full
          const int32_t st = __shfl_sync(FULL, e.x, 0), ct = -__shfl_sync(FULL, e.y, 0);
          if (tasks && ct >= kTaskMin && cur < cur_end) {
            const int64_t len = min((int64_t)ct, cur_end - cur);
            const unsigned nt = (unsigned)((len + kTaskChunk - 1) / kTaskChunk);
            unsigned tb = 0;
            if (lane == 0) tb = atomicAdd(n_tasks, nt);
            tb = __shfl_sync(FULL, tb, 0);
            if (tb + nt <= task_cap) {
              for (unsigned c = lane; c < nt; c += 32) {
                EmitTask x;
                x.out = cur + (int64_t)c * kTaskChunk;
                x.start = st + (int32_t)c * kTaskChunk;
                x.count = (int32_t)min((int64_t)kTaskChunk, len - (int64_t)c * kTaskChunk);
                x.qi = (int32_t)qi;
                x.pad = 0;
                tasks[tb + c] = x;
              }
              cur += ct;
              continue;
            }
            // the buffer is full: the slots left in it hold no work
            for (unsigned c = lane; c < nt && tb + c < task_cap; c += 32)
              tasks[tb + c] = EmitTask{};
          }
        }
        const int32_t ct = lane < lead ? abs(e.y) : 0;
        int32_t inc = ct;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int32_t v = __shfl_up_sync(FULL, inc, o);
          if (lane >= o) inc += v;
        }
        const int32_t tot = __shfl_sync(FULL, inc, 31);
        const int32_t delta = e.x - (inc - ct);
        const unsigned wholes = __ballot_sync(FULL, lane < lead && e.y < 0);
        work += tot >> 5;
#pragma unroll 2
        for (int32_t t = lane; t - lane < tot; t += 32) {
          int j = 0;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const int32_t v = __shfl_sync(FULL, inc, j + o - 1);
            if (v <= t) j += o;
          }
          const int32_t p = __shfl_sync(FULL, delta, j) + t;
          bool hit = t < tot;
          double d2 = 0.0;
          int32_t id = 0;
          if (hit) {
            id = CKD_LDT(&tv.ids[p]);
            hit = bq.hit(p, (wholes >> (j & 31)) & 1u, d2);
          }
          const unsigned hm = __ballot_sync(FULL, hit);
          if (hit) {
            const int64_t o = cur + __popc(hm & lt);
            if (o < cur_end) {
              oidx[o] = id;
              if (QT::kDist) odist[o] = want_d2 ? d2 : sqrt(d2);
            }
          }
          cur += __popc(hm);
        }
      }
    }
    if (!FILL) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(FULL, cnt, o);
      if (lane == 0) {
        if (parts.run) parts.list[r].count = (int32_t)cnt;
        else counts[qi] = cnt;
      }
    }
    __syncwarp();
  }
}

template <class QT>
ckd_status range_warp_count(const ckd_tree* t, const double* q, const int32_t* rows, int64_t nq,
                            const unsigned* n_rows, double r2, int64_t* counts,
                            const int32_t* qroot, int sms, cudaStream_t s) {
  const unsigned g = (unsigned)std::min<int64_t>(cdiv(nq, 4), (int64_t)sms * 16);
  k_range_warp<QT, false><<<g, 128, 0, s>>>(t->view(), q, rows, nq, r2, counts, nullptr, nullptr,
                                            nullptr, 0, nullptr, nullptr, 0, qroot, n_rows,
                                            Parts{});
  CKD_LAUNCH_CHECK();
  return CKD_OK;
}

// The fill's warps, and those of the parts when its long rows are cut (`n_parts`: a zero).
template <class QT>
ckd_status range_warp_fill(const ckd_tree* t, const double* q, const int32_t* rows, int64_t nq,
                           const unsigned* n_rows, double r2, const int64_t* offsets, int64_t* idx,
                           double* dist, int want_d2, EmitTask* tasks, unsigned* n_tasks,
                           unsigned task_cap, const int32_t* qroot, bool cut, unsigned* n_parts,
                           int sms, cudaStream_t s) {
  const TreeView tv = t->view();
  const unsigned g = (unsigned)std::min<int64_t>(cdiv(nq, 4), (int64_t)sms * 16);
  Scratch sc(s);
  Parts parts{};
  parts.n = n_parts;
  parts.cap = (unsigned)std::min<int64_t>(1 << 20, std::max<int64_t>(1 << 14, nq * 256));
  if (cut && sc.alloc(&parts.list, sizeof(Part) * parts.cap) != cudaSuccess)
    cudaGetLastError();  // without room the rows are walked whole
  k_range_warp<QT, true><<<g, 128, 0, s>>>(tv, q, rows, nq, r2, nullptr, offsets, idx, dist,
                                           want_d2, tasks, n_tasks, task_cap, qroot, n_rows, parts);
  CKD_LAUNCH_CHECK();
  if (!parts.list) return CKD_OK;
  parts.run = true;
  const unsigned gp = (unsigned)sms * 16;
  k_range_warp<QT, false><<<gp, 128, 0, s>>>(tv, q, nullptr, 0, r2, nullptr, nullptr, nullptr,
                                             nullptr, 0, nullptr, nullptr, 0, qroot, nullptr,
                                             parts);
  CKD_LAUNCH_CHECK();
  k_range_warp<QT, true><<<gp, 128, 0, s>>>(tv, q, nullptr, 0, r2, nullptr, offsets, idx, dist,
                                            want_d2, tasks, n_tasks, task_cap, qroot, nullptr,
                                            parts);
  CKD_LAUNCH_CHECK();
  return CKD_OK;
}

// ---------------------------------------------------- ball, eight lanes per query
// The same walk with G lanes of a warp per query, for large batches of small balls
// on evenly filled trees (range_narrow), where rows are of like length: short ranges
// and few pending nodes leave most lanes of a whole warp idle.  10^5 queries on 2^20
// uniform points, 5 results each: count 262 -> 160, fill 279 -> 187 us.  Boxes, whose
// sizes are known on the device only, keep the whole warp.
template <int G>
__host__ __device__ constexpr int range_stack(int depth) { return 2 * depth + 4 + 2 * G; }
template <int G>
constexpr int kRangeRun = G / 2;  // ranges that wait before they are scanned (count)

template <class QT, bool FILL, int G>
__global__ void __launch_bounds__(128) k_range_group(
    TreeView tv, const double* __restrict__ Q, const int32_t* __restrict__ order, int64_t nq,
    int depth, double r2, int64_t* __restrict__ counts, const int64_t* __restrict__ offsets,
    int64_t* __restrict__ oidx, double* __restrict__ odist, int want_d2) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int NG = 128 / G, KL = kRangeRun<G> + 2 * G;
  extern __shared__ __align__(16) unsigned char rsm[];
  const int scap = range_stack<G>(depth);
  const int lane = threadIdx.x & 31, gl = lane & (G - 1), grp = threadIdx.x / G;
  const int gsh = lane & ~(G - 1);
  constexpr unsigned gm = (1u << G) - 1u;
  const unsigned lt = (1u << gl) - 1u;
  auto ballot = [&](bool p) -> unsigned { return (__ballot_sync(FULL, p) >> gsh) & gm; };
  int2* stk = reinterpret_cast<int2*>(rsm) + (size_t)grp * scap;
  int2* list = reinterpret_cast<int2*>(rsm) + (size_t)NG * scap + grp * KL;
  const int64_t slot = (int64_t)blockIdx.x * NG + grp;
  if (slot - grp % (32 / G) >= nq) return;  // a warp without queries leaves together
  bool valid = slot < nq;
  const int64_t qi = valid ? (order ? (int64_t)order[slot] : slot) : 0;
  int64_t cur = FILL ? offsets[qi] : 0;
  const int64_t cur_end = FILL ? offsets[qi + 1] : 0;
  if (FILL && cur == cur_end) valid = false;
  QT qt(tv, Q, qi, r2);
  int64_t cnt = 0;  // per lane
  int top = 0, nl = 0;
  if (valid) {
    const int2 first = qt.root(0, kBallRoot);
    top = first.y == kNone ? 0 : 1;
    if (gl == 0) stk[0] = first;
  }
  __syncwarp();
  // the range of a group that holds flattened index t, from the lanes' inclusive counts
  auto find = [&](int32_t inc, int32_t t) -> int {
    int j = 0;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      const int32_t v = __shfl_sync(FULL, inc, j + o - 1, G);
      if (v <= t) j += o;
    }
    return j;
  };
  while (__any_sync(FULL, top > 0)) {
    const int n = min(min(top, G), max(1, depth + 2 * G - top));
    int2 e = make_int2(0, kNone);
    if (gl < n) e = stk[top - 1 - gl];
    __syncwarp();
    top -= n;
    int lead = 0;  // lanes below hold the ranges that come next (fill)
    if (FILL) {
      const unsigned nm = ballot(gl >= n || e.y == 0);
      lead = nm ? __ffs(nm) - 1 : G;
    }
    int2 a = make_int2(0, kNone), b = make_int2(0, kNone);
    if (gl < n && gl >= lead) {
      if (e.y == 0) expand(qt, e.x, kBallUnit, a, b);
      else a = e;
    }
    if (!FILL) {
      if (a.y < 0 && a.y != kNone) {
        cnt -= a.y;
        a.y = kNone;
      }
      if (b.y < 0 && b.y != kNone) {
        cnt -= b.y;
        b.y = kNone;
      }
      const unsigned ga = ballot(a.y > 0), gb = ballot(b.y > 0);
      const int o = nl + __popc(ga & lt) + __popc(gb & lt);
      if (a.y > 0) list[o] = a;
      if (b.y > 0) list[o + (a.y > 0 ? 1 : 0)] = b;
      nl += __popc(ga) + __popc(gb);
      if (a.y > 0) a.y = kNone;
      if (b.y > 0) b.y = kNone;
    }
    // back onto the stack, the first lane's entries on top, left above right
    const unsigned ma = ballot(a.y != kNone), mb = ballot(b.y != kNone);
    const int total = __popc(ma) + __popc(mb);
    const int above = __popc(ma & lt) + __popc(mb & lt);
    if (a.y != kNone) stk[top + total - 1 - above] = a;
    if (b.y != kNone) stk[top + total - 1 - above - (a.y != kNone ? 1 : 0)] = b;
    top += total;
    __syncwarp();
    if (!FILL) {
      const bool run = nl > 0 && (nl >= kRangeRun<G> || top == 0);
      if (!__any_sync(FULL, run)) continue;
      const int nls = run ? nl : 0;
#pragma unroll 1
      for (int u0 = 0; __any_sync(FULL, u0 < nls); u0 += G) {
        const int2 x = u0 + gl < nls ? list[u0 + gl] : make_int2(0, 0);
        int32_t inc = x.y;
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
          const int32_t v = __shfl_up_sync(FULL, inc, o, G);
          if (gl >= o) inc += v;
        }
        const int32_t tot = __shfl_sync(FULL, inc, G - 1, G);
        const int32_t delta = x.x - (inc - x.y);
#pragma unroll 2
        for (int32_t t = gl; __any_sync(FULL, t - gl < tot); t += G) {
          const int32_t p = __shfl_sync(FULL, delta, find(inc, t), G) + t;
          double d2;
          if (t < tot && qt.hit(p, false, d2)) ++cnt;
        }
      }
      if (run) nl = 0;
      __syncwarp();
    } else {
      if (!__any_sync(FULL, lead > 0)) continue;
      const int32_t ct = gl < lead ? abs(e.y) : 0;
      int32_t inc = ct;
#pragma unroll
      for (int o = 1; o < G; o <<= 1) {
        const int32_t v = __shfl_up_sync(FULL, inc, o, G);
        if (gl >= o) inc += v;
      }
      const int32_t tot = __shfl_sync(FULL, inc, G - 1, G);
      const int32_t delta = e.x - (inc - ct);
      const unsigned wholes = ballot(gl < lead && e.y < 0);
#pragma unroll 2
      for (int32_t t = gl; __any_sync(FULL, t - gl < tot); t += G) {
        const int j = find(inc, t);
        const int32_t p = __shfl_sync(FULL, delta, j, G) + t;
        bool hit = t < tot;
        double d2 = 0.0;
        int32_t id = 0;
        if (hit) {
          id = CKD_LDT(&tv.ids[p]);
          hit = qt.hit(p, (wholes >> j) & 1u, d2);
        }
        const unsigned hm = ballot(hit);
        if (hit) {
          const int64_t o = cur + __popc(hm & lt);
          if (o < cur_end) {
            oidx[o] = id;
            if (QT::kDist) odist[o] = want_d2 ? d2 : sqrt(d2);
          }
        }
        cur += __popc(hm);
      }
      if (cur >= cur_end) top = 0;  // all of the row's results are found
    }
  }
  if (!FILL) {
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) cnt += __shfl_xor_sync(FULL, cnt, o);
    if (gl == 0 && valid) counts[qi] = cnt;
  }
}

template <class QT, bool FILL>
ckd_status range_group_launch(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq,
                              double r2, int64_t* counts, const int64_t* offsets, int64_t* idx,
                              double* dist, int want_d2, cudaStream_t s) {
  constexpr int G = 8, NG = 128 / G;
  const size_t sm = (size_t)NG * (range_stack<G>(t->depth) + kRangeRun<G> + 2 * G) * sizeof(int2);
  k_range_group<QT, FILL, G><<<(unsigned)cdiv(nq, NG), 128, sm, s>>>(
      t->view(), q, order, nq, t->depth, r2, counts, offsets, idx, dist, want_d2);
  CKD_LAUNCH_CHECK();
  return CKD_OK;
}

// rows of the fill split by length: heavy ones (>= kHeavyRow) to `heavy`, the rest
// to `light`, both in the processing order (`order`, the leaf order when given)
__global__ void k_split_rows(const int64_t* __restrict__ offsets, const int32_t* __restrict__ order,
                             int64_t nq, int64_t heavy_row, int32_t* __restrict__ heavy,
                             unsigned* __restrict__ n_heavy, int32_t* __restrict__ light,
                             unsigned* __restrict__ n_light) {
  const int64_t slot = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool valid = slot < nq;
  const int64_t i = valid ? (order ? (int64_t)order[slot] : slot) : 0;
  const bool h = valid && offsets[i + 1] - offsets[i] >= heavy_row;
  const unsigned hm = __ballot_sync(0xffffffffu, h);
  const unsigned lm = __ballot_sync(0xffffffffu, valid && !h);
  unsigned hb = 0, lb = 0;
  if (lane == 0) {
    if (hm) hb = atomicAdd(n_heavy, (unsigned)__popc(hm));
    if (lm) lb = atomicAdd(n_light, (unsigned)__popc(lm));
  }
  hb = __shfl_sync(0xffffffffu, hb, 0);
  lb = __shfl_sync(0xffffffffu, lb, 0);
  const unsigned below = (1u << lane) - 1u;
  if (h) heavy[hb + __popc(hm & below)] = (int32_t)i;
  if (valid && !h) light[lb + __popc(lm & below)] = (int32_t)i;
}

// Per-lane box search: each lane walks the tree for its own box with a private
// stack, left child first, so a row comes out in the same order as the packet
// kernel below (left-first DFS, leaf order) without the warp serialising the union
// of 32 boxes' paths.  Stack depth <= tree depth + 1 (<= 2 pushes per pop).
constexpr int kBoxLaneStack = 128;
// A subtree of at least this many points whose split the box straddles (both
// children would be visited) is tested against the box as a whole: when
// its tight bounding box lies strictly inside the query box, every split below it
// lies strictly inside too (a sliding-midpoint split lies between, or on, its node's
// points), so the strict descent (:1296-1300) reaches every leaf and the inclusive
// test (:1319) accepts every point: the subtree's whole leaf-ordered range is the
// answer, in the depth-first order of its leaves.
constexpr int32_t kBoxWholeMin = 64;
template <int D>
__device__ __forceinline__ bool box_holds_node(const TreeView& tv, int32_t node,
                                               const double (&lo)[D], const double (&hi)[D]) {
  const double* b = tv.box + (int64_t)node * 2 * D;
  bool in = true;
#pragma unroll
  for (int j = 0; j < D; ++j) in = in && lo[j] < __ldg(b + 2 * j) && __ldg(b + 2 * j + 1) < hi[j];
  return in;
}

template <int D, bool FILL>
__global__ void __launch_bounds__(128) k_box_lane(TreeView tv, const double* __restrict__ boxes,
                                                  int64_t nb, int64_t* __restrict__ counts,
                                                  const int64_t* __restrict__ offsets,
                                                  int64_t* __restrict__ oidx,
                                                  const int32_t* __restrict__ broot) {
  const int64_t bi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (bi >= nb) return;
  double lo[D], hi[D];
#pragma unroll
  for (int j = 0; j < D; ++j) {
    lo[j] = boxes[bi * 2 * D + 2 * j];
    hi[j] = boxes[bi * 2 * D + 2 * j + 1];
  }
  int64_t cnt = 0;
  int64_t cur = FILL ? offsets[bi] : 0;
  const int64_t cur_end = FILL ? offsets[bi + 1] : 0;
  int32_t stk[kBoxLaneStack];
  int top = 0;
  stk[0] = broot ? broot[bi] : 0;
  while (top >= 0) {
    const int32_t node = stk[top--];
    const NodeMeta m = load_meta(tv.meta, node);
    if (m.left < 0) {
      for (int i = 0; i < m.count; ++i) {
        const int32_t p = m.start + i;
        bool in = true;
#pragma unroll
        for (int j = 0; j < D; ++j) {
          const double x = __ldg(&tv.pts[(int64_t)j * tv.n + p]);
          in = in && !(x < lo[j] || x > hi[j]);  // :1319
        }
        if (in) {
          if (FILL) {
            if (cur < cur_end) oidx[cur++] = __ldg(&tv.ids[p]);
          } else {
            ++cnt;
          }
        }
      }
    } else {
      double bl = 0.0, bh = 0.0;
#pragma unroll
      for (int j = 0; j < D; ++j)
        if (j == m.axis) {
          bl = lo[j];
          bh = hi[j];
        }
      const bool gl = bl < m.split, gr = bh > m.split;
      if (gl && gr && m.count >= kBoxWholeMin && box_holds_node<D>(tv, node, lo, hi)) {
        if (FILL) {
          for (int i = 0; i < m.count && cur < cur_end; ++i)
            oidx[cur++] = __ldg(&tv.ids[m.start + i]);
        } else {
          cnt += m.count;
        }
        continue;
      }
      if (gr) stk[++top] = m.left + 1;  // :1300 (visited second)
      if (gl) stk[++top] = m.left;      // :1296 (visited first)
    }
  }
  if (!FILL) counts[bi] = cnt;
}

// Copies of the recorded whole-subtree chunks of box rows, a warp per chunk.
__global__ void __launch_bounds__(128) k_box_emit(const int32_t* __restrict__ ids,
                                                  const EmitTask* __restrict__ tasks,
                                                  const unsigned* __restrict__ n_tasks,
                                                  unsigned task_cap, int64_t* __restrict__ oidx) {
  const int lane = threadIdx.x & 31;
  const int64_t nt = min((int64_t)*n_tasks, (int64_t)task_cap);
  const int64_t nwarps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t t = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < nt;
       t += nwarps) {
    const EmitTask e = tasks[t];
#pragma unroll 8
    for (int32_t i = lane; i < e.count; i += 32) oidx[e.out + i] = __ldg(&ids[e.start + i]);
  }
}

template <int D, bool FILL>
__global__ void __launch_bounds__(128) k_box(TreeView tv, const double* __restrict__ boxes,
                                             int64_t nb, int32_t* __restrict__ gstack,
                                             int stack_len, int64_t* __restrict__ counts,
                                             const int64_t* __restrict__ offsets,
                                             int64_t* __restrict__ oidx,
                                             const int32_t* __restrict__ broot) {
  __shared__ int32_t snode[4][kStack];
  __shared__ unsigned smask[4][kStack];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int64_t gw = (int64_t)blockIdx.x * nw + w;
  int32_t* stn = gstack ? gstack + gw * 2 * stack_len : snode[w];
  unsigned* stm = gstack ? reinterpret_cast<unsigned*>(gstack + gw * 2 * stack_len + stack_len)
                         : smask[w];
  int64_t bi = gw * 32 + lane;
  bool valid = bi < nb;
  double lo[D], hi[D];
#pragma unroll
  for (int j = 0; j < D; ++j) {
    lo[j] = valid ? boxes[bi * 2 * D + 2 * j] : 0.0;
    hi[j] = valid ? boxes[bi * 2 * D + 2 * j + 1] : -1.0;
  }
  const unsigned bit = 1u << lane;
  unsigned vm = __ballot_sync(0xffffffffu, valid);
  int64_t cnt = 0;
  int64_t cur = (FILL && valid) ? offsets[bi] : 0;
  const int64_t cur_end = (FILL && valid) ? offsets[bi + 1] : 0;
  int top = 0;
  if (broot) {
    // forest: one start entry per distinct tree among the warp's boxes
    const int32_t r = valid ? broot[bi] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, r);
    const bool leader = valid && (__ffs(same) - 1) == lane;
    const unsigned lead = __ballot_sync(0xffffffffu, leader);
    if (leader) {
      const int slot = __popc(lead & (bit - 1u));
      stn[slot] = r;
      stm[slot] = same;
    }
    top = __popc(lead) - 1;
  } else if (lane == 0) {
    stn[0] = 0;
    stm[0] = vm;
  }
  __syncwarp();
  while (top >= 0) {
    int32_t node = stn[top];
    unsigned mask = stm[top];
    --top;
    __syncwarp();
    bool mine = (mask & bit) != 0;
    NodeMeta m = load_meta(tv.meta, node);
    if (m.left < 0) {
      for (int i = 0; i < m.count; ++i) {
        int32_t p = m.start + i;
        bool in = mine;
#pragma unroll
        for (int j = 0; j < D; ++j) {
          double x = __ldg(&tv.pts[(int64_t)j * tv.n + p]);
          in = in && !(x < lo[j] || x > hi[j]);  // :1319
        }
        if (in) {
          if (FILL) {
            if (cur < cur_end) oidx[cur++] = __ldg(&tv.ids[p]);
          } else {
            ++cnt;
          }
        }
      }
    } else {
      double bl = 0.0, bh = 0.0;
#pragma unroll
      for (int j = 0; j < D; ++j)
        if (j == m.axis) {
          bl = lo[j];
          bh = hi[j];
        }
      unsigned lm = __ballot_sync(0xffffffffu, mine && bl < m.split);  // :1296
      unsigned rm = __ballot_sync(0xffffffffu, mine && bh > m.split);  // :1300
      if (lane == 0) {
        int t2 = top;
        if (rm) {
          ++t2;
          stn[t2] = m.left + 1;
          stm[t2] = rm;
        }
        if (lm) {
          ++t2;
          stn[t2] = m.left;
          stm[t2] = lm;
        }
      }
      top += (rm ? 1 : 0) + (lm ? 1 : 0);
      __syncwarp();
    }
  }
  if (!FILL && valid) counts[bi] = cnt;
}

// Each row of a fill ordered by (d2, id), and the distances' roots.
ckd_status sort_rows(const int64_t* offsets, int64_t nq, int64_t* idx, double* dist, int sms,
                     cudaStream_t s) {
  Scratch sc(s);
  int32_t* big = nullptr;
  int64_t* toff = nullptr;
  unsigned long long* sel = nullptr;
  CKD_CUDA(sc.alloc(&big, sizeof(int32_t) * nq));
  CKD_CUDA(sc.alloc(&toff, sizeof(int64_t) * nq));
  CKD_CUDA(sc.alloc(&sel, 2 * sizeof(unsigned long long)));
  CKD_CUDA(cudaMemsetAsync(sel, 0, 2 * sizeof(unsigned long long), s));
  k_sort_rows<<<(unsigned)cdiv(nq, 128), 128, 0, s>>>(offsets, nq, idx, dist, big, sel, toff);
  CKD_LAUNCH_CHECK();
  unsigned long long hs[2] = {0, 0};
  CKD_CUDA(cudaMemcpyAsync(hs, sel, sizeof(hs), cudaMemcpyDeviceToHost, s));
  CKD_CUDA(cudaStreamSynchronize(s));
  if (hs[0] > 0) {
    int64_t* tidx = nullptr;
    double* tdist = nullptr;
    if (hs[1] > 0) {
      CKD_CUDA(sc.alloc(&tidx, sizeof(int64_t) * hs[1]));
      CKD_CUDA(sc.alloc(&tdist, sizeof(double) * hs[1]));
    }
    const unsigned g = (unsigned)std::min<unsigned long long>(hs[0], (unsigned long long)sms * 8);
    k_sort_big<<<g, 256, 0, s>>>(offsets, big, sel, toff, idx, dist, tidx, tdist);
    CKD_LAUNCH_CHECK();
  }
  return CKD_OK;
}

// Batches up to which every query takes a warp of its own.  Beyond, the packet
// kernel goes first: 32 queries adjacent in leaf order share their nodes, which is
// faster while the balls are small against their spacing (10^6 queries on 2^20
// uniform points, 5 results each: count 1.05 against 2.29 ms) and far slower
// where density is uneven (3 x 10^5 queries on 2^22 clustered points, 1290 results
// each: 12.1 against 2.1 ms).  There a packet that has visited kPacketBudget nodes
// hands its queries over, unless they lie denser than half the points (2^22
// clustered points, 950 results each, count with / without handing over: 2^20
// queries 8.3 / 12.4 ms, 2^22 queries 27.4 / 23.4 ms); on an even tree it shares
// enough to go on (10^6 queries on 2^20 uniform points, 2700 results each: 13.3
// against 16.5 ms).  Even trees that the caches hold change over earlier (10^4 uniform
// points, 20 results each, packets / warps, us: 90k queries 504 / 481, 199k 597 / 730).
// The fill gives the packets rows of fewer than 64 results only (3 x 10^5 rows of 287:
// 13.4 ms as packets, 2.2 as warps; of 30: 1.09 and 1.05), on even trees with rows of up
// to kPacketMean on average those of fewer than kHeavyRow: 32 neighbours' balls share most
// of their nodes there, and packets thinned out by the longer of like rows lose by it (3 x
// 10^5 queries of 2^20 uniform points, count and fill, the line at 256 / at 64, ms: 60
// results 2.40 / 3.35, 80 2.64 / 4.02, 130 3.31 / 4.30, 160 3.83 / 4.20, 200 5.02 / 4.61).
constexpr int kPacketBudget = 512;
constexpr double kPacketMean = 150.0;
// results a ball holds on average where the points fill their extent evenly; infinite on
// an uneven tree or where the extent is not known
double even_hits(const ckd_tree* t, double r) {
  constexpr double kBall[9] = {1.0, 2.0, 3.14159, 4.18879, 4.93480, 5.26379, 5.16771, 4.72477, 4.05871};
  if (tree_uneven(t)) return INFINITY;
  double hits = (double)t->n * kBall[t->d];
  for (int j = 0; j < t->d; ++j) {
    if (!(t->extent[j] > 0.0)) return INFINITY;  // unknown or flat
    hits *= r / t->extent[j];
  }
  return hits;
}
int64_t ball_warp_max(const ckd_tree* t, double r) {
  return t->n < 32768 && even_hits(t, r) < kPacketMean ? 100000 : 200000;
}
int64_t packet_row(const ckd_tree* t, int64_t nq, double r, int64_t total) {
  const double mean = total >= 0 && !tree_uneven(t) ? (double)total / (double)nq : even_hits(t, r);
  return mean < kPacketMean ? kHeavyRow : 64;
}
bool ball_warp_ok(const ckd_tree* t) { return t->screen_ok && t->depth < kBallReserve - 3; }

// Whether a ball search takes eight lanes per query: small balls (the count of a
// uniform filling of the tree's extent) in large batches on an even tree.  Measured on
// uniform points, count + fill, a warp / eight lanes (us): 2^20 points, 5 results a
// row: 8000 queries 77 / 88, 16000 120 / 100, 100000 541 / 347; 30 results: 32000 256 /
// 251, 100000 724 / 573 (2^22 points: 304 / 368 and 839 / 806); 290 results and more, and
// clustered points at any size: the warp.
bool range_narrow(const ckd_tree* t, int64_t nq, double r) {
  return nq >= 12000 && even_hits(t, r) <= (nq >= 100000 ? 64.0 : 16.0);
}

// Whether a fill cuts its long rows: batches with fewer rows than the GPU's resident
// warps, or few long rows among more (forests), where density is uneven and the caller
// knows that rows are long on average.  Measured, fill walked whole / cut (us), 2^22
// clustered points: 300 balls of 9500 results 1220 / 523, 4001 of 730 605 / 289 and of
// 34800 2415 / 2019; 2^20 points in one cluster: 1000 boxes of 200 171 / 95, of 84000
// 2057 / 1083; 2^19 clustered, 8000 balls of 960: 390 / 442.  200 trees of 2.5e7 points:
// 12800 boxes of 2460 results 2257 / 993, 51200 balls of 2130 3782 / 4351; of 1.6e6: 12800
// balls of 130 190 / 200.  Rows of a few results gain nothing and would pay for two more
// launches (12 us); on 2^17 points the walks are as short as those.
bool cut_long_rows(const ckd_tree* t, int64_t nq, int64_t total) {
  return nq <= (t->n_trees > 1 ? 16384 : 4736) && t->n >= (1 << 19) && total >= nq * 192 &&
         (t->n_trees > 1 || tree_uneven(t));
}

template <int D, bool PER>
ckd_status ball_launch(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq,
                       double r, bool fill, int sorted, int64_t* counts, const int64_t* offsets,
                       int64_t* idx, double* dist, cudaStream_t s, const int32_t* qroot, int64_t total) {
  TreeView tv = t->view();
  const int threads = 128, nw = threads / 32;
  int64_t warps = cdiv(nq, 32);
  unsigned blocks = (unsigned)cdiv(warps, nw);
  // rows of the warp kernel (null: all, in processing order), and the packet
  // kernel's rows before it for large batches and for trees that the warp kernel
  // does not take
  const bool warp = ball_warp_ok(t), packet = !warp || nq > ball_warp_max(t, r);
  // a packet stack holds at most one pending sibling per level, plus the roots
  int stack_len = std::max(kStack, t->depth + 4 + (qroot ? 32 : 0));
  Scratch sc(s);
  int32_t* gstack = nullptr;
  if (packet && stack_len > kStack)
    CKD_CUDA(sc.alloc(&gstack, sizeof(int32_t) * 2 * stack_len * (int64_t)blocks * nw));
  double r2 = r * r;  // radius**2 (cosmokdtree.f90:1112)
  int dev = 0, sms = 148;
  CKD_CUDA(cudaGetDevice(&dev));
  CKD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  if (warp && !packet && !qroot && range_narrow(t, nq, r)) {
    if (!fill)
      return range_group_launch<BallQuery<D, PER>, false>(t, q, order, nq, r2, counts, nullptr,
                                                          nullptr, nullptr, 0, s);
    CKD_TRY((range_group_launch<BallQuery<D, PER>, true>(t, q, order, nq, r2, nullptr, offsets, idx,
                                                         dist, sorted ? 1 : 0, s)));
    return sorted ? sort_rows(offsets, nq, idx, dist, sms, s) : CKD_OK;
  }
  int32_t *heavy = nullptr, *light = nullptr;
  unsigned* cnt = nullptr;  // heavy rows, light rows, emission tasks, parts
  if (packet || fill) {
    CKD_CUDA(sc.alloc(&cnt, 4 * sizeof(unsigned)));
    CKD_CUDA(cudaMemsetAsync(cnt, 0, 4 * sizeof(unsigned), s));
  }
  if (packet) {
    if (warp || fill) CKD_CUDA(sc.alloc(&heavy, sizeof(int32_t) * nq));
    if (fill) {
      CKD_CUDA(sc.alloc(&light, sizeof(int32_t) * nq));
      k_split_rows<<<(unsigned)cdiv(nq, 256), 256, 0, s>>>(
          offsets, order, nq, warp ? packet_row(t, nq, r, total) : kHeavyRow, heavy, cnt, light, cnt + 1);
      CKD_LAUNCH_CHECK();
    }
    int32_t* bail = warp && tree_uneven(t) && nq * 2 <= t->n ? heavy : nullptr;
    const int w2 = sorted ? 1 : 0;
    if (fill && qroot)
      k_ball<D, PER, true, true><<<blocks, threads, 0, s>>>(
          tv, q, light, nq, cnt + 1, r2, gstack, stack_len, nullptr, offsets, idx, dist, w2, qroot,
          bail, cnt, kPacketBudget);
    else if (fill)
      k_ball<D, PER, true><<<blocks, threads, 0, s>>>(
          tv, q, light, nq, cnt + 1, r2, gstack, stack_len, nullptr, offsets, idx, dist, w2,
          nullptr, bail, cnt, kPacketBudget);
    else if (qroot)
      k_ball<D, PER, false, true><<<blocks, threads, 0, s>>>(
          tv, q, order, nq, nullptr, r2, gstack, stack_len, counts, nullptr, nullptr, nullptr, 0,
          qroot, bail, cnt, kPacketBudget);
    else
      k_ball<D, PER, false><<<blocks, threads, 0, s>>>(
          tv, q, order, nq, nullptr, r2, gstack, stack_len, counts, nullptr, nullptr, nullptr, 0,
          nullptr, bail, cnt, kPacketBudget);
    CKD_LAUNCH_CHECK();
  }
  const unsigned task_cap =
      (unsigned)std::min<int64_t>(kTaskCap, std::max<int64_t>(1 << 16, nq * 64));
  EmitTask* tasks = nullptr;
  if (fill) CKD_CUDA(sc.alloc(&tasks, sizeof(EmitTask) * task_cap));
  if (warp) {
    const int32_t* rows = packet ? heavy : order;
    const unsigned* n_rows = packet ? cnt : nullptr;
    if (fill)
      CKD_TRY((range_warp_fill<BallQuery<D, PER>>(t, q, rows, nq, n_rows, r2, offsets, idx, dist,
                                                  sorted ? 1 : 0, tasks, cnt + 2, task_cap, qroot,
                                                  cut_long_rows(t, nq, total), cnt + 3, sms, s)));
    else
      CKD_TRY((range_warp_count<BallQuery<D, PER>>(t, q, rows, nq, n_rows, r2, counts, qroot, sms,
                                                   s)));
  } else if (fill) {
    const int64_t hblocks = std::min<int64_t>(cdiv(nq, 4), (int64_t)sms * 8);
    const int hstack_len = std::max(kHeavyStack, t->depth + 4);
    int32_t* hstack = nullptr;
    if (hstack_len > kHeavyStack)
      CKD_CUDA(sc.alloc(&hstack, sizeof(int32_t) * hstack_len * hblocks * 4));
    k_ball_fill_warp<D, PER><<<(unsigned)std::max<int64_t>(1, hblocks), 128, 0, s>>>(
        tv, q, heavy, cnt, r2, hstack, hstack_len, offsets, idx, dist, sorted ? 1 : 0, tasks,
        cnt + 2, task_cap, qroot);
    CKD_LAUNCH_CHECK();
  }
  if (fill) {
    k_ball_emit<D, PER><<<(unsigned)sms * 8, 128, 0, s>>>(tv, q, tasks, cnt + 2, task_cap, idx,
                                                          dist, sorted ? 1 : 0);
    CKD_LAUNCH_CHECK();
  }
  return fill && sorted ? sort_rows(offsets, nq, idx, dist, sms, s) : CKD_OK;
}

// Boxes per call up to which the warp kernel is used on a single tree; beyond, a lane
// per box is faster for evenly filled boxes.  Forest boxes always take the warp
// kernel: their trees are clusters whose central boxes hold most of the points.
constexpr int64_t kBoxWarpMax = 32768;

template <int D>
ckd_status box_launch(const ckd_tree* t, const double* boxes, int64_t nb, bool fill,
                      int64_t* counts, const int64_t* offsets, int64_t* idx, cudaStream_t s,
                      const int32_t* broot, int64_t total) {
  TreeView tv = t->view();
  const int threads = 128, nw = threads / 32;
  if (t->depth < kBallReserve - 3 && (nb <= kBoxWarpMax || broot) && box_warp_enabled()) {
    int dev = 0, sms = 148;
    CKD_CUDA(cudaGetDevice(&dev));
    CKD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (!fill)
      return range_warp_count<BoxQuery<D>>(t, boxes, nullptr, nb, nullptr, 0.0, counts, broot, sms,
                                           s);
    Scratch sc(s);
    const unsigned task_cap =
        (unsigned)std::min<int64_t>(kTaskCap, std::max<int64_t>(1 << 16, nb * 64));
    // tasks, their counter and that of the parts behind them; without room for them the
    // warps copy whole ranges themselves
    EmitTask* tasks = nullptr;
    unsigned* ntask = nullptr;
    if (sc.alloc(&tasks, sizeof(EmitTask) * (task_cap + 1)) == cudaSuccess) {
      ntask = reinterpret_cast<unsigned*>(tasks + task_cap);
      CKD_CUDA(cudaMemsetAsync(ntask, 0, 2 * sizeof(unsigned), s));
    } else {
      cudaGetLastError();
    }
    CKD_TRY((range_warp_fill<BoxQuery<D>>(t, boxes, nullptr, nb, nullptr, 0.0, offsets, idx, nullptr,
                                          0, tasks, ntask, task_cap, broot,
                                          tasks && cut_long_rows(t, nb, total),
                                          tasks ? ntask + 1 : nullptr, sms, s)));
    if (tasks) {
      k_box_emit<<<(unsigned)sms * 8, 128, 0, s>>>(tv.ids, tasks, ntask, task_cap, idx);
      CKD_LAUNCH_CHECK();
    }
    return CKD_OK;
  }
  if (t->depth < kBoxLaneStack - 2) {
    const unsigned lb = (unsigned)cdiv(nb, threads);
    if (fill)
      k_box_lane<D, true><<<lb, threads, 0, s>>>(tv, boxes, nb, nullptr, offsets, idx, broot);
    else
      k_box_lane<D, false><<<lb, threads, 0, s>>>(tv, boxes, nb, counts, nullptr, nullptr, broot);
    CKD_LAUNCH_CHECK();
    return CKD_OK;
  }
  int64_t warps = cdiv(nb, 32);
  unsigned blocks = (unsigned)cdiv(warps, nw);
  // a packet stack grows by at most one entry per level past its start entries
  int stack_len = std::max(kStack, t->depth + 4 + (broot ? 32 : 0));
  Scratch sc(s);
  int32_t* gstack = nullptr;
  if (stack_len > kStack)
    CKD_CUDA(sc.alloc(&gstack, sizeof(int32_t) * 2 * stack_len * (int64_t)blocks * nw));
  if (fill)
    k_box<D, true><<<blocks, threads, 0, s>>>(tv, boxes, nb, gstack, stack_len, nullptr, offsets,
                                              idx, broot);
  else
    k_box<D, false><<<blocks, threads, 0, s>>>(tv, boxes, nb, gstack, stack_len, counts, nullptr,
                                               nullptr, broot);
  CKD_LAUNCH_CHECK();
  return CKD_OK;
}

}  // namespace

bool want_order(const ckd_tree* t, int64_t nq);
ckd_status query_order_roots(const ckd_tree* t, const double* q, int64_t nq, int32_t* order,
                             const int32_t* qroot, cudaStream_t s);

// Leaf order of a ball search's queries.  A warp per query gains from it only
// through the caches, where density is uneven and rows are long (10^5 queries on 2^22 clustered points, 218 results
// each: count + fill 1473 ordered, 1920 us in the caller's order; on 2^20 uniform
// points 611 against 533, the ordering included).
bool want_ball_order(const ckd_tree* t, int64_t nq, double r) {
  if (query_order_mode() != 0 || nq > ball_warp_max(t, r) || !ball_warp_ok(t)) return want_order(t, nq);
  return nq >= 50000 && tree_uneven(t) && want_order(t, nq);
}

ckd_status ball_run(const ckd_tree* t, const double* q, int64_t nq, double r, bool fill, int sorted,
                    int64_t* counts, const int64_t* offsets, int64_t* idx, double* dist,
                    cudaStream_t s, const int32_t* qroot, int64_t total) {
  int32_t* order = nullptr;
  Scratch sc(s);
  if (want_ball_order(t, nq, r)) {
    CKD_CUDA(sc.alloc(&order, sizeof(int32_t) * nq));
    CKD_TRY(query_order_roots(t, q, nq, order, qroot, s));
  }
  ckd_status st;
#define CKD_BALL_CASE(DD)                                                                      \
  case DD:                                                                                     \
    st = t->periodic ? ball_launch<DD, true>(t, q, order, nq, r, fill, sorted, counts, offsets, \
                                             idx, dist, s, qroot, total)                       \
                     : ball_launch<DD, false>(t, q, order, nq, r, fill, sorted, counts,         \
                                              offsets, idx, dist, s, qroot, total);                   \
    break;
  switch (t->d) {
    CKD_BALL_CASE(1)
    CKD_BALL_CASE(2)
    CKD_BALL_CASE(3)
    CKD_BALL_CASE(4)
    CKD_BALL_CASE(5)
    CKD_BALL_CASE(6)
    CKD_BALL_CASE(7)
    CKD_BALL_CASE(8)
    default: st = fail(CKD_ERR_BAD_DIM, "dimensionality must be 1..8");
  }
#undef CKD_BALL_CASE
  return st;
}

ckd_status box_run(const ckd_tree* t, const double* boxes, int64_t nb, bool fill, int64_t* counts,
                   const int64_t* offsets, int64_t* idx, cudaStream_t s, const int32_t* broot,
                   int64_t total) {
  switch (t->d) {
    case 1: return box_launch<1>(t, boxes, nb, fill, counts, offsets, idx, s, broot, total);
    case 2: return box_launch<2>(t, boxes, nb, fill, counts, offsets, idx, s, broot, total);
    case 3: return box_launch<3>(t, boxes, nb, fill, counts, offsets, idx, s, broot, total);
    case 4: return box_launch<4>(t, boxes, nb, fill, counts, offsets, idx, s, broot, total);
    case 5: return box_launch<5>(t, boxes, nb, fill, counts, offsets, idx, s, broot, total);
    case 6: return box_launch<6>(t, boxes, nb, fill, counts, offsets, idx, s, broot, total);
    case 7: return box_launch<7>(t, boxes, nb, fill, counts, offsets, idx, s, broot, total);
    case 8: return box_launch<8>(t, boxes, nb, fill, counts, offsets, idx, s, broot, total);
  }
  return fail(CKD_ERR_BAD_DIM, "dimensionality must be 1..8");
}

}  // namespace ckd
