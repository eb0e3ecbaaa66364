// knn.cu -- exact k-nearest-neighbour search (cosmokdtree.f90:504-905): query
// ordering, the per-lane and packet kernels, the kernel choice, forests, the
// learned-bound path and the allocation-free entry point.
//
// One query per lane.  Each lane keeps its k best (squared distance, id) in a
// max-heap (root = current k-th); a candidate enters iff it ranks strictly before
// the root under (d2, id) order, the canonical form of the strict test at
// cosmokdtree.f90:658.  The heap starts full of (HUGE(0.0), -1) sentinels
// (cosmokdtree.f90:517-518).  Distances are FP64, separately rounded, so results
// are bit-identical to the CPU restatement.
#include <algorithm>
#include <cmath>
#include <mutex>

#include "ckd_common.cuh"
#include "ckd_knn.cuh"
#include "ckd_knn_lane.cuh"
#include "ckd_mlp.cuh"
#include "ckd_scan.cuh"
#include "ckd_traverse.cuh"

namespace ckd {

// a group of lanes per query (ckd_knn_group.cuh): sorted rows, k <= 128
#define CKD_KG(DD)                                                                            \
  ckd_status knn_group_d##DD(const ckd_tree*, const double*, const int32_t*, int64_t, int,    \
                             double*, int64_t*, const int32_t*, cudaStream_t);                \
  ckd_status knn_group_bound_d##DD(const ckd_tree*, const double*, const int32_t*, int64_t,   \
                                   int, double*, int64_t*, const double*, const int32_t*,     \
                                   int32_t*, unsigned*, cudaStream_t);
CKD_KG(1) CKD_KG(2) CKD_KG(3) CKD_KG(4) CKD_KG(5) CKD_KG(6) CKD_KG(7) CKD_KG(8)
#undef CKD_KG

namespace {

constexpr int kStack = 96;   // per-warp traversal stack of the packet kernel

// process-wide traversal statistics of the screened kernel (diagnostics)
__device__ unsigned long long g_knn_stats[8];
bool g_stats_on = false;
unsigned long long* knn_stats_buffer() {
  if (!g_stats_on) return nullptr;
  void* p = nullptr;
  cudaGetSymbolAddress(&p, g_knn_stats);
  return reinterpret_cast<unsigned long long*>(p);
}

// ---------------------------------------------------------- heap storage
// Shared-memory heap: slot s of lane l at [s * 32 + l].
struct SmemHeap {
  double* key;
  int32_t* id;
  int lane;
  __device__ __forceinline__ double k(int s) const { return key[s * 32 + lane]; }
  __device__ __forceinline__ int64_t i(int s) const { return id[s * 32 + lane]; }
  __device__ __forceinline__ void set(int s, double d, int64_t x) {
    key[s * 32 + lane] = d;
    id[s * 32 + lane] = (int32_t)x;
  }
};
// Heap in the caller's output row (keys in dist, ids in idx).
struct RowHeap {
  double* key;
  int64_t* id;
  __device__ __forceinline__ double k(int s) const { return key[s]; }
  __device__ __forceinline__ int64_t i(int s) const { return id[s]; }
  __device__ __forceinline__ void set(int s, double d, int64_t x) {
    key[s] = d;
    id[s] = x;
  }
};

__device__ __forceinline__ bool before(double d1, int64_t i1, double d2, int64_t i2) {
  return d1 < d2 || (d1 == d2 && i1 < i2);
}

// cosmokdtree.f90:859-905: the root is replaced, then sifted down.
template <typename H>
__device__ __forceinline__ void heap_replace_root(H& h, int k, double d2, int64_t id) {
  int i = 0;
  for (;;) {
    int l = 2 * i + 1;
    if (l >= k) break;
    int c = l;
    double dc = h.k(l);
    int64_t ic = h.i(l);
    if (l + 1 < k) {
      double dr = h.k(l + 1);
      int64_t ir = h.i(l + 1);
      if (before(dc, ic, dr, ir)) {
        c = l + 1;
        dc = dr;
        ic = ir;
      }
    }
    if (!before(d2, id, dc, ic)) break;
    h.set(i, dc, ic);
    i = c;
  }
  h.set(i, d2, id);
}

// sift-down inside [0, end) used by the final heap sort
template <typename H>
__device__ __forceinline__ void heap_sift(H& h, int end, double d2, int64_t id) {
  int i = 0;
  for (;;) {
    int l = 2 * i + 1;
    if (l >= end) break;
    int c = l;
    double dc = h.k(l);
    int64_t ic = h.i(l);
    if (l + 1 < end) {
      double dr = h.k(l + 1);
      int64_t ir = h.i(l + 1);
      if (before(dc, ic, dr, ir)) {
        c = l + 1;
        dc = dr;
        ic = ir;
      }
    }
    if (!before(d2, id, dc, ic)) break;
    h.set(i, dc, ic);
    i = c;
  }
  h.set(i, d2, id);
}

// ascending (d2, id) in place (replaces the quicksort of cosmokdtree.f90:1553-1643)
template <typename H>
__device__ __forceinline__ void heap_sort(H& h, int k) {
  for (int end = k - 1; end > 0; --end) {
    double dr = h.k(0);
    int64_t ir = h.i(0);
    double de = h.k(end);
    int64_t ie = h.i(end);
    h.set(end, dr, ir);
    heap_sift(h, end, de, ie);
  }
}

// Packet traversal shared by the shared-memory and output-row heap variants.
template <int D, bool PER, typename H>
__device__ __forceinline__ void knn_walk(const TreeView& tv, const double (&q)[D], bool valid, H& h,
                                         int k, int32_t* stk, int lane) {
  double wd = valid ? CKD_HUGE : -1.0;  // lanes without a query never need a node
  int64_t wid = -1;
  int top = 0;
  if (lane == 0) stk[0] = 0;
  __syncwarp();
  while (top >= 0) {
    int32_t node = stk[top];
    --top;
    __syncwarp();
    NodeMeta m = load_meta(tv.meta, node);
    double md = box_mind2<D, PER>(tv, q, node);
    bool need = md <= wd;
    unsigned nm = __ballot_sync(0xffffffffu, need);
    if (nm == 0) continue;
    if (m.left < 0) {
      for (int i = 0; i < m.count; ++i) {
        int32_t p = m.start + i;
        double d2 = point_d2<D, PER>(tv, q, p);
        if (need && d2 <= wd) {
          int64_t id = __ldg(&tv.ids[p]);
          if (before(d2, id, wd, wid)) {
            heap_replace_root(h, k, d2, id);
            wd = h.k(0);
            wid = h.i(0);
          }
        }
      }
    } else {
      double qa = 0.0;
#pragma unroll
      for (int j = 0; j < D; ++j)
        if (j == m.axis) qa = q[j];
      unsigned lv = __ballot_sync(0xffffffffu, need && qa < m.split);
      bool left_first = 2 * __popc(lv) >= __popc(nm);
      int32_t nearc = left_first ? m.left : m.left + 1;
      int32_t farc = left_first ? m.left + 1 : m.left;
      if (lane == 0) {
        stk[top + 1] = farc;
        stk[top + 2] = nearc;
      }
      top += 2;
      __syncwarp();
    }
  }
}

template <int D, bool PER>
__global__ void __launch_bounds__(128) k_knn_smem(TreeView tv, const double* __restrict__ Q,
                                                  const int32_t* __restrict__ order, int64_t nq,
                                                  int k, int sorted, int32_t* __restrict__ gstack,
                                                  int stack_len, double* __restrict__ dist,
                                                  int64_t* __restrict__ idx) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double* keys = reinterpret_cast<double*>(smem) + (size_t)w * k * 32;
  int32_t* ids = reinterpret_cast<int32_t*>(reinterpret_cast<double*>(smem) + (size_t)nw * k * 32) +
                 (size_t)w * k * 32;
  int32_t* stk;
  int64_t gw = (int64_t)blockIdx.x * nw + w;
  if (gstack)
    stk = gstack + gw * stack_len;
  else
    stk = reinterpret_cast<int32_t*>(reinterpret_cast<int32_t*>(reinterpret_cast<double*>(smem) +
                                                                (size_t)nw * k * 32) +
                                     (size_t)nw * k * 32) +
          (size_t)w * kStack;
  int64_t slot = gw * 32 + lane;
  bool valid = slot < nq;
  int64_t qi = valid ? (order ? (int64_t)order[slot] : slot) : 0;
  double q[D];
#pragma unroll
  for (int j = 0; j < D; ++j) q[j] = valid ? Q[qi * D + j] : 0.0;
  SmemHeap h{keys, ids, lane};
  for (int s = 0; s < k; ++s) h.set(s, CKD_HUGE, -1);
  knn_walk<D, PER>(tv, q, valid, h, k, stk, lane);
  if (sorted) heap_sort(h, k);
  __syncwarp();
  // coalesced write-out: for each lane's query, the warp writes its row
  for (int qq = 0; qq < 32; ++qq) {
    int64_t s2 = gw * 32 + qq;
    if (s2 >= nq) break;
    int64_t row = order ? (int64_t)order[s2] : s2;
    for (int j = lane; j < k; j += 32) {
      double d2 = keys[j * 32 + qq];
      int32_t id = ids[j * 32 + qq];
      dist[row * k + j] = sqrt(d2);
      idx[row * k + j] = id < 0 ? -2 : (int64_t)id;
    }
  }
}

template <int D, bool PER>
__global__ void __launch_bounds__(128) k_knn_rows(TreeView tv, const double* __restrict__ Q,
                                                  const int32_t* __restrict__ order, int64_t nq,
                                                  int k, int sorted, int32_t* __restrict__ gstack,
                                                  int stack_len, double* __restrict__ dist,
                                                  int64_t* __restrict__ idx) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int64_t gw = (int64_t)blockIdx.x * nw + w;
  int32_t* stk = gstack + gw * stack_len;
  int64_t slot = gw * 32 + lane;
  bool valid = slot < nq;
  int64_t qi = valid ? (order ? (int64_t)order[slot] : slot) : 0;
  double q[D];
#pragma unroll
  for (int j = 0; j < D; ++j) q[j] = valid ? Q[qi * D + j] : 0.0;
  double dummy_k[1];
  int64_t dummy_i[1];
  RowHeap h{valid ? dist + qi * k : dummy_k, valid ? idx + qi * k : dummy_i};
  int kk = valid ? k : 1;
  for (int s = 0; s < kk; ++s) h.set(s, CKD_HUGE, -1);
  knn_walk<D, PER>(tv, q, valid, h, kk, stk, lane);
  if (!valid) return;
  if (sorted) heap_sort(h, k);
  for (int s = 0; s < k; ++s) {
    double d2 = h.k(s);
    int64_t id = h.i(s);
    h.set(s, sqrt(d2), id < 0 ? -2 : id);
  }
}

// The per-lane kernel: one warp per 32 query slots (knn_lane_run).
template <int D, bool PER, bool BOUNDED = false, bool PAIR = false>
__global__ void __launch_bounds__(128, 6) k_knn_lane2(TreeView tv, const double* __restrict__ Q,
                                                   const int32_t* __restrict__ order, int64_t nq,
                                                   int k, int sorted, double* __restrict__ dist,
                                                   int64_t* __restrict__ idx,
                                                   unsigned long long* __restrict__ stats,
                                                   const double* __restrict__ r2 = nullptr,
                                                   int32_t* __restrict__ miss = nullptr,
                                                   unsigned* __restrict__ nmiss = nullptr,
                                                   const int32_t* __restrict__ qleaf = nullptr,
                                                   const int32_t* __restrict__ qroot = nullptr) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint2* Hw = reinterpret_cast<uint2*>(smem) + (size_t)w * 32 * (k + 1);
  const int64_t gw = (int64_t)blockIdx.x * nw + w;
  knn_lane_run<D, PER, BOUNDED, PAIR>(tv, Q, order, nq, k, sorted, dist, idx, stats, r2, miss,
                                      nmiss, qleaf, qroot, 0, Hw, lane, gw);
}
// ------------------------------------------------------------ query order
// The leaf of each query, its bin (the leaf's first point >> shift) and its rank among
// the bin's queries so far.  The descent reads the first half of a node's record.
template <int D>
__global__ void k_locate(const NodeMeta* __restrict__ meta, const double* __restrict__ Q,
                         int64_t nq, int shift, int2* __restrict__ key,
                         int32_t* __restrict__ hist, int32_t* __restrict__ qleaf,
                         const int32_t* __restrict__ qroot) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  double q[D];
#pragma unroll
  for (int j = 0; j < D; ++j) q[j] = Q[i * D + j];
  int32_t node = qroot ? qroot[i] : 0;
  for (;;) {
    const int4 m = __ldg(reinterpret_cast<const int4*>(meta + node));  // split, left, axis
    if (m.z < 0) break;
    double qa = 0.0;
#pragma unroll
    for (int j = 0; j < D; ++j)
      if (j == m.w) qa = q[j];
    node = qa < __hiloint2double(m.y, m.x) ? m.z : m.z + 1;
  }
  const int32_t b = __ldg(&meta[node].start) >> shift;
  if (qleaf) qleaf[i] = node;
  key[i] = make_int2(b, atomicAdd(&hist[b], 1));
}

__global__ void k_bucket_place(const int2* __restrict__ key, int64_t nq,
                               const int32_t* __restrict__ off, int32_t* __restrict__ order) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  const int2 k = key[i];
  order[off[k.x] + k.y] = (int32_t)i;
}

__global__ void k_bucket_scatter(const int32_t* __restrict__ key, int64_t nq,
                                 const int32_t* __restrict__ off, int32_t* __restrict__ cursor,
                                 int32_t* __restrict__ order) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  int32_t b = key[i];
  int32_t pos = off[b] + atomicAdd(&cursor[b], 1);
  order[pos] = (int32_t)i;
}

ckd_status knn_group(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq, int k,
                     double* dist, int64_t* idx, const int32_t* qroot, cudaStream_t s) {
  switch (t->d) {
#define CKD_KG(DD) \
  case DD: return knn_group_d##DD(t, q, order, nq, k, dist, idx, qroot, s);
    CKD_KG(1) CKD_KG(2) CKD_KG(3) CKD_KG(4) CKD_KG(5) CKD_KG(6) CKD_KG(7) CKD_KG(8)
#undef CKD_KG
  }
  return fail(CKD_ERR_BAD_DIM, "dimensionality must be 1..8");
}

ckd_status knn_group_bound(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq,
                           int k, double* dist, int64_t* idx, const double* r2,
                           const int32_t* qleaf, int32_t* miss, unsigned* nmiss, cudaStream_t s) {
  switch (t->d) {
#define CKD_KG(DD) \
  case DD: return knn_group_bound_d##DD(t, q, order, nq, k, dist, idx, r2, qleaf, miss, nmiss, s);
    CKD_KG(1) CKD_KG(2) CKD_KG(3) CKD_KG(4) CKD_KG(5) CKD_KG(6) CKD_KG(7) CKD_KG(8)
#undef CKD_KG
  }
  return fail(CKD_ERR_BAD_DIM, "dimensionality must be 1..8");
}

// Whether the automatic choice takes a group of lanes per query
// (ckd_knn_group.cuh) instead of the per-lane kernel.  Sorted rows only: an unsorted
// row is in the order of its kernel's heap.  A lane per query takes about as long for
// 1000 queries as for 50000, the groups' time grows with the batch from a few thousand on.
// Where they cross depends, besides k, on what fills a lane's time: small trees stay in the
// caches (lower lines), short leaves and uneven density leave lanes waiting (higher
// lines).  The lines are fitted to both kernels' times on 100 trees of 3000 to 4 M points,
// 1-D to 8-D, leaf 1 to 128, uniform, clustered, lattices and forests, batches of 15000 to
// 10^6 from the points or uniform (20600 pairs of times, a slower choice counted three
// times); where they are taken, the groups are the slower kernel by more than 5 % in 2 %
// of them.  With one line for all trees and leaves it was 15 %, by a factor of two at
// worst.  Us, per-lane / groups, 3-D points, leaf 16: 2^20 uniform, k = 8: 75k queries 250 /
// 214, 110k 276 / 292; k = 32: 75k 531 / 421, 110k 563 / 585; leaf 64, k = 8: 110k 260 / 417;
// 2^22 clustered, k = 16: 110k 723 / 554, 200k 991 / 846; 6-D 2^22, leaf 32, k = 8: 110k
// 2388 / 2297, 200k 3707 / 4013, k = 32: 200k 9834 / 6233.
bool use_knn_group(const ckd_tree* t, int64_t nq, int k, int sorted) {
  if (!sorted || k > 128 || !t->screen_ok || t->depth >= kLaneStack - 1 || knn_variant() != 0 ||
      g_stats_on)
    return false;
  if (nq <= 4000 || k > kSmemK || (k == kSmemK && t->d > 2) || (k >= 48 && t->d > 4)) return true;
  // thousands of queries at 2^18 points and leaf 16, the exponents of the points (between
  // 2^13 and 2^22) and of 16 / leaf, and the factor for uneven trees
  struct Line {
    double base, size, leaf, uneven;
  };
  Line l;
  if (t->d <= 2)
    l = k == 1                ? Line{250, 0.2, 0, 0.8}
        : k <= 8 && t->d == 1 ? Line{220, 0.2, 0, 1.1}
        : k <= 8              ? Line{110, 0.25, 0, 1.2}
        : k <= 16             ? Line{94, 0.2, 0, 1.6}
        : k <= 32             ? Line{90, 0.3, 0, 1.6}
        : k < 48              ? Line{90, 0.25, 0, 1.2}
        : k < 56              ? Line{150, 0.4, 0, 1}
                              : Line{600, 0.3, 0, 1};
  else if (t->d <= 4)
    l = k == 1    ? Line{220, 0.1, 0.15, 0.36}
        : k <= 8  ? Line{80, 0.15, 0.42, 1}
        : k <= 16 ? Line{75, 0.17, 0.45, 1.45}
        : k <= 32 ? Line{125, 0.19, 0.5, 1.5}
        : k < 48  ? Line{350, 0.4, 0, 1.2}
                  : Line{800, 0.36, 0, 0.65};
  else
    l = k == 1    ? Line{25, 0.15, 0.2, 2}
        : k <= 8  ? Line{75, 0.17, 0.3, 1.15}
        : k <= 16 ? Line{105, 0.24, 0.6, 1.5}
        : k <= 32 ? Line{165, 0.3, 0.5, 1.8}
                  : Line{300, 0.14, 0.5, 1.2};
  const double size = std::min(std::max((double)t->n, 8192.0), 4194304.0);
  double line = 1000.0 * l.base * std::pow(size / 262144.0, l.size) *
                std::pow(16.0 / t->leaf, l.leaf) * (tree_uneven(t) ? l.uneven : 1.0);
  // many equal points, which leave leaves of a point or two: the nearest few of a
  // query tie and every subtree at distance zero is read (2^18 points in 2^13 places, k = 1:
  // 90k queries 119 / 203)
  if (k < 8 && (double)t->n_leaves * t->leaf > 4.0 * (double)t->n) line = std::min(line, 35000.0);
  return (double)nq <= line;
}

// Whether the learned-bound search takes a group of lanes per query for its bounded
// pass (us a call with ordering, network and reruns, per-lane / groups, 2^22 clustered
// points): k = 8: 20k queries 475 / 376, 50k 543 / 541, 100k 560 / 790; k = 32: 50k
// 972 / 710, 100k 1092 / 1090, 300k 2133 / 2559; 6-D: k = 8: 100k 2280 / 2102, k = 32: 300k
// 8838 / 8180.  For 33 <= k <= 64 the lists have room for 64, so the line rises with k (k = 33:
// 300k 3321 / 2699, 500k 4175 / 4253; k = 40: 500k 5223 / 4490, 1M 7920 / 8532; k = 48: 1M
// 10150 / 8989; k = 64: 1M 15242 / 9886).  Targets in the void about a single cluster cross
// earlier (k = 33: 200k 8748 / 10296; k = 64: 300k 15620 / 18857), which the lines below
// k = 56 make room for.
bool use_bound_group(const ckd_tree* t, int64_t nq, int k, int sorted) {
  if (!sorted || learned_kernel() != 3 || knn_variant() != 0 || g_stats_on) return false;
  if (t->d > 4) return k >= 48 || nq <= 32768 + 10000 * (int64_t)k;
  if (k <= 32) return nq <= 30000 + 2200 * (int64_t)k;
  return k >= 56 || nq <= (k <= 36 ? 150000 : k <= 44 ? 250000 : 450000);
}

// Kernel choice (ckd_set_knn_variant): 0 automatic, 1 FP64 packet traversal,
// 7 per-lane compact heap, 8 the same expanding nodes from child-pair records.
// Automatic takes a group of lanes per query where use_knn_group says so, else 8; trees too
// deep for their stacks, coordinates beyond the FP32 screen's range, unsorted
// rows of k > 64 and k > 128 take the packet kernel.
template <int D, bool PER>
ckd_status knn_launch(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq, int k,
                      int sorted, double* dist, int64_t* idx, cudaStream_t s,
                      int force_variant = -1) {
  TreeView tv = t->view();
  const int var = force_variant >= 0 ? force_variant : knn_variant();
  if (force_variant < 0) timing_begin(s);
  struct TimingEnd {
    cudaStream_t s;
    bool on;
    ~TimingEnd() {
      if (on) timing_end(s);
    }
  } timing_guard{s, force_variant < 0};
  if (use_knn_group(t, nq, k, sorted)) return knn_group(t, q, order, nq, k, dist, idx, nullptr, s);
  if (k <= kSmemK && t->screen_ok && var != 1 && t->depth < kLaneStack - 1) {
    const int nw7 = std::min(4, knn_warps_per_block());
    const unsigned blocks7 = (unsigned)cdiv(cdiv(nq, 32), nw7);
    size_t sm = (size_t)nw7 * compact_heap_bytes(k);
    const int bps = knn_blocks_per_sm();
    if (bps > 0) sm = std::max(sm, (size_t)(200 * 1024) / bps);
    if (var != 7) {
      CKD_CUDA(cudaFuncSetAttribute(k_knn_lane2<D, PER, false, true>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
      k_knn_lane2<D, PER, false, true><<<blocks7, nw7 * 32, sm, s>>>(
          tv, q, order, nq, k, sorted, dist, idx, knn_stats_buffer());
    } else {
      CKD_CUDA(cudaFuncSetAttribute(k_knn_lane2<D, PER>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
      k_knn_lane2<D, PER><<<blocks7, nw7 * 32, sm, s>>>(tv, q, order, nq, k, sorted, dist, idx,
                                                        knn_stats_buffer());
    }
    CKD_LAUNCH_CHECK();
    return CKD_OK;
  }
  const int threads = 128, nw = threads / 32;
  int64_t warps = cdiv(nq, 32);
  unsigned blocks = (unsigned)cdiv(warps, nw);
  int stack_len = std::max(kStack, t->depth + 4);
  int32_t* gstack = nullptr;
  bool use_gstack = stack_len > kStack || k > kSmemK;
  if (use_gstack)
    CKD_CUDA(dev_alloc((void**)&gstack, sizeof(int32_t) * stack_len * (int64_t)blocks * nw, s));
  struct Free {
    int32_t* p;
    cudaStream_t s;
    ~Free() {
      if (p) dev_free(p, s);
    }
  } free_guard{gstack, s};
  if (k <= kSmemK) {
    size_t sm = (size_t)nw * k * 32 * (sizeof(double) + sizeof(int32_t)) +
                (use_gstack ? 0 : (size_t)nw * kStack * sizeof(int32_t));
    CKD_CUDA(cudaFuncSetAttribute(k_knn_smem<D, PER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sm));
    k_knn_smem<D, PER><<<blocks, threads, sm, s>>>(tv, q, order, nq, k, sorted,
                                                   use_gstack ? gstack : nullptr, stack_len, dist,
                                                   idx);
  } else {
    k_knn_rows<D, PER><<<blocks, threads, 0, s>>>(tv, q, order, nq, k, sorted, gstack, stack_len,
                                                  dist, idx);
  }
  CKD_LAUNCH_CHECK();
  return CKD_OK;
}

template <int D>
ckd_status knn_dispatch_d(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq,
                          int k, int sorted, double* dist, int64_t* idx, cudaStream_t s) {
  if (t->periodic) return knn_launch<D, true>(t, q, order, nq, k, sorted, dist, idx, s);
  return knn_launch<D, false>(t, q, order, nq, k, sorted, dist, idx, s);
}

// Counting sort of the queries by leaf.  A query's rank in its bin comes from the
// histogram's own atomics, and bins hold several positions while there are fewer queries
// than points (a bin a query keeps the leaves apart): 2^24 self-queries 2969 -> 2498 us,
// 10^5 queries of 2^20 points 41 -> 34 us, against one bin a point and a second
// pass of atomics.
template <int D>
ckd_status order_impl(const ckd_tree* t, const double* q, int64_t nq, int32_t* order,
                      int32_t* qleaf, cudaStream_t s, const int32_t* qroot = nullptr) {
  int shift = 0;
  while ((t->n >> (shift + 1)) >= std::max<int64_t>(nq, 4096)) ++shift;
  const int64_t bins = (t->n >> shift) + 1;
  Scratch sc(s);
  int2* key = nullptr;
  int32_t *hist = nullptr, *off = nullptr;
  CKD_CUDA(sc.alloc(&key, sizeof(int2) * nq));
  CKD_CUDA(sc.alloc(&hist, sizeof(int32_t) * bins));
  CKD_CUDA(sc.alloc(&off, sizeof(int32_t) * (bins + 1)));
  CKD_CUDA(cudaMemsetAsync(hist, 0, sizeof(int32_t) * bins, s));
  unsigned g = (unsigned)cdiv(nq, 256);
  k_locate<D><<<g, 256, 0, s>>>(t->meta, q, nq, shift, key, hist, qleaf, qroot);
  CKD_LAUNCH_CHECK();
  CKD_TRY(scan_i32(hist, off, bins, s));
  k_bucket_place<<<g, 256, 0, s>>>(key, nq, off, order);
  CKD_LAUNCH_CHECK();
  return CKD_OK;
}

}  // namespace

ckd_status knn_stats(int enable, int64_t* out) {
  void* p = nullptr;
  CKD_CUDA(cudaGetSymbolAddress(&p, g_knn_stats));
  if (out) {
    CKD_CUDA(cudaDeviceSynchronize());
    CKD_CUDA(cudaMemcpy(out, p, sizeof(int64_t) * 8, cudaMemcpyDeviceToHost));
  }
  CKD_CUDA(cudaMemset(p, 0, sizeof(unsigned long long) * 8));
  CKD_CUDA(cudaDeviceSynchronize());
  g_stats_on = enable != 0;
  return CKD_OK;
}

ckd_status query_order(const ckd_tree* t, const double* q, int64_t nq, int32_t* order,
                       cudaStream_t s) {
  switch (t->d) {
#define CKD_QO(DD) \
  case DD: return order_impl<DD>(t, q, nq, order, nullptr, s);
    CKD_QO(1) CKD_QO(2) CKD_QO(3) CKD_QO(4) CKD_QO(5) CKD_QO(6) CKD_QO(7) CKD_QO(8)
#undef CKD_QO
  }
  return fail(CKD_ERR_BAD_DIM, "dimensionality must be 1..8");
}

// leaf order of queries that each start at their own tree's root (forests)
ckd_status query_order_roots(const ckd_tree* t, const double* q, int64_t nq, int32_t* order,
                             const int32_t* qroot, cudaStream_t s) {
  switch (t->d) {
#define CKD_QO(DD) \
  case DD: return order_impl<DD>(t, q, nq, order, nullptr, s, qroot);
    CKD_QO(1) CKD_QO(2) CKD_QO(3) CKD_QO(4) CKD_QO(5) CKD_QO(6) CKD_QO(7) CKD_QO(8)
#undef CKD_QO
  }
  return fail(CKD_ERR_BAD_DIM, "dimensionality must be 1..8");
}

// Queries of the group kernel gain from leaf order through L1 and L2 alone, so it
// pays later than for the per-lane kernel (us, caller's order / ordered): 3-D, k = 16:
// 50k 416 / 466, 100k 701 / 663 (2^22 clustered points), k = 8: 150k 471 / 481, 200k
// 618 / 612 (2^20 uniform); 6-D, where a query reads many leaves: 25k, k = 8: 615 / 587,
// k = 1: 117 / 197.
bool want_order_group(const ckd_tree* t, int64_t nq, int k) {
  const int mode = query_order_mode();
  if (mode != 0) return mode == 1 && nq > 1;
  if (nq * 8 < t->n / 64) return false;
  return t->d <= 4 ? nq >= 100000 && nq * std::min(k, 16) >= 1600000
                   : nq * std::min(k, 4) >= 100000;
}

// Queries are ordered by leaf when there are enough of them to fill many warps.
// (tuning key 6: 0 automatic, 1 always, 2 never)
bool want_order(const ckd_tree* t, int64_t nq) {
  const int mode = query_order_mode();
  if (mode == 1) return nq > 1;
  if (mode == 2) return false;
  return nq >= 4096 && nq * 8 >= t->n / 64;
}

ckd_status knn_ordered(const ckd_tree* t, const double* q, const int32_t* order, int64_t nq, int k,
                       int sorted, double* dist, int64_t* idx, cudaStream_t s) {
  switch (t->d) {
    case 1: return knn_dispatch_d<1>(t, q, order, nq, k, sorted, dist, idx, s);
    case 2: return knn_dispatch_d<2>(t, q, order, nq, k, sorted, dist, idx, s);
    case 3: return knn_dispatch_d<3>(t, q, order, nq, k, sorted, dist, idx, s);
    case 4: return knn_dispatch_d<4>(t, q, order, nq, k, sorted, dist, idx, s);
    case 5: return knn_dispatch_d<5>(t, q, order, nq, k, sorted, dist, idx, s);
    case 6: return knn_dispatch_d<6>(t, q, order, nq, k, sorted, dist, idx, s);
    case 7: return knn_dispatch_d<7>(t, q, order, nq, k, sorted, dist, idx, s);
    case 8: return knn_dispatch_d<8>(t, q, order, nq, k, sorted, dist, idx, s);
  }
  return fail(CKD_ERR_BAD_DIM, "dimensionality must be 1..8");
}

ckd_status knn_run(const ckd_tree* t, const double* q, int64_t nq, int k, int sorted, double* dist,
                   int64_t* idx, cudaStream_t s) {
  Scratch sc(s);
  int32_t* order = nullptr;
  if (use_knn_group(t, nq, k, sorted) ? want_order_group(t, nq, k) : want_order(t, nq)) {
    CKD_CUDA(sc.alloc(&order, sizeof(int32_t) * nq));
    CKD_TRY(query_order(t, q, nq, order, s));
  }
  return knn_ordered(t, q, order, nq, k, sorted, dist, idx, s);
}

// ===================================================================
// kNN over a forest (ckd_forest_knn): every query carries its tree (qroot =
// the tree's root node); the queries of all trees are ordered by leaf and
// searched by one launch that starts each query at its own root.  Expanding from the
// child-pair records, like the single-tree search, against each node's own record: 2.9 M
// queries of 200 trees, k = 8: 6.25 -> 5.38 ms a call, k = 31: 13.3 -> 11.8 ms.
namespace {

template <int D, bool PER>
ckd_status forest_knn_impl(const ckd_tree* t, const double* q, const int32_t* qroot, int64_t nq,
                           int k, int sorted, double* dist, int64_t* idx, cudaStream_t s) {
  Scratch sc(s);
  int32_t* order = nullptr;
  const bool warp = use_knn_group(t, nq, k, sorted);
  if (!warp || want_order_group(t, nq, k)) {
    CKD_CUDA(sc.alloc(&order, sizeof(int32_t) * nq));
    CKD_TRY(order_impl<D>(t, q, nq, order, nullptr, s, qroot));
  }
  timing_begin(s);
  if (warp) {
    CKD_TRY(knn_group(t, q, order, nq, k, dist, idx, qroot, s));
    timing_end(s);
    return CKD_OK;
  }
  const int nw = std::min(4, knn_warps_per_block());
  const unsigned blocks = (unsigned)cdiv(cdiv(nq, 32), nw);
  size_t sm = (size_t)nw * compact_heap_bytes(k);
  const int bps = knn_blocks_per_sm();
  if (bps > 0) sm = std::max(sm, (size_t)(200 * 1024) / bps);
  CKD_CUDA(cudaFuncSetAttribute(k_knn_lane2<D, PER, false, true>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  k_knn_lane2<D, PER, false, true><<<blocks, nw * 32, sm, s>>>(
      t->view(), q, order, nq, k, sorted, dist, idx, knn_stats_buffer(), nullptr, nullptr, nullptr,
      nullptr, qroot);
  CKD_LAUNCH_CHECK();
  timing_end(s);
  return CKD_OK;
}

}  // namespace

ckd_status forest_knn(const ckd_tree* t, const double* q, const int32_t* qroot, int64_t nq, int k,
                      int sorted, double* dist, int64_t* idx, cudaStream_t s) {
  if (!(t->screen_ok && t->depth < kLaneStack - 1 && k <= kSmemK))
    return fail(CKD_ERR_BAD_ARG,
                "forest kNN needs k <= 64, trees shallower than 127 levels and coordinates "
                "below 1e18");
  switch (t->d * 2 + (t->periodic ? 1 : 0)) {
#define CKD_FK(DD)                                                                        \
  case 2 * DD: return forest_knn_impl<DD, false>(t, q, qroot, nq, k, sorted, dist, idx, s); \
  case 2 * DD + 1: return forest_knn_impl<DD, true>(t, q, qroot, nq, k, sorted, dist, idx, s);
    CKD_FK(1) CKD_FK(2) CKD_FK(3) CKD_FK(4) CKD_FK(5) CKD_FK(6) CKD_FK(7) CKD_FK(8)
#undef CKD_FK
  }
  return fail(CKD_ERR_BAD_DIM, "dimensionality must be 1..8");
}

// ===================================================================
// kNN with the learned bound (ckd_knn_learned)
//
// locate + order the queries, predict each query's squared k-th distance
// (k_mlp_radius), run the bounded per-lane search, then rerun the queries it
// could not settle with the plain search.  The bounded kernel needs the FP32
// screen, k <= kSmemK and a stack deep enough for the tree; otherwise every query
// takes the plain path.
namespace {

template <int D, bool PER>
ckd_status knn_learned_impl(const ckd_tree* t, const ckd_mlp* net, const double* q, int64_t nq,
                            int k, int sorted, double* dist, int64_t* idx, int64_t* nfb_out,
                            cudaStream_t s) {
  int32_t *order = nullptr, *qleaf = nullptr, *miss = nullptr;
  double* r2 = nullptr;
  unsigned* nmiss = nullptr;
  Scratch sc(s);
  CKD_CUDA(sc.alloc(&order, sizeof(int32_t) * nq));
  CKD_CUDA(sc.alloc(&qleaf, sizeof(int32_t) * nq));
  CKD_CUDA(sc.alloc(&r2, sizeof(double) * nq));
  CKD_CUDA(sc.alloc(&miss, sizeof(int32_t) * nq));
  CKD_CUDA(sc.alloc(&nmiss, sizeof(unsigned)));
  CKD_CUDA(cudaMemsetAsync(nmiss, 0, sizeof(unsigned), s));
  ckd_status st = order_impl<D>(t, q, nq, order, qleaf, s);
  if (st == CKD_OK) {
    timing_begin(s);
    st = mlp_radius(t, net, q, order, qleaf, nq, k, r2, s);
  }
  if (st == CKD_OK && use_bound_group(t, nq, k, sorted)) {
    st = knn_group_bound(t, q, order, nq, k, dist, idx, r2, qleaf, miss, nmiss, s);
  } else if (st == CKD_OK) {
    const int nw = std::min(4, knn_warps_per_block());
    const unsigned blocks = (unsigned)cdiv(cdiv(nq, 32), nw);
    size_t sm = (size_t)nw * compact_heap_bytes(k);
    const int bps = knn_blocks_per_sm();
    if (bps > 0) sm = std::max(sm, (size_t)(200 * 1024) / bps);
    const bool pair = learned_kernel() != 0;
    cudaError_t e = pair ? cudaFuncSetAttribute(k_knn_lane2<D, PER, true, true>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm)
                         : cudaFuncSetAttribute(k_knn_lane2<D, PER, true>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(k_knn_lane2)");
    if (pair)
      k_knn_lane2<D, PER, true, true><<<blocks, nw * 32, sm, s>>>(
          t->view(), q, order, nq, k, sorted, dist, idx, knn_stats_buffer(), r2, miss, nmiss, qleaf);
    else
      k_knn_lane2<D, PER, true><<<blocks, nw * 32, sm, s>>>(t->view(), q, order, nq, k, sorted,
                                                            dist, idx, knn_stats_buffer(), r2,
                                                            miss, nmiss, qleaf);
    note_launch();
    e = cudaGetLastError();
    if (e != cudaSuccess) st = cuda_fail(e, "k_knn_lane2 (bounded)");
  }
  unsigned nm = 0;
  if (st == CKD_OK) {
    cudaError_t e = cudaMemcpyAsync(&nm, nmiss, sizeof(unsigned), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) st = cuda_fail(e, "reading the fallback count");
    else if ((int64_t)nm > nq) st = fail(CKD_ERR_CUDA, "internal error: fallback list overflow");
  }
  if (st == CKD_OK && nm > 0)
    st = knn_launch<D, PER>(t, q, miss, (int64_t)nm, k, sorted, dist, idx, s, 8);
  if (st == CKD_OK) timing_end(s);
  if (nfb_out) *nfb_out = nm;
  return st;
}

}  // namespace

ckd_status knn_learned(const ckd_tree* t, const ckd_mlp* net, const double* q, int64_t nq, int k,
                       int sorted, double* dist, int64_t* idx, int64_t* nfb, cudaStream_t s) {
  if (!(t->screen_ok && t->depth < kLaneStack - 1 && k <= kSmemK)) {
    if (nfb) *nfb = nq;
    return knn_run(t, q, nq, k, sorted, dist, idx, s);
  }
  switch (t->d * 2 + (t->periodic ? 1 : 0)) {
#define CKD_LB(DD)                                                                          \
  case 2 * DD: return knn_learned_impl<DD, false>(t, net, q, nq, k, sorted, dist, idx, nfb, s); \
  case 2 * DD + 1: return knn_learned_impl<DD, true>(t, net, q, nq, k, sorted, dist, idx, nfb, s);
    CKD_LB(1) CKD_LB(2) CKD_LB(3) CKD_LB(4) CKD_LB(5) CKD_LB(6) CKD_LB(7) CKD_LB(8)
#undef CKD_LB
  }
  return fail(CKD_ERR_BAD_DIM, "dimensionality must be 1..8");
}

// ===================================================================
// kNN without any device allocation (ckd_knn_noalloc)
//
// For callers that cannot allocate device memory during a search: host
// applications that reserve all device memory up front and hand nothing to the
// CUDA allocator afterwards, or latency-critical loops that cannot afford the
// implicit synchronisation of an allocation.  The query-ordering scratch of the
// search (per-query keys and the processing order, a histogram of coarse leaf
// bins and its prefix sums) lives in one file-scope device array instead of
// pool allocations; the search kernel itself needs only shared memory.
//
// Limits: at most kNoAllocMaxQ queries per call, k <= 64, tree depth < 92.
// Every call shares the array, so calls whose work overlaps on the GPU (two
// streams, or two host threads) race on it and must be serialised by the
// caller.  The first call on a device looks up the array's device address
// (cudaGetSymbolAddress, with that device current); make that first call
// before any stream capture.  The lookup is repeated when the device's current
// context changed since (cudaDeviceReset, a caller-made context), so such a call
// should also come outside a capture.  The array holds ~18 MB on every device
// that loads the library, until the process exits.
namespace {

constexpr int64_t kNoAllocMaxQ = int64_t(1) << 21;  // queries per call
constexpr int kNoAllocBins = 1 << 18;              // coarse leaf bins
constexpr size_t kNoAllocBytes =
    sizeof(int32_t) * (2 * (size_t)kNoAllocMaxQ + 2 * (size_t)kNoAllocBins + 64);

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

std::mutex g_noalloc_mu;
void* g_noalloc_ptr[64] = {nullptr};
void* g_noalloc_ctx[64] = {nullptr};

// the driver's current context (cuCtxGetCurrent, fetched through the runtime so
// the library needs no link against the driver library); null if unavailable
void* current_context() {
  using CtxFn = int (*)(void**);
  static CtxFn fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<CtxFn>(f);
  }();
  void* ctx = nullptr;
  if (!fn || fn(&ctx) != 0) return nullptr;
  return ctx;
}

// Device address of the scratch array in the current device's context, looked up
// once per device and again whenever that device's current context is another
// one than at the last lookup (after cudaDeviceReset, or when the caller made a
// context of its own current): a context's module copy of the array has its own
// address.
ckd_status noalloc_scratch(void** out) {
  int dev = 0;
  CKD_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(CKD_ERR_NO_DEVICE, "device index out of range");
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  void* ctx = current_context();
  if (!g_noalloc_ptr[dev] || !ctx || ctx != g_noalloc_ctx[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(no-allocation scratch)");
    g_noalloc_ptr[dev] = p;
    // cudaGetSymbolAddress made the primary context current if none was
    g_noalloc_ctx[dev] = ctx ? ctx : current_context();
  }
  *out = g_noalloc_ptr[dev];
  return CKD_OK;
}

// leaf of each query, binned coarsely by the leaf's first point
template <int D>
__global__ void k_locate_bins(const NodeMeta* __restrict__ meta, const double* __restrict__ Q,
                              int64_t nq, int shift, int32_t* __restrict__ key,
                              int32_t* __restrict__ hist) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nq) return;
  double q[D];
#pragma unroll
  for (int j = 0; j < D; ++j) q[j] = Q[i * D + j];
  NodeMeta m = load_meta(meta, 0);
  while (m.left >= 0) {
    double qa = 0.0;
#pragma unroll
    for (int j = 0; j < D; ++j)
      if (j == m.axis) qa = q[j];
    m = load_meta(meta, qa < m.split ? m.left : m.left + 1);
  }
  int32_t b = m.start >> shift;
  key[i] = b;
  atomicAdd(&hist[b], 1);
}

// exclusive scan of n <= kNoAllocBins counts by one block (out[n] = total)
__global__ void __launch_bounds__(1024) k_scan_one_block(const int32_t* __restrict__ in, int n,
                                                         int32_t* __restrict__ out) {
  __shared__ int32_t tmp[32];
  const int per = (n + blockDim.x - 1) / blockDim.x;
  const int b0 = threadIdx.x * per, b1 = min(n, b0 + per);
  int32_t s = 0;
  for (int i = b0; i < b1; ++i) s += in[i];
  int32_t tot;
  int32_t pre = block_exclusive_scan<int32_t, 1024>(s, tmp, tot);
  for (int i = b0; i < b1; ++i) {
    int32_t v = in[i];
    out[i] = pre;
    pre += v;
  }
  if (threadIdx.x == 0) out[n] = tot;
}

template <int D, bool PER>
ckd_status knn_noalloc_impl(const ckd_tree* t, const double* q, int64_t nq, int k, int sorted,
                            double* dist, int64_t* idx, cudaStream_t s) {
  void* base = nullptr;
  CKD_TRY(noalloc_scratch(&base));
  int32_t* order = reinterpret_cast<int32_t*>(base);
  int32_t* key = order + kNoAllocMaxQ;
  int32_t* hist = key + kNoAllocMaxQ;
  int32_t* off = hist + kNoAllocBins;
  int shift = 0;
  while ((t->n >> shift) >= kNoAllocBins) ++shift;
  const int nbins = (int)((t->n >> shift) + 1);
  CKD_CUDA(cudaMemsetAsync(hist, 0, sizeof(int32_t) * nbins, s));
  const unsigned g = (unsigned)cdiv(nq, 256);
  k_locate_bins<D><<<g, 256, 0, s>>>(t->meta, q, nq, shift, key, hist);
  CKD_LAUNCH_CHECK();
  k_scan_one_block<<<1, 1024, 0, s>>>(hist, nbins, off);
  CKD_LAUNCH_CHECK();
  CKD_CUDA(cudaMemsetAsync(hist, 0, sizeof(int32_t) * nbins, s));
  k_bucket_scatter<<<g, 256, 0, s>>>(key, nq, off, hist, order);
  CKD_LAUNCH_CHECK();
  TreeView tv = t->view();
  const int nw = 4;
  const unsigned blocks = (unsigned)cdiv(cdiv(nq, 32), nw);
  if (t->screen_ok && t->depth < kLaneStack - 1) {
    size_t sm = (size_t)nw * compact_heap_bytes(k);
    CKD_CUDA(cudaFuncSetAttribute(k_knn_lane2<D, PER, false, true>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    k_knn_lane2<D, PER, false, true><<<blocks, nw * 32, sm, s>>>(tv, q, order, nq, k, sorted, dist,
                                                                 idx, nullptr);
  } else {
    size_t sm = (size_t)nw * k * 32 * (sizeof(double) + sizeof(int32_t)) +
                (size_t)nw * kStack * sizeof(int32_t);
    CKD_CUDA(cudaFuncSetAttribute(k_knn_smem<D, PER>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sm));
    k_knn_smem<D, PER><<<blocks, nw * 32, sm, s>>>(tv, q, order, nq, k, sorted, nullptr, kStack,
                                                   dist, idx);
  }
  CKD_LAUNCH_CHECK();
  return CKD_OK;
}

}  // namespace

ckd_status knn_noalloc(const ckd_tree* t, const double* q, int64_t nq, int k, int sorted,
                       double* dist, int64_t* idx, cudaStream_t s) {
  if (nq > kNoAllocMaxQ)
    return fail(CKD_ERR_BAD_ARG, "ckd_knn_noalloc: at most 2097152 queries per call");
  if (k > kSmemK) return fail(CKD_ERR_BAD_ARG, "ckd_knn_noalloc: k must be <= 64");
  if (t->depth >= kStack - 4)
    return fail(CKD_ERR_BAD_ARG, "ckd_knn_noalloc: tree deeper than 91 levels");
  switch (t->d * 2 + (t->periodic ? 1 : 0)) {
#define CKD_NA(DD)                                                                     \
  case 2 * DD: return knn_noalloc_impl<DD, false>(t, q, nq, k, sorted, dist, idx, s); \
  case 2 * DD + 1: return knn_noalloc_impl<DD, true>(t, q, nq, k, sorted, dist, idx, s);
    CKD_NA(1) CKD_NA(2) CKD_NA(3) CKD_NA(4) CKD_NA(5) CKD_NA(6) CKD_NA(7) CKD_NA(8)
#undef CKD_NA
  }
  return fail(CKD_ERR_BAD_DIM, "dimensionality must be 1..8");
}

}  // namespace ckd