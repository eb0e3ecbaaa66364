// build.cu -- level-synchronous sliding-midpoint k-d tree construction on one GPU.
//
// Restates the recursion of src/cosmokdtree.f90:286-451 breadth-first: every
// level processes all open nodes of all sizes at once.
//
//   k_seg_box     per-node bounding box of the open nodes (segmented min/max)
//   k_decide      axis (longest cell side, spread tie-break), midpoint, slide mode
//   k_flags       left flag per position of a midpoint split, per-tile sums and
//                 segment-end prefixes; slide point of a sliding split = first
//                 position holding the extreme (atomicMin)
//   scan          tile offsets
//   k_children    n_left per node, child pairs, child cells, next open list
//   k_scatter     stable out-of-place partition into the other buffer; points of
//                 closed children land in the final leaf-ordered arrays
//   k_finish      (after the levels) every closed node of more than `leaf` points:
//                 its whole subtree by one block in shared memory
//
// The levels close a node at finish_max(D) points (or at `leaf`, when that is more),
// which is what "leaf" means in their kernels.
//
// The working set of a level holds only the points of open nodes (more than
// `leaf` points), compacted into SoA ping-pong buffers X[2][d][n] (stride n):
// open node a owns working positions [wst[a], wst[a] + count), in the order of
// its final leaf-ordered range [start, start + count), and every position
// carries its node's id (NID).  A point whose child is a leaf goes straight to
// its final place in the leaf-ordered arrays and leaves the working set, so the
// per-level passes touch only the points still being split.  The partition is
// stable, so every segment stays sorted by original index and "first
// occurrence" (Fortran minloc/maxloc, cosmokdtree.f90:372-373) is the lowest
// index holding the extreme.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ckd_common.cuh"
#include "ckd_scan.cuh"

namespace ckd {

namespace {

constexpr int kBT = 256;          // threads per tile kernel
constexpr int kItems = 8;         // passes per tile
constexpr int kTile = kBT * kItems;
constexpr int kMaxLevels = 8192;  // depth guard (degenerate duplicate clusters peel one point per level)

// What the flag pass needs of an open node, in one 32-byte record.
struct __align__(16) FlagRec {
  double split;
  int32_t axis, md, wst, count;
  int32_t pad[2];
};

// What the scatter needs of an open node, in two int4: {start, wst, nleft, count}
// and {pbase (midpoint split) or slide point, left child, working start of the
// left / right child or -1 for a leaf child, -2 for the slide point's leaf}.
struct BuildBufs {
  int d = 0;
  int64_t n = 0;
  // one block holds every buffer below; only arrays that had to grow leave it
  char* arena = nullptr;
  size_t arena_bytes = 0;
  bool outside(const void* p) const {
    return p && !(static_cast<const char*>(p) >= arena && static_cast<const char*>(p) < arena + arena_bytes);
  }
  double* X[2] = {nullptr, nullptr};
  int32_t* I[2] = {nullptr, nullptr};
  int32_t* NID[2] = {nullptr, nullptr};
  // per node of the finished tree (capacity tcap)
  int64_t tcap = 0;
  NodeMeta* meta = nullptr;
  double* cell = nullptr;
  double* box = nullptr;
  // per node of the level passes (capacity cap)
  int64_t cap = 0;
  unsigned long long* keys = nullptr;  // [cap][2d] ordered min/max keys
  int32_t* ext = nullptr;              // slide point position
  int32_t* mode = nullptr;             // 0 midpoint, 1 slide left, 2 slide right
  int32_t* pstart = nullptr;           // local exclusive prefix at segment start
  int32_t* pend = nullptr;             // local inclusive prefix at segment end
  int32_t* nleft = nullptr;
  int32_t* pbase = nullptr;
  int32_t* wst = nullptr;              // first working position of an open node
  FlagRec* frec = nullptr;
  int4* srec = nullptr;                // [cap][2]
  // per level
  int32_t* act[2] = {nullptr, nullptr};
  // per open node: (open children << 32) | points of the open children, and
  // the exclusive prefix of that (next list slot, next working start)
  int64_t* nxt_cnt = nullptr;
  int64_t* nxt_off = nullptr;
  int32_t* tile_sum = nullptr;
  int32_t* tile_off = nullptr;
  unsigned* flags = nullptr;  // left flags of the working positions, one bit each
  int32_t* scal = nullptr;  // device scalars: [0] next open count, [1] error flag
  // level state {open nodes, working points, nodes so far, levels with open nodes},
  // double-buffered: a level reads lst[p] and its last node kernel writes lst[1-p]
  int4* lst = nullptr;
};

// ------------------------------------------------------------------ kernels

// row-major (n x d) FP64/FP32 -> SoA FP64.  Tree t of a forest owns positions
// [off[t], off[t+1]) and is rooted at node t; ids are local to their tree
// (0..n_t-1), NID[0] = the tree's root, NID[1] = -1.  off == nullptr: one tree.
template <typename T>
__global__ void k_init_points(const T* __restrict__ in, int64_t n, int d, double* __restrict__ X,
                              int32_t* __restrict__ I, int32_t* __restrict__ N0,
                              int32_t* __restrict__ N1, const int64_t* __restrict__ off,
                              int32_t n_trees) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  for (int j = 0; j < d; ++j) X[(int64_t)j * n + p] = (double)in[p * d + j];
  int32_t t = 0;
  if (off) {  // last tree with off[t] <= p
    int32_t lo = 0, hi = n_trees - 1;
    while (lo < hi) {
      int32_t mid = (lo + hi + 1) >> 1;
      if (off[mid] <= p) lo = mid;
      else hi = mid - 1;
    }
    t = lo;
  }
  I[p] = (int32_t)(p - (off ? off[t] : 0));
  N0[p] = t;
  N1[p] = -1;
}

// Working set of the first level when some roots are already leaves: the points
// of the open roots, compacted in tree order (wst[t] = -1 for a leaf root).
template <int D>
__global__ void k_compact_roots(const double* __restrict__ X, const int32_t* __restrict__ I,
                                const int32_t* __restrict__ NID, const int32_t* __restrict__ wst,
                                const int64_t* __restrict__ off, int64_t n,
                                double* __restrict__ Xo, int32_t* __restrict__ Io,
                                int32_t* __restrict__ NIDo) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int32_t t = NID[p];
  const int32_t w0 = wst[t];
  if (w0 < 0) return;
  const int64_t w = w0 + (p - off[t]);
#pragma unroll
  for (int j = 0; j < D; ++j) Xo[(int64_t)j * n + w] = X[(int64_t)j * n + p];
  Io[w] = I[p];
  NIDo[w] = t;
}

// minimum of a 64-bit key over the warp
__device__ __forceinline__ unsigned long long warp_min_key(unsigned long long k) {
  const unsigned hi = (unsigned)(k >> 32);
  const unsigned mh = __reduce_min_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_min_sync(0xffffffffu, hi == mh ? (unsigned)k : 0xffffffffu);
  return ((unsigned long long)mh << 32) | ml;
}

// Whether a tile of working positions is full and lies in one node: a node's positions
// are contiguous, so equal ids at both ends are enough.  True for most tiles while
// nodes hold many tiles; the box, flag and scatter passes then do not read the ids,
// and the first two need no segments (2^24 clustered points, all levels: boxes 2340 ->
// 1670 us, flags 977 -> 740 us, 28 -> 24 and 12 -> 8 bytes a point).
__device__ __forceinline__ bool tile_of_one_node(const int32_t* __restrict__ NID, int64_t base,
                                                 int64_t nw) {
  return base + kTile <= nw && __ldg(NID + base) == __ldg(NID + base + kTile - 1);
}

// Segmented min/max over the working positions.  Tiles of one node (all of them while
// nodes are large) take a plain reduction without reading the ids.  Else each thread reduces kItems
// consecutive positions in registers; one segmented warp scan per dimension
// joins the pieces of runs that cross thread boundaries.  Runs that end
// inside a warp chunk go straight to atomicMin/atomicMax; the first and last
// run of every warp chunk are merged per block by thread 0.
template <int D>
__global__ void __launch_bounds__(kBT, 5) k_seg_box(const double* __restrict__ X,
                                                 const int32_t* __restrict__ NID,
                                                 int64_t n, int64_t nw,
                                                 unsigned long long* __restrict__ keys,
                                                 const int4* __restrict__ st = nullptr) {
  constexpr int W = kBT / 32;
  __shared__ int32_t rec_id[W][2];
  __shared__ unsigned long long rec_v[W][2][2 * D];
  if (st) nw = st->y;  // working points of this level (device state)
  const int64_t base = (int64_t)blockIdx.x * kTile;
  if (base >= nw) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (tile_of_one_node(NID, base, nw) && (n & 1) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0) {
    // whole tile in one node (its positions are contiguous): no ids, no segments;
    // coordinates in coalesced pairs
    unsigned long long kmn[D], kmx[D];  // minima of the keys and of their complements
#pragma unroll
    for (int j = 0; j < D; ++j) {
      const ulonglong2* __restrict__ Xj =
          reinterpret_cast<const ulonglong2*>(X + (int64_t)j * n + base) + threadIdx.x;
      kmn[j] = kmx[j] = ~0ull;
#pragma unroll
      for (int i = 0; i < kItems / 2; ++i) {
        const ulonglong2 v = __ldg(Xj + i * kBT);
        const unsigned long long k0 = dkey_bits(v.x), k1 = dkey_bits(v.y);
        const unsigned long long mn = k0 < k1 ? k0 : k1, mx = ~(k0 < k1 ? k1 : k0);
        kmn[j] = mn < kmn[j] ? mn : kmn[j];
        kmx[j] = mx < kmx[j] ? mx : kmx[j];
      }
    }
#pragma unroll
    for (int j = 0; j < D; ++j) {
      const unsigned long long mn = warp_min_key(kmn[j]), mx = warp_min_key(kmx[j]);
      if (lane == 0) {
        rec_v[w][0][2 * j] = mn;
        rec_v[w][0][2 * j + 1] = mx;
      }
    }
    __syncthreads();
    if (threadIdx.x < 2 * D) {
      unsigned long long v = rec_v[0][0][threadIdx.x];
#pragma unroll
      for (int x = 1; x < W; ++x) v = rec_v[x][0][threadIdx.x] < v ? rec_v[x][0][threadIdx.x] : v;
      unsigned long long* k = &keys[(int64_t)NID[base] * 2 * D + threadIdx.x];
      if (threadIdx.x & 1) atomicMax(k, ~v);
      else atomicMin(k, v);
    }
    return;
  }
  const int64_t p0 = (int64_t)blockIdx.x * kTile + (int64_t)threadIdx.x * kItems;
  // node of every position (-1 past the working set), run breaks inside the thread
  static_assert(kItems == 8, "two int4 / four double2 loads per thread");
  int32_t a[kItems];
  // vector loads when the thread's 8 positions are all working positions and
  // aligned (NID from the pool; X rows start at j * n, even for even n)
  const bool full = p0 + kItems <= nw;
  const bool vec = full && (n & 1) == 0 && (reinterpret_cast<uintptr_t>(NID) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  if (vec) {
    const int4 u = __ldg(reinterpret_cast<const int4*>(NID + p0));
    const int4 v = __ldg(reinterpret_cast<const int4*>(NID + p0) + 1);
    a[0] = u.x, a[1] = u.y, a[2] = u.z, a[3] = u.w, a[4] = v.x, a[5] = v.y, a[6] = v.z, a[7] = v.w;
  } else {
#pragma unroll
    for (int i = 0; i < kItems; ++i) a[i] = p0 + i < nw ? NID[p0 + i] : -1;
  }
  unsigned brk = 0;
#pragma unroll
  for (int i = 1; i < kItems; ++i) brk |= (a[i] != a[i - 1]) ? (1u << i) : 0u;
  const int32_t hd = a[0], tl = a[kItems - 1];
  const bool single = brk == 0;
  // scan steps that stay inside the tail run (equal ids of open nodes are contiguous)
  unsigned take = 0;
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int32_t au = __shfl_up_sync(0xffffffffu, tl, 1 << s);
    take |= (lane >= (1 << s) && au == tl) ? (1u << s) : 0u;
  }
  const int32_t prev_tl = __shfl_up_sync(0xffffffffu, tl, 1);
  const int32_t next_hd = __shfl_down_sync(0xffffffffu, hd, 1);
  const int32_t first_id = __shfl_sync(0xffffffffu, hd, 0);
  const bool join_prev = lane > 0 && prev_tl == hd;  // head run continues the previous lane's tail
  const bool tail_end = lane == 31 || next_hd != tl;
#pragma unroll 1
  for (int j = 0; j < D; ++j) {
    // coordinates read as raw 64-bit patterns (NaNs keep their bits)
    const unsigned long long* __restrict__ Xj =
        reinterpret_cast<const unsigned long long*>(X) + (int64_t)j * n;
    unsigned long long kk[kItems];
    if (vec) {
#pragma unroll
      for (int h = 0; h < kItems / 2; ++h) {
        const ulonglong2 x = __ldg(reinterpret_cast<const ulonglong2*>(Xj + p0) + h);
        kk[2 * h] = dkey_bits(x.x);
        kk[2 * h + 1] = dkey_bits(x.y);
      }
    } else {
#pragma unroll
      for (int i = 0; i < kItems; ++i) kk[i] = a[i] >= 0 ? dkey_bits(Xj[p0 + i]) : 0ull;
    }
    unsigned long long hmn = kk[0], hmx = kk[0], cmn = kk[0], cmx = kk[0];
    int32_t ca = a[0];
    bool head_open = true;
#pragma unroll
    for (int i = 1; i < kItems; ++i) {
      if (brk & (1u << i)) {
        if (head_open) {
          hmn = cmn;
          hmx = cmx;
          head_open = false;
        } else if (ca >= 0) {  // a run that starts and ends inside this thread
          atomicMin(&keys[(int64_t)ca * 2 * D + 2 * j], cmn);
          atomicMax(&keys[(int64_t)ca * 2 * D + 2 * j + 1], cmx);
        }
        ca = a[i];
        cmn = kk[i];
        cmx = kk[i];
      } else {
        cmn = kk[i] < cmn ? kk[i] : cmn;
        cmx = kk[i] > cmx ? kk[i] : cmx;
      }
    }
    // segmented inclusive scan of the tail runs
#pragma unroll
    for (int s = 0; s < 5; ++s) {
      const unsigned long long u = __shfl_up_sync(0xffffffffu, cmn, 1 << s);
      const unsigned long long v = __shfl_up_sync(0xffffffffu, cmx, 1 << s);
      if (take & (1u << s)) {
        cmn = u < cmn ? u : cmn;
        cmx = v > cmx ? v : cmx;
      }
    }
    const unsigned long long pmn = __shfl_up_sync(0xffffffffu, cmn, 1);
    const unsigned long long pmx = __shfl_up_sync(0xffffffffu, cmx, 1);
    // run ends: the head run when it ends inside this thread, the tail run when
    // the next lane starts another node (or at the end of the chunk)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      int32_t id;
      unsigned long long mn, mx;
      bool is_end;
      if (e == 0) {
        is_end = !single;
        id = hd;
        mn = hmn;
        mx = hmx;
        if (join_prev) {
          mn = pmn < mn ? pmn : mn;
          mx = pmx > mx ? pmx : mx;
        }
      } else {
        is_end = tail_end;
        id = tl;
        mn = cmn;
        mx = cmx;
      }
      if (!is_end) continue;
      if (id == first_id) {
        if (j == 0) rec_id[w][0] = id;
        rec_v[w][0][2 * j] = mn;
        rec_v[w][0][2 * j + 1] = mx;
        if (lane == 31 && e == 1 && j == 0) rec_id[w][1] = -2;  // one run spans the chunk
      } else if (e == 1 && lane == 31) {
        if (j == 0) rec_id[w][1] = id;
        rec_v[w][1][2 * j] = mn;
        rec_v[w][1][2 * j + 1] = mx;
      } else if (id >= 0) {
        atomicMin(&keys[(int64_t)id * 2 * D + 2 * j], mn);
        atomicMax(&keys[(int64_t)id * 2 * D + 2 * j + 1], mx);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int32_t cur = -1;
    unsigned long long v[2 * D];
    auto flush = [&]() {
      if (cur >= 0) {
#pragma unroll
        for (int j = 0; j < D; ++j) {
          atomicMin(&keys[(int64_t)cur * 2 * D + 2 * j], v[2 * j]);
          atomicMax(&keys[(int64_t)cur * 2 * D + 2 * j + 1], v[2 * j + 1]);
        }
      }
    };
    for (int c = 0; c < W; ++c) {
      for (int r = 0; r < 2; ++r) {
        const int32_t id = rec_id[c][r];
        if (id == -2) continue;  // no separate last run
        if (id == cur) {
#pragma unroll
          for (int j = 0; j < D; ++j) {
            v[2 * j] = rec_v[c][r][2 * j] < v[2 * j] ? rec_v[c][r][2 * j] : v[2 * j];
            v[2 * j + 1] = rec_v[c][r][2 * j + 1] > v[2 * j + 1] ? rec_v[c][r][2 * j + 1] : v[2 * j + 1];
          }
        } else {
          flush();
          cur = id;
#pragma unroll
          for (int j = 0; j < 2 * D; ++j) v[j] = rec_v[c][r][j];
        }
      }
    }
    flush();
  }
}

// The split of a node with tight box [lo, hi] and cell [clo, chi]
// (cosmokdtree.f90:347-410): axis, splitting value and mode (0 midpoint, 1 slide
// left, 2 slide right).
template <int D>
__device__ __forceinline__ void split_rule(const double (&lo)[D], const double (&hi)[D],
                                           const double (&clo)[D], const double (&chi)[D],
                                           int& axis, double& mid, int& md) {
  // longest cell side; exact ties go to the larger data spread (:355-365)
  double maxside = dsub(chi[0], clo[0]);
  double spread = dsub(hi[0], lo[0]);
  double cl = clo[0], ch = chi[0], minx = lo[0], maxx = hi[0];
  axis = 0;
#pragma unroll
  for (int j = 1; j < D; ++j) {
    const double side = dsub(chi[j], clo[j]), sp = dsub(hi[j], lo[j]);
    if (side > maxside || (side == maxside && sp > spread)) {
      maxside = side;
      spread = sp;
      axis = j;
      cl = clo[j];
      ch = chi[j];
      minx = lo[j];
      maxx = hi[j];
    }
  }
  mid = dmul(0.5, dadd(cl, ch));  // :367
  md = 0;
  if (minx >= mid) {  // :376
    mid = minx;
    md = 1;
  } else if (maxx < mid) {  // :391
    mid = maxx;
    md = 2;
  }
}

// Split decision per open node (cosmokdtree.f90:347-410).
template <int D>
__global__ void k_decide(const int32_t* __restrict__ act, const int4* __restrict__ st,
                         NodeMeta* __restrict__ meta,
                         double* __restrict__ cell, double* __restrict__ box,
                         const unsigned long long* __restrict__ keys, int32_t* __restrict__ mode,
                         int32_t* __restrict__ ext, const int32_t* __restrict__ wst,
                         FlagRec* __restrict__ frec) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= st->x) return;
  int32_t a = act[i];
  double lo[D], hi[D], clo[D], chi[D];
#pragma unroll
  for (int j = 0; j < D; ++j) {
    lo[j] = dkey_inv(keys[(int64_t)a * 2 * D + 2 * j]);
    hi[j] = dkey_inv(keys[(int64_t)a * 2 * D + 2 * j + 1]);
    box[(int64_t)a * 2 * D + 2 * j] = lo[j];
    box[(int64_t)a * 2 * D + 2 * j + 1] = hi[j];
  }
#pragma unroll
  for (int j = 0; j < D; ++j) {
    clo[j] = cell[(int64_t)a * 2 * D + 2 * j];
    chi[j] = cell[(int64_t)a * 2 * D + 2 * j + 1];
  }
  int axis, md;
  double mid;
  split_rule<D>(lo, hi, clo, chi, axis, mid, md);
  meta[a].split = mid;
  meta[a].axis = axis;
  mode[a] = md;
  ext[a] = 0x7fffffff;
  FlagRec r;
  r.split = mid;
  r.axis = axis;
  r.md = md;
  r.wst = wst[a];
  r.count = meta[a].count;
  r.pad[0] = r.pad[1] = 0;
  frec[a] = r;
}

// Exclusive prefix, in position order, of one tile's 0/1 flags, visited as
// p = base + it * kBT + threadIdx.x: msk[it] is the warp's ballot of pass it.
// Leaves in cpre[it * W + w] the offset of warp w's 32 positions of pass it and
// returns the tile total.  Two barriers per tile.
__device__ __forceinline__ int32_t tile_chunk_prefix(const unsigned (&msk)[kItems],
                                                     int32_t* cpre) {
  constexpr int W = kBT / 32, NC = kItems * W;
  static_assert(NC == 64, "two warp chunks per lane in the chunk scan");
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) {
#pragma unroll
    for (int it = 0; it < kItems; ++it) cpre[it * W + w] = __popc(msk[it]);
  }
  __syncthreads();
  if (w == 0) {
    const int32_t x0 = cpre[2 * lane], x1 = cpre[2 * lane + 1], s = x0 + x1;
    const int32_t inc = warp_inclusive_scan(s);
    cpre[2 * lane] = inc - s;
    cpre[2 * lane + 1] = inc - s + x0;
    if (lane == 31) cpre[NC] = inc;
  }
  __syncthreads();
  return cpre[NC];
}

// Per-tile left counts and the segment-start / segment-end local prefixes of the
// midpoint splits (x < split goes left, cosmokdtree.f90:470).  A sliding split
// sends exactly one point, the first holding the extreme (:376-403), to the
// side that would be empty; its positions count 0 here and record that point.
// Each thread takes 8 consecutive positions (vector loads of the node ids and,
// when they all belong to one node, of that node's split coordinate), so the
// chain node id -> split record -> coordinate costs three loads per thread
// instead of three per position.  The left flags go to a bitmap (bit p & 31 of
// word p >> 5) that the scatter reads back.
__global__ void __launch_bounds__(kBT) k_flags(const double* __restrict__ X,
                                               const int32_t* __restrict__ NID,
                                               const FlagRec* __restrict__ frec,
                                               int32_t* __restrict__ ext, int64_t n,
                                               const int4* __restrict__ st,
                                               int32_t* __restrict__ tile_sum,
                                               int32_t* __restrict__ pstart,
                                               int32_t* __restrict__ pend,
                                               unsigned* __restrict__ flags) {
  static_assert(kItems == 8, "8 consecutive positions per thread");
  __shared__ int32_t tmp[kBT / 32];
  const int64_t nw = st->y;
  if ((int64_t)blockIdx.x * kTile >= nw) {  // past this level's working set
    if (threadIdx.x == 0) tile_sum[blockIdx.x] = 0;
    return;
  }
  const int lane = threadIdx.x & 31;
  const int64_t base = (int64_t)blockIdx.x * kTile;
  if (tile_of_one_node(NID, base, nw)) {
    // one split for the whole tile: 32 consecutive positions a warp and pass, whose
    // ballot is a word of the bitmap; the node starts or ends here only at the tile's
    // own ends
    const int w = threadIdx.x >> 5;
    const int32_t a1 = __ldg(NID + base);
    const FlagRec r = frec[a1];
    const double* __restrict__ xr = X + (int64_t)r.axis * n + base + threadIdx.x;
    double x[kItems];
#pragma unroll
    for (int i = 0; i < kItems; ++i) x[i] = __ldg(xr + i * kBT);
    int32_t sum = 0;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const unsigned word = __ballot_sync(0xffffffffu, r.md == 0 && x[i] < r.split);
      if (r.md != 0 && x[i] == r.split)
        atomicMin(&ext[a1], (int32_t)(base + i * kBT + threadIdx.x));
      if (lane == 0) flags[(base >> 5) + i * (kBT / 32) + w] = word;
      sum += __popc(word);
    }
    if (lane == 0) tmp[w] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
      int32_t tot = 0;
#pragma unroll
      for (int i = 0; i < kBT / 32; ++i) tot += tmp[i];
      tile_sum[blockIdx.x] = tot;
      if (r.wst == base) pstart[a1] = 0;
      if (r.wst + r.count == base + kTile) pend[a1] = tot;
    }
    return;
  }
  const int64_t p0 = base + (int64_t)threadIdx.x * kItems;
  int32_t a[kItems];
  const bool full = p0 + kItems <= nw;
  const bool vec = full && (n & 1) == 0 && (reinterpret_cast<uintptr_t>(NID) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(X) & 15) == 0;
  if (vec) {
    const int4 u = __ldg(reinterpret_cast<const int4*>(NID + p0));
    const int4 v = __ldg(reinterpret_cast<const int4*>(NID + p0) + 1);
    a[0] = u.x, a[1] = u.y, a[2] = u.z, a[3] = u.w, a[4] = v.x, a[5] = v.y, a[6] = v.z, a[7] = v.w;
  } else {
#pragma unroll
    for (int i = 0; i < kItems; ++i) a[i] = p0 + i < nw ? NID[p0 + i] : -1;
  }
  bool single = a[0] >= 0;
#pragma unroll
  for (int i = 1; i < kItems; ++i) single = single && a[i] == a[0];
  unsigned f8 = 0, se = 0;  // left flags; segment start (bit 2i) and end (bit 2i+1)
  auto one = [&](int i, const FlagRec& r, double x) {
    const int64_t p = p0 + i;
    if (r.md == 0) f8 |= (x < r.split ? 1u : 0u) << i;
    else if (x == r.split) atomicMin(&ext[a[i]], (int32_t)p);
    if (p == r.wst) se |= 1u << (2 * i);
    if (p == (int64_t)r.wst + r.count - 1) se |= 2u << (2 * i);
  };
  if (single && vec) {
    const FlagRec r = frec[a[0]];
    const double2* xr = reinterpret_cast<const double2*>(X + (int64_t)r.axis * n + p0);
#pragma unroll
    for (int h = 0; h < kItems / 2; ++h) {
      const double2 x = __ldg(xr + h);
      one(2 * h, r, x.x);
      one(2 * h + 1, r, x.y);
    }
  } else {
    FlagRec r;
    int32_t ra = -1;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      if (a[i] < 0) continue;
      if (a[i] != ra) {
        r = frec[a[i]];
        ra = a[i];
      }
      one(i, r, X[(int64_t)r.axis * n + p0 + i]);
    }
  }
  int32_t tot;
  const int32_t ex = block_exclusive_scan<int32_t, kBT>(__popc(f8), tmp, tot);
  if (se) {
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const unsigned b = (se >> (2 * i)) & 3u;
      if (b == 0) continue;
      const int32_t e = ex + __popc(f8 & ((1u << i) - 1u));
      if (b & 1u) pstart[a[i]] = e;
      if (b & 2u) pend[a[i]] = e + (int32_t)((f8 >> i) & 1u);
    }
  }
  // 4 lanes (32 positions) per bitmap word
  unsigned word = f8 << (8 * (lane & 3));
  word |= __shfl_xor_sync(0xffffffffu, word, 1);
  word |= __shfl_xor_sync(0xffffffffu, word, 2);
  if ((lane & 3) == 0) flags[p0 >> 5] = word;
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = tot;
}

// One open node's left count and its children's records (cosmokdtree.f90:412-448);
// returns the left count and leaves the node's prefix base in P0.
template <int D>
__device__ __forceinline__ int32_t make_children(
    int32_t a, int32_t c0, const NodeMeta& pm, NodeMeta* meta, double* cell,
    const int32_t* __restrict__ pstart, const int32_t* __restrict__ pend, const int32_t* tile_off,
    int32_t w0, int md, int32_t ext, unsigned long long* __restrict__ keys, int32_t* err,
    int32_t& P0) {
  int32_t nl;
  P0 = 0;
  if (md == 0) {
    int64_t s = w0, e = (int64_t)w0 + pm.count - 1;
    P0 = tile_off[s / kTile] + pstart[a];
    nl = tile_off[e / kTile] + pend[a] - P0;
  } else {
    nl = md == 1 ? 1 : pm.count - 1;
    if (ext == 0x7fffffff) nl = 0;  // no slide point found: flagged below
  }
  if (nl <= 0 || nl >= pm.count) {  // cannot happen for a valid sliding-midpoint split
    atomicExch(err, 1);
    nl = nl <= 0 ? 1 : pm.count - 1;
  }
  meta[a].left = c0;
  for (int side = 0; side < 2; ++side) {
    int32_t c = c0 + side;
    NodeMeta cm;
    cm.split = 0.0;
    cm.left = -1;
    cm.axis = -1;
    cm.start = side == 0 ? pm.start : pm.start + nl;
    cm.count = side == 0 ? nl : pm.count - nl;
    cm.depth = pm.depth + 1;
    cm.parent = a;
    meta[c] = cm;
#pragma unroll
    for (int j = 0; j < D; ++j) {  // :419-422
      double lo = cell[(int64_t)a * 2 * D + 2 * j], hi = cell[(int64_t)a * 2 * D + 2 * j + 1];
      if (j == pm.axis) {
        if (side == 0) hi = pm.split;
        else lo = pm.split;
      }
      cell[(int64_t)c * 2 * D + 2 * j] = lo;
      cell[(int64_t)c * 2 * D + 2 * j + 1] = hi;
      keys[(int64_t)c * 2 * D + 2 * j] = ~0ull;
      keys[(int64_t)c * 2 * D + 2 * j + 1] = 0ull;
    }
  }
  return nl;
}

// n_left, child pairs and cells; counts the next open list and its working points
template <int D>
__global__ void k_children(const int32_t* __restrict__ act, const int4* __restrict__ st, int mb,
                           NodeMeta* __restrict__ meta,
                           double* __restrict__ cell, const int32_t* __restrict__ pstart,
                           const int32_t* __restrict__ pend, const int32_t* __restrict__ tile_off,
                           const int32_t* __restrict__ wst, const int32_t* __restrict__ mode,
                           const int32_t* __restrict__ ext, int32_t* __restrict__ nleft,
                           int32_t* __restrict__ pbase, unsigned long long* __restrict__ keys,
                           int leaf, int64_t* __restrict__ nxt_cnt, int32_t* __restrict__ err) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int m = st->x;
  if (i >= m) {  // zeros up to the launch bound, so the scan over mb entries is exact
    if (i < mb) nxt_cnt[i] = 0;
    return;
  }
  const int32_t a = act[i];
  const NodeMeta pm = meta[a];
  int32_t P0;
  const int32_t nl = make_children<D>(a, st->z + 2 * i, pm, meta, cell, pstart, pend, tile_off,
                                      wst[a], mode[a], ext[a], keys, err, P0);
  nleft[a] = nl;
  pbase[a] = P0;
  const int nr = pm.count - nl;
  const int cnt = (nl > leaf ? 1 : 0) + (nr > leaf ? 1 : 0);
  const int pts = (nl > leaf ? nl : 0) + (nr > leaf ? nr : 0);
  nxt_cnt[i] = ((int64_t)cnt << 32) | (int64_t)pts;
}

// The node work of a level between the flags and the scatter, by one block: the scan
// of the tiles' left counts, the children, the next open list, its working starts
// and the scatter records.  With at most a few thousand open nodes five launches of
// almost idle kernels (24 us and their gaps) cost more than one busy block (with the
// records of the tree written by two kernels and one block of memory for all of the
// build: 20011 clustered points 658 -> 573 us, 2^24 12.66 -> 12.24 ms); past kNodesMax
// nodes the parallel kernels are taken.
constexpr int kNodesT = 1024;
constexpr int kNodesMax = 4096;      // open nodes of a level (its launch bound)
constexpr unsigned kNodesTiles = 32768;
template <int D>
__global__ void __launch_bounds__(kNodesT) k_level_nodes(
    const int32_t* __restrict__ act, const int4* __restrict__ st, int4* __restrict__ st_next,
    int ntw, NodeMeta* meta, double* cell, const int32_t* __restrict__ pstart,
    const int32_t* __restrict__ pend, const int32_t* __restrict__ tile_sum, int32_t* tile_off,
    int32_t* wst, const int32_t* __restrict__ mode, const int32_t* __restrict__ ext,
    unsigned long long* __restrict__ keys, int leaf, int32_t* __restrict__ nxt,
    int4* __restrict__ srec, int32_t* err) {
  __shared__ int32_t tmp[kNodesT / 32];
  __shared__ int64_t tmp2[kNodesT / 32];
  const int tid = threadIdx.x;
  const int4 cs = *st;
  const int m = cs.x;
  {  // tile offsets
    const int used = (int)min((int64_t)ntw, ((int64_t)cs.y + kTile - 1) / kTile);
    const int per = (used + kNodesT - 1) / kNodesT;
    const int b0 = min(used, tid * per), b1 = min(used, b0 + per);
    int32_t s = 0;
    for (int i = b0; i < b1; ++i) s += tile_sum[i];
    int32_t tot;
    int32_t pre = block_exclusive_scan<int32_t, kNodesT>(s, tmp, tot);
    for (int i = b0; i < b1; ++i) {
      const int32_t v = tile_sum[i];
      tile_off[i] = pre;
      pre += v;
    }
  }
  __syncthreads();
  int64_t done = 0;  // (open children << 32) | their points, of the nodes before this pass
  for (int i0 = 0; i0 < m; i0 += kNodesT) {
    const int i = i0 + tid;
    int32_t a = 0, nl = 0, nr = 0, P0 = 0, w0 = 0, e = 0, c0 = 0;
    int md = 0;
    int4 r0 = make_int4(0, 0, 0, 0);
    if (i < m) {
      a = act[i];
      c0 = cs.z + 2 * i;
      const NodeMeta pm = meta[a];
      md = mode[a];
      e = ext[a];
      w0 = wst[a];
      nl = make_children<D>(a, c0, pm, meta, cell, pstart, pend, tile_off, w0, md, e, keys, err, P0);
      nr = pm.count - nl;
      r0 = make_int4(pm.start, w0, nl, pm.count);
    }
    const bool ol = nl > leaf, orr = nr > leaf;
    const int64_t v = ((int64_t)((ol ? 1 : 0) + (orr ? 1 : 0)) << 32) |
                      (int64_t)((ol ? nl : 0) + (orr ? nr : 0));
    int64_t tot;
    const int64_t at = done + block_exclusive_scan<int64_t, kNodesT>(v, tmp2, tot);
    done += tot;
    if (i < m) {
      int32_t o = (int32_t)(at >> 32), w = (int32_t)(at & 0xffffffffll);
      int32_t wl = md == 1 ? -2 : -1, wr = md == 2 ? -2 : -1;
      if (ol) {
        nxt[o++] = c0;
        wst[c0] = w;
        wl = w;
        w += nl;
      }
      if (orr) {
        nxt[o] = c0 + 1;
        wst[c0 + 1] = w;
        wr = w;
      }
      srec[2 * (int64_t)a] = r0;
      srec[2 * (int64_t)a + 1] = make_int4(md == 0 ? P0 : e, c0, wl, wr);
    }
  }
  if (tid == 0)
    *st_next = make_int4((int32_t)(done >> 32), (int32_t)(done & 0xffffffffll), cs.z + 2 * m,
                         cs.w + (m > 0 ? 1 : 0));
}

// next open list (children in list order, so in leaf order) and their working starts
__global__ void k_next_list(const int32_t* __restrict__ act, const int4* __restrict__ st,
                            int4* __restrict__ st_next, int mb,
                            const NodeMeta* __restrict__ meta,
                            const int64_t* __restrict__ nxt_off, int leaf,
                            const int32_t* __restrict__ mode, const int32_t* __restrict__ ext,
                            const int32_t* __restrict__ nleft, const int32_t* __restrict__ pbase,
                            int32_t* __restrict__ nxt, int32_t* __restrict__ wst,
                            int4* __restrict__ srec) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int4 cs = *st;
  const int m = cs.x;
  if (i == 0) {  // the next level's state
    const int64_t tot = nxt_off[mb];
    *st_next = make_int4((int32_t)(tot >> 32), (int32_t)(tot & 0xffffffffll), cs.z + 2 * m,
                         cs.w + (m > 0 ? 1 : 0));
  }
  if (i >= m) return;
  const int32_t a = act[i];
  const NodeMeta pm = meta[a];
  const int32_t c0 = pm.left;
  int32_t o = (int32_t)(nxt_off[i] >> 32), w = (int32_t)(nxt_off[i] & 0xffffffffll);
  const int32_t n0 = meta[c0].count, n1 = meta[c0 + 1].count;
  const int md = mode[a];
  int32_t wl = md == 1 ? -2 : -1, wr = md == 2 ? -2 : -1;
  if (n0 > leaf) {
    nxt[o++] = c0;
    wst[c0] = w;
    wl = w;
    w += n0;
  }
  if (n1 > leaf) {
    nxt[o] = c0 + 1;
    wst[c0 + 1] = w;
    wr = w;
  }
  srec[2 * (int64_t)a] = make_int4(pm.start, wst[a], nleft[a], pm.count);
  srec[2 * (int64_t)a + 1] = make_int4(md == 0 ? pbase[a] : ext[a], c0, wl, wr);
}

// bulk asynchronous copies (global -> this CTA's shared memory) completing on an
// mbarrier; every wait is bounded
constexpr unsigned kBarWaitLimit = 1u << 24;
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ bool bar_wait0(uint32_t bar) {
  for (unsigned it = 0; it < kBarWaitLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P1;\n\t}" : "=r"(done) : "r"(bar), "r"(0u) : "memory");
    if (done) return true;
  }
  return false;
}

// scatter tile staging: dynamic shared memory of the staged scatter
__host__ __device__ constexpr size_t scatter_smem(int d) {
  return (size_t)d * kTile * sizeof(double) + (size_t)kTile * sizeof(int32_t);
}

// Stable partition of every open segment: points of open children go to the
// next working set, points of new leaves to the final leaf-ordered arrays.
// STAGED: the tile's coordinate rows and ids are brought into shared memory by
// bulk asynchronous copies issued at the start (one per row, 16-byte aligned
// because the working rows have an even stride), overlapping the first pass and
// the tile scan; the second pass then reads them from shared memory.
template <int D, bool STAGED>
__global__ void __launch_bounds__(kBT) k_scatter(
    const double* __restrict__ X, const int32_t* __restrict__ I, const int32_t* __restrict__ NID,
    const int4* __restrict__ srec, const int32_t* __restrict__ tile_off,
    const unsigned* __restrict__ flags, int64_t n, const int4* __restrict__ st,
    double* __restrict__ Xo,
    int32_t* __restrict__ Io, int32_t* __restrict__ NIDo, double* __restrict__ Pf,
    int32_t* __restrict__ If, int32_t* __restrict__ err) {
  constexpr int W = kBT / 32;
  __shared__ int32_t cpre[kItems * W + 1];
  __shared__ __align__(8) unsigned long long bar;
  extern __shared__ __align__(16) unsigned char stage[];
  double* sx = reinterpret_cast<double*>(stage);
  int32_t* si = reinterpret_cast<int32_t*>(stage + (size_t)D * kTile * sizeof(double));
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * kTile;
  const int64_t nw = st->y;
  if (base >= nw) return;  // past this level's working set (the whole block)
  if (STAGED) {
    if (threadIdx.x == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar)) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      const int64_t cnt = min((int64_t)kTile, nw - base);
      const uint32_t bx = (uint32_t)(((cnt + 1) & ~1ll) * 8), bi = (uint32_t)(((cnt + 3) & ~3ll) * 4);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&bar)),
                   "r"(D * bx + bi)
                   : "memory");
#pragma unroll
      for (int j = 0; j < D; ++j)
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
            "[%3];" ::"r"(smem_u32(sx + j * kTile)),
            "l"(X + (int64_t)j * n + base), "r"(bx), "r"(smem_u32(&bar))
            : "memory");
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
          "[%3];" ::"r"(smem_u32(si)),
          "l"(I + base), "r"(bi), "r"(smem_u32(&bar))
          : "memory");
    }
  }
  unsigned msk[kItems];
  int32_t av[kItems];
  const bool one = tile_of_one_node(NID, base, nw);
  const int32_t one_id = __ldg(NID + base);
#pragma unroll
  for (int it = 0; it < kItems; ++it) {
    const int64_t p = base + (int64_t)it * kBT + threadIdx.x;
    av[it] = one ? one_id : p < nw ? NID[p] : -1;
    msk[it] = flags[(base >> 5) + it * W + w];  // the flag pass's ballot of these 32 positions
  }
  tile_chunk_prefix(msk, cpre);
  if (STAGED && !bar_wait0(smem_u32(&bar))) {
    atomicExch(err, 3);             // copies did not land: report, let them finish, leave
    bar_wait0(smem_u32(&bar));
    return;
  }
  const int32_t run = tile_off[blockIdx.x];
  const unsigned lt = (1u << lane) - 1u;
#pragma unroll
  for (int it = 0; it < kItems; ++it) {
    const int32_t a = av[it];
    if (a < 0) continue;
    const int64_t p = base + (int64_t)it * kBT + threadIdx.x;
    const int4 r0 = srec[2 * (int64_t)a], r1 = srec[2 * (int64_t)a + 1];
    const int32_t start = r0.x, nl = r0.z, count = r0.w;
    const int32_t q = (int32_t)(p - r0.y);  // position in the segment
    int f;
    int32_t rank;  // rank in the child
    if (r1.z == -2 || r1.w == -2) {  // the slide point alone on one side, the others keep their order
      const bool sp = p == r1.x;
      f = (r1.z == -2) == sp ? 1 : 0;
      rank = sp ? 0 : q - (p > r1.x ? 1 : 0);
    } else {
      f = (int)((msk[it] >> lane) & 1u);
      const int32_t ex = run + cpre[it * W + w] + __popc(msk[it] & lt);
      const int32_t rl = ex - r1.x;  // left points before p in the segment
      rank = f ? rl : q - rl;
    }
    const int32_t ccount = f ? nl : count - nl;
    if (rank < 0 || rank >= ccount) {  // never for a consistent scan
      atomicExch(err, 2);
      continue;
    }
    const int t = (int)(p - base);
    const int32_t id = STAGED ? si[t] : I[p];
    double xv[D];
#pragma unroll
    for (int j = 0; j < D; ++j) xv[j] = STAGED ? sx[j * kTile + t] : X[(int64_t)j * n + p];
    const int32_t wc = f ? r1.z : r1.w;  // child's working start, negative for a leaf
    if (wc < 0) {
      const int64_t dst = (int64_t)start + (f ? 0 : nl) + rank;
#pragma unroll
      for (int j = 0; j < D; ++j) Pf[(int64_t)j * n + dst] = xv[j];
      If[dst] = id;
    } else {
      const int64_t wd = (int64_t)wc + rank;
#pragma unroll
      for (int j = 0; j < D; ++j) Xo[(int64_t)j * n + wd] = xv[j];
      Io[wd] = id;
      NIDo[wd] = r1.y + (f ? 0 : 1);
    }
  }
}

// ------------------------------------------------------ subtrees in shared memory
// A node of at most finish_max(D) points leaves the level passes: its points go to
// its range of the leaf-ordered arrays, and one block builds the rest of its subtree
// in shared memory, with the level passes' rules (split_rule, the stable
// partition, the first point at the extreme for a slide).  The points stay where
// they were loaded, as ordered keys; a 16-bit permutation is partitioned, ping-pong,
// level by level, and the points of a new leaf are written to their final place.  Nodes of more than
// kFinBlock points are split by the whole block, the others by a warp each.  A
// level's children take their ids from one atomic add on the node count, so
// children follow their parents and a pair stays adjacent, but the numbering
// below finish_max depends on the order of the blocks.
// A level pass costs ~45 us of launches and, at 2^24 points, 104 bytes a point; this
// replaces the last ten or so.  Whole builds before / after (us): 1000 points 559 /
// 286, 20011 clustered 1376 / 658, 2^20 uniform 1460 / 990, 2^24 clustered 14214 /
// 12664 (2.6 ms of it here).  Bound by issue and by waiting at the levels' barriers
// (24 warps an SM, 47 % of issue slots): about 950 warp instructions a split node,
// most nodes holding fewer than 40 points.  Not faster: 1024 or 512 points a block,
// 128 or 512 threads, small subtrees queued for warps that need no barrier.
constexpr int kFinT = 256;
constexpr int kFinBlock = 512;
constexpr int64_t kFinGrowMax = (int64_t)4 << 30;  // bytes of the largest node arrays taken at once
__host__ __device__ constexpr int finish_max(int d) { return d <= 3 ? 2048 : 1024; }
__host__ __device__ constexpr int finish_open(int m, int leaf) { return m / (leaf + 1) + 1; }
__host__ __device__ constexpr size_t finish_smem(int d, int leaf) {
  const size_t m = finish_max(d);
  return m * (8 * d + 4 + 2 * 2) + 2 * (size_t)finish_open((int)m, leaf) * 8;
}

// nodes the level passes left: leaves of the list so far with more than `leaf` points
__global__ void k_finish_list(const NodeMeta* __restrict__ meta, int32_t n_nodes, int leaf,
                              int32_t* __restrict__ list, int32_t* __restrict__ n_list) {
  const int32_t a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= n_nodes) return;
  if (meta[a].left < 0 && meta[a].count > leaf) list[atomicAdd(n_list, 1)] = a;
}

// ctr: {node count, deepest level + 1, depth error, next list entry, length of the list,
// length of redo}.  A subtree whose nodes no longer fit (node_cap) puts its points back and
// goes to `redo`, for a launch with more room.  The node ids that it had taken stay its
// own: log holds, per level, the first (at the subtree's positions, the last of which says
// how many), and the next launch (`resume`) takes them again.
template <int D>
__global__ void __launch_bounds__(kFinT) k_finish(const int32_t* __restrict__ list,
                                                  const int32_t* __restrict__ n_list,
                                                  NodeMeta* meta, double* cell, double* box,
                                                  double* Pf, int32_t* If, int64_t n, int leaf,
                                                  int32_t node_cap, int32_t max_levels,
                                                  int32_t* ctr, int32_t* redo, int32_t* log,
                                                  bool resume) {
  constexpr int M = finish_max(D), W = kFinT / 32, NP = M / kFinT;
  static_assert(NP * W <= 64, "one warp scans the chunk counts");
  extern __shared__ __align__(16) unsigned char fsm[];
  unsigned long long* X = reinterpret_cast<unsigned long long*>(fsm);    // [D][M] keys
  int32_t* I = reinterpret_cast<int32_t*>(X + (size_t)D * M);            // [M]
  uint16_t* perm0 = reinterpret_cast<uint16_t*>(I + M);                  // [2][M]
  const int lcap = finish_open(M, leaf);
  int2* open = reinterpret_cast<int2*>(perm0 + 2 * M);                   // [2][lcap] {node, start | count << 16}
  __shared__ unsigned long long red[W][2 * D];
  __shared__ int32_t cpre[65];
  __shared__ int32_t s_job, s_full, s_base, s_next, s_ext;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int32_t jobs = *n_list;
  int deepest = 0;
  for (;;) {
    if (tid == 0) {
      s_job = atomicAdd(&ctr[3], 1);
      s_full = *(volatile int32_t*)&ctr[0] >= node_cap;
    }
    __syncthreads();
    const int32_t job = s_job;
    if (job >= jobs) break;
    const int32_t root = list[job];
    const int32_t g0 = meta[root].start, c0 = meta[root].count;
    int depth = meta[root].depth;
    const int known = resume ? log[g0 + c0 - 1] : 0;  // levels whose ids were taken before
    if (known == 0 && s_full) {
      if (tid == 0) {
        log[g0 + c0 - 1] = 0;
        redo[atomicAdd(&ctr[5], 1)] = root;
      }
      __syncthreads();  // s_job and s_full serve the next subtree
      continue;
    }
    for (int i = tid; i < c0; i += kFinT) {
#pragma unroll
      for (int j = 0; j < D; ++j) X[j * M + i] = dkey(Pf[(int64_t)j * n + g0 + i]);
      I[i] = If[g0 + i];
      perm0[i] = (uint16_t)i;
    }
    if (tid == 0) open[0] = make_int2(root, c0 << 16);
    int m = 1, cur = 0;
    bool ok = true;
    for (int level = 0; m > 0; ++level) {
      const uint16_t* pa = perm0 + (cur ? M : 0);
      uint16_t* pb = perm0 + (cur ? 0 : M);
      const int2* oa = open + (cur ? lcap : 0);
      int2* ob = open + (cur ? 0 : lcap);
      if (tid == 0) {
        s_base = level < known ? log[g0 + level] : atomicAdd(&ctr[0], 2 * m);
        log[g0 + level] = s_base;
        s_next = 0;
      }
      __syncthreads();  // also: the points, the open list and the permutation are in place
      const int32_t base = s_base;
      if (depth >= max_levels) {
        if (tid == 0) ctr[2] = 1;
        ok = false;
        break;  // the same for the whole block
      }
      if (base > node_cap - 2 * m) {
        for (int i = tid; i < c0; i += kFinT) {
#pragma unroll
          for (int j = 0; j < D; ++j) Pf[(int64_t)j * n + g0 + i] = dkey_inv(X[j * M + i]);
          If[g0 + i] = I[i];
        }
        if (tid == 0) {
          log[g0 + c0 - 1] = level + 1;
          redo[atomicAdd(&ctr[5], 1)] = root;
        }
        ok = false;
        break;
      }
      // the children of open node e (node a, local start s, count c), split as told,
      // with nl points on the left: records and the next open list
      auto children = [&](int e, int32_t a, int s, int c, int nl, int axis, double mid,
                          const double (&lo)[D], const double (&hi)[D], int ln) {
        const int32_t l = base + 2 * e;
        if (ln < 2 * D) {
          double v = lo[0];
#pragma unroll
          for (int j = 0; j < D; ++j) {
            if (ln == 2 * j) v = lo[j];
            if (ln == 2 * j + 1) v = hi[j];
          }
          box[(int64_t)a * 2 * D + ln] = v;
          double cl = cell[(int64_t)a * 2 * D + ln];
          const bool ax = (ln >> 1) == axis;
          cell[(int64_t)l * 2 * D + ln] = ax && (ln & 1) ? mid : cl;         // :419-422
          cell[(int64_t)(l + 1) * 2 * D + ln] = ax && !(ln & 1) ? mid : cl;
        }
        if (ln < 2) {
          NodeMeta cm;
          cm.split = 0.0;
          cm.left = -1;
          cm.axis = -1;
          cm.start = g0 + s + (ln ? nl : 0);
          cm.count = ln ? c - nl : nl;
          cm.depth = depth + 1;
          cm.parent = a;
          meta[l + ln] = cm;
          if (cm.count > leaf) {
            const int o = atomicAdd(&s_next, 1);
            ob[o] = make_int2(l + ln, (s + (ln ? nl : 0)) | (cm.count << 16));
          }
        }
        if (ln == 2) {
          meta[a].split = mid;
          meta[a].left = l;
          meta[a].axis = axis;
        }
      };
      // a point's place: in the child's segment of the other permutation, or, when
      // the child is a leaf, in the leaf-ordered arrays
      auto place = [&](uint16_t ix, int pos, int ccount) {
        if (ccount > leaf) {
          pb[pos] = ix;
        } else {
#pragma unroll
          for (int j = 0; j < D; ++j) Pf[(int64_t)j * n + g0 + pos] = dkey_inv(X[j * M + ix]);
          If[g0 + pos] = I[ix];
        }
      };
      // ---- large nodes, the whole block each
      for (int e = 0; e < m; ++e) {
        const int32_t a = oa[e].x;
        const int s = oa[e].y & 0xffff, c = (unsigned)oa[e].y >> 16;
        if (c <= kFinBlock) continue;
        unsigned long long kmn[D], kmx[D];
#pragma unroll
        for (int j = 0; j < D; ++j) kmn[j] = kmx[j] = ~0ull;
        for (int i = tid; i < c; i += kFinT) {
          const int ix = pa[s + i];
#pragma unroll
          for (int j = 0; j < D; ++j) {
            const unsigned long long k = X[j * M + ix];
            kmn[j] = k < kmn[j] ? k : kmn[j];
            kmx[j] = ~k < kmx[j] ? ~k : kmx[j];
          }
        }
#pragma unroll
        for (int j = 0; j < D; ++j) {
          kmn[j] = warp_min_key(kmn[j]);
          kmx[j] = warp_min_key(kmx[j]);
          if (lane == 0) {
            red[w][2 * j] = kmn[j];
            red[w][2 * j + 1] = kmx[j];
          }
        }
        if (tid == 0) s_ext = 0x7fffffff;
        __syncthreads();
        double lo[D], hi[D], clo[D], chi[D];
#pragma unroll
        for (int j = 0; j < D; ++j) {
          unsigned long long a0 = red[0][2 * j], a1 = red[0][2 * j + 1];
#pragma unroll
          for (int x = 1; x < W; ++x) {
            a0 = red[x][2 * j] < a0 ? red[x][2 * j] : a0;
            a1 = red[x][2 * j + 1] < a1 ? red[x][2 * j + 1] : a1;
          }
          lo[j] = dkey_inv(a0);
          hi[j] = dkey_inv(~a1);
          clo[j] = cell[(int64_t)a * 2 * D + 2 * j];
          chi[j] = cell[(int64_t)a * 2 * D + 2 * j + 1];
        }
        int axis, md;
        double mid;
        split_rule<D>(lo, hi, clo, chi, axis, mid, md);
        const unsigned long long* xa = X + axis * M;
        // the FP64 comparisons as key comparisons (the two zeros are equal)
        const unsigned long long km = dkey(mid == 0.0 ? -0.0 : mid), wide = mid == 0.0 ? 1 : 0;
        unsigned msk[NP];
#pragma unroll
        for (int it = 0; it < NP; ++it) {
          const int i = it * kFinT + tid;
          bool f = false;
          if (i < c) {
            const unsigned long long k = xa[pa[s + i]];
            f = md == 0 ? k < km : k - km <= wide;
            if (md != 0 && f) atomicMin(&s_ext, i);
          }
          msk[it] = __ballot_sync(0xffffffffu, f);
          if (lane == 0) cpre[it * W + w] = __popc(msk[it]);
        }
        __syncthreads();
        if (w == 0) {
          const int x0 = 2 * lane < NP * W ? cpre[2 * lane] : 0;
          const int x1 = 2 * lane + 1 < NP * W ? cpre[2 * lane + 1] : 0;
          const int inc = warp_inclusive_scan(x0 + x1);
          cpre[2 * lane] = inc - x0 - x1;
          cpre[2 * lane + 1] = inc - x1;
          if (lane == 31) cpre[64] = inc;
        }
        __syncthreads();
        const int ext = s_ext;
        const int nl = md == 0 ? cpre[64] : md == 1 ? 1 : c - 1;
#pragma unroll
        for (int it = 0; it < NP; ++it) {
          const int i = it * kFinT + tid;
          if (i >= c) continue;
          bool f;
          int r;  // rank in the child
          if (md == 0) {
            f = (msk[it] >> lane) & 1u;
            const int lp = cpre[it * W + w] + __popc(msk[it] & lt);
            r = f ? lp : i - lp;
          } else {  // the slide point alone on one side, the others keep their order
            f = (i == ext) == (md == 1);
            r = i == ext ? 0 : i - (i > ext ? 1 : 0);
          }
          place(pa[s + i], s + (f ? r : nl + r), f ? nl : c - nl);
        }
        children(e, a, s, c, nl, axis, mid, lo, hi, tid);
        __syncthreads();  // red, cpre and s_ext serve the next large node
      }
      // ---- the others, a warp each
      for (int e = w; e < m; e += W) {
        const int32_t a = oa[e].x;
        const int s = oa[e].y & 0xffff, c = (unsigned)oa[e].y >> 16;
        if (c > kFinBlock) continue;
        double lo[D], hi[D], clo[D], chi[D];
        {
          unsigned long long kmn[D], kmx[D];
#pragma unroll
          for (int j = 0; j < D; ++j) kmn[j] = kmx[j] = ~0ull;
          for (int i = lane; i < c; i += 32) {
            const int ix = pa[s + i];
#pragma unroll
            for (int j = 0; j < D; ++j) {
              const unsigned long long k = X[j * M + ix];
              kmn[j] = k < kmn[j] ? k : kmn[j];
              kmx[j] = ~k < kmx[j] ? ~k : kmx[j];
            }
          }
#pragma unroll
          for (int j = 0; j < D; ++j) {
            lo[j] = dkey_inv(warp_min_key(kmn[j]));
            hi[j] = dkey_inv(~warp_min_key(kmx[j]));
            clo[j] = cell[(int64_t)a * 2 * D + 2 * j];
            chi[j] = cell[(int64_t)a * 2 * D + 2 * j + 1];
          }
        }
        int axis, md;
        double mid;
        split_rule<D>(lo, hi, clo, chi, axis, mid, md);
        const unsigned long long* xa = X + axis * M;
        // the FP64 comparisons as key comparisons (the two zeros are equal)
        const unsigned long long km = dkey(mid == 0.0 ? -0.0 : mid), wide = mid == 0.0 ? 1 : 0;
        int nl = 0, ext = -1;
        for (int b = 0; b < c; b += 32) {
          bool f = false;
          if (b + lane < c) {
            const unsigned long long k = xa[pa[s + b + lane]];
            f = md == 0 ? k < km : k - km <= wide;
          }
          const unsigned fm = __ballot_sync(0xffffffffu, f);
          if (md == 0) {
            nl += __popc(fm);
          } else if (fm) {
            ext = b + __ffs(fm) - 1;
            break;
          }
        }
        if (md != 0) nl = md == 1 ? 1 : c - 1;
        int lp = 0;  // left points before this chunk
        for (int b = 0; b < c; b += 32) {
          const int i = b + lane;
          const uint16_t ix = i < c ? pa[s + i] : (uint16_t)0;
          bool f = false;
          int r = 0;
          if (md == 0) {
            f = i < c && xa[ix] < km;
            const unsigned fm = __ballot_sync(0xffffffffu, f);
            r = f ? lp + __popc(fm & lt) : i - lp - __popc(fm & lt);
            lp += __popc(fm);
          } else {
            f = (i == ext) == (md == 1);
            r = i == ext ? 0 : i - (i > ext ? 1 : 0);
          }
          if (i < c) place(ix, s + (f ? r : nl + r), f ? nl : c - nl);
        }
        children(e, a, s, c, nl, axis, mid, lo, hi, lane);
      }
      ++depth;
      __syncthreads();
      m = s_next;
      cur ^= 1;
      __syncthreads();  // s_next is read before the next level clears it
    }
    if (ok) deepest = max(deepest, depth);
    __syncthreads();  // s_job and the shared arrays serve the next subtree
  }
  if (tid == 0) atomicMax(&ctr[1], deepest);
}

// bounding boxes of the leaves from the final leaf-ordered points
template <int D>
__global__ void k_leaf_box(const NodeMeta* __restrict__ meta, int32_t n_nodes, int leaf,
                           const double* __restrict__ Pf, int64_t n, double* __restrict__ box) {
  int32_t a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= n_nodes) return;
  NodeMeta m = meta[a];
  if (m.count > leaf) return;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    double lo = Pf[(int64_t)j * n + m.start], hi = lo;
    for (int i = 1; i < m.count; ++i) {
      double v = Pf[(int64_t)j * n + m.start + i];
      lo = v < lo ? v : lo;
      hi = v > hi ? v : hi;
    }
    box[(int64_t)a * 2 * D + 2 * j] = lo;
    box[(int64_t)a * 2 * D + 2 * j + 1] = hi;
  }
}

// Per point: the FP64 coordinates as a packed record of (d + 3) / 4 double4s and the
// absolute coordinates rounded to FP32 in float4s (both zero padded).
template <int D>
__global__ void k_point_records(const double* __restrict__ Pf, int64_t n, double4* __restrict__ P64,
                                float4* __restrict__ P32) {
  constexpr int NV = (D + 3) / 4;
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  double v[4 * NV];
  float f[4 * NV];
#pragma unroll
  for (int j = 0; j < 4 * NV; ++j) {
    v[j] = j < D ? Pf[(int64_t)(j < D ? j : 0) * n + p] : 0.0;
    f[j] = j < D ? __double2float_rn(v[j]) : 0.0f;
  }
#pragma unroll
  for (int h = 0; h < NV; ++h) {
    P64[p * NV + h] = make_double4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
    P32[p * NV + h] = make_float4(f[4 * h], f[4 * h + 1], f[4 * h + 2], f[4 * h + 3]);
  }
}

// The nodes' boxes and cells at their final place, with the FP32 forms: boxes rounded
// outwards (lo down, hi up: every FP32 gap computed from them is a lower bound of the
// FP64 gap up to the screen's rounding slack), cells inwards.  One value a thread:
// with a node a thread its 48-byte strides took 400 us for all node records of 2^24
// clustered points, against 232 us for this and the next kernel.
__global__ void k_node_boxes(const double* __restrict__ bbox, const double* __restrict__ bcell,
                             int64_t count, double* __restrict__ box, double* __restrict__ cell,
                             float* __restrict__ box32, float* __restrict__ cell32) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const double x = bbox[i], c = bcell[i];
  const bool hi = i & 1;
  box[i] = x;
  cell[i] = c;
  box32[i] = hi ? __double2float_ru(x) : __double2float_rd(x);
  cell32[i] = hi ? __double2float_rd(c) : __double2float_ru(c);
}

// Per node: the record at its final place, a leaf's FP64 centre, and an internal node's
// child-pair record (both children's outward FP32 boxes, ids, leaf flags and position
// ranges), so one load serves a whole expansion.
template <int D>
__global__ void k_node_records(const NodeMeta* __restrict__ bmeta, int32_t n_nodes,
                               const double* __restrict__ bbox, NodeMeta* __restrict__ meta,
                               float4* __restrict__ pair, double* __restrict__ centre) {
  constexpr int NV = (D + 3) / 4;
  constexpr int PF = pair_f4(D);
  int32_t a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= n_nodes) return;
  const NodeMeta m = bmeta[a];
  meta[a] = m;
  if (m.left < 0) {
    const double2* bx = reinterpret_cast<const double2*>(bbox + (int64_t)a * 2 * D);
#pragma unroll
    for (int j = 0; j < D; ++j) centre[(int64_t)a * D + j] = leaf_centre(bx[j].x, bx[j].y);
    return;
  }
  float4* rec = pair + (int64_t)a * PF;
  for (int side = 0; side < 2; ++side) {
    const double2* cx = reinterpret_cast<const double2*>(bbox + (int64_t)(m.left + side) * 2 * D);
    float lo[4 * NV], hi[4 * NV];
#pragma unroll
    for (int j = 0; j < 4 * NV; ++j) {
      const double2 x = j < D ? cx[j < D ? j : 0] : make_double2(0.0, 0.0);
      lo[j] = j < D ? __double2float_rd(x.x) : 0.0f;
      hi[j] = j < D ? __double2float_ru(x.y) : 0.0f;
    }
#pragma unroll
    for (int h = 0; h < NV; ++h) {
      rec[side * 2 * NV + h] = make_float4(lo[4 * h], lo[4 * h + 1], lo[4 * h + 2], lo[4 * h + 3]);
      rec[side * 2 * NV + NV + h] =
          make_float4(hi[4 * h], hi[4 * h + 1], hi[4 * h + 2], hi[4 * h + 3]);
    }
  }
  const NodeMeta ml = bmeta[m.left], mr = bmeta[m.left + 1];
  int4 info = make_int4(m.left, m.left + 1, ml.left < 0 ? 1 : 0, mr.left < 0 ? 1 : 0);
  rec[4 * NV] = *reinterpret_cast<float4*>(&info);
  int4 range = make_int4(ml.start, ml.count, mr.start, mr.count);
  rec[4 * NV + 1] = *reinterpret_cast<float4*>(&range);
}

// roots: node t = root of tree t (positions off[t] .. off[t+1]-1)
template <int D>
__global__ void k_root_init(NodeMeta* meta, double* cell, unsigned long long* keys,
                            const int64_t* __restrict__ off, int32_t n_trees, const double* L,
                            int periodic) {
  int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_trees) return;
  NodeMeta m;
  m.split = 0.0;
  m.left = -1;
  m.axis = -1;
  m.start = (int32_t)off[t];
  m.count = (int32_t)(off[t + 1] - off[t]);
  m.depth = 0;
  m.parent = -1;
  meta[t] = m;
  for (int j = 0; j < D; ++j) {
    cell[(int64_t)t * 2 * D + 2 * j] = periodic ? -L[j] / 2. : 0.0;  // :218-224 (every axis)
    cell[(int64_t)t * 2 * D + 2 * j + 1] = periodic ? L[j] / 2. : 0.0;
    keys[(int64_t)t * 2 * D + 2 * j] = ~0ull;
    keys[(int64_t)t * 2 * D + 2 * j + 1] = 0ull;
  }
}

// non-periodic root cells = the data bounding box of each tree (:226-229)
template <int D>
__global__ void k_root_cells(double* cell, const unsigned long long* __restrict__ keys,
                             int32_t n_trees) {
  int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_trees) return;
  for (int j = 0; j < 2 * D; ++j) cell[(int64_t)t * 2 * D + j] = dkey_inv(keys[(int64_t)t * 2 * D + j]);
}

// ------------------------------------------------------------------ host side

template <typename T>
cudaError_t grow(const BuildBufs& B, T** p, int64_t old_n, int64_t new_n, cudaStream_t s) {
  T* q = nullptr;
  cudaError_t e = dev_alloc((void**)&q, sizeof(T) * new_n, s);
  if (e != cudaSuccess) return e;
  if (*p && old_n > 0) {
    e = cudaMemcpyAsync(q, *p, sizeof(T) * old_n, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) {
      dev_free(q, s);
      return e;
    }
    if (B.outside(*p)) dev_free(*p, s);
  }
  *p = q;
  return cudaSuccess;
}

ckd_status ensure_tree_cap(BuildBufs& B, int64_t need, cudaStream_t s) {
  if (need <= B.tcap) return CKD_OK;
  int64_t nc = std::max<int64_t>(need, B.tcap * 2);
  int d2 = 2 * B.d;
  CKD_CUDA(grow(B, &B.meta, B.tcap, nc, s));
  CKD_CUDA(grow(B, &B.cell, B.tcap * d2, nc * d2, s));
  CKD_CUDA(grow(B, &B.box, B.tcap * d2, nc * d2, s));
  B.tcap = nc;
  return CKD_OK;
}

ckd_status ensure_node_cap(BuildBufs& B, int64_t need, cudaStream_t s) {
  CKD_TRY(ensure_tree_cap(B, need, s));
  if (need <= B.cap) return CKD_OK;
  int64_t nc = std::max<int64_t>(need, B.cap * 2);
  int d2 = 2 * B.d;
  CKD_CUDA(grow(B, &B.keys, B.cap * d2, nc * d2, s));
  CKD_CUDA(grow(B, &B.ext, B.cap, nc, s));
  CKD_CUDA(grow(B, &B.mode, B.cap, nc, s));
  CKD_CUDA(grow(B, &B.pstart, B.cap, nc, s));
  CKD_CUDA(grow(B, &B.pend, B.cap, nc, s));
  CKD_CUDA(grow(B, &B.nleft, B.cap, nc, s));
  CKD_CUDA(grow(B, &B.pbase, B.cap, nc, s));
  CKD_CUDA(grow(B, &B.wst, B.cap, nc, s));
  CKD_CUDA(grow(B, &B.frec, B.cap, nc, s));
  CKD_CUDA(grow(B, &B.srec, B.cap * 2, nc * 2, s));
  B.cap = nc;
  return CKD_OK;
}

void free_bufs(BuildBufs& B, cudaStream_t s) {
  void* ps[] = {B.meta, B.cell,  B.box, B.keys,  B.ext,  B.mode, B.pstart,
                B.pend, B.nleft, B.pbase, B.wst, B.frec, B.srec};
  for (void* p : ps)
    if (B.outside(p)) dev_free(p, s);
  if (B.arena) dev_free(B.arena, s);
  B = BuildBufs();
}

template <int D>
ckd_status build_impl(ckd_tree* t, const void* pts_dev, int dtype, cudaStream_t s) {
  const int64_t n = t->n;
  // the level passes end at nodes that a block finishes in shared memory
  const int tree_leaf = t->leaf;
  const bool finish = tree_leaf < finish_max(D);
  const int leaf = finish ? finish_max(D) : tree_leaf;
  BuildBufs B;
  B.d = D;
  B.n = n;
  struct Guard {
    BuildBufs* b;
    cudaStream_t s;
    ~Guard() { free_bufs(*b, s); }
  } guard{&B, s};

  const int64_t ntiles = cdiv(n, kTile);
  const int32_t T = (int32_t)t->n_trees;
  const int64_t max_open = n / (leaf + 1) + 2 + T;
  B.tcap = (int64_t)T + std::min<int64_t>(2 * n, 4 * (n / tree_leaf) + 64);  // grown on need
  B.cap = (int64_t)T + 4 * (n / leaf) + 64;
  B.tcap = std::max(B.tcap, B.cap);
  int64_t* off_dev = nullptr;
  double* Ldev = nullptr;
  int32_t *flist = nullptr, *fctr = nullptr;  // nodes to finish (two lists); k_finish's counters
  for (int pass = 0; pass < 2; ++pass) {
    Carve c(B.arena);
    for (int b = 0; b < 2; ++b) {
      c.take(&B.X[b], (size_t)D * n);
      c.take(&B.I[b], n + 4);  // + the bulk copy's rounding
      c.take(&B.NID[b], n);
      c.take(&B.act[b], max_open);
    }
    c.take(&B.nxt_cnt, max_open);
    c.take(&B.nxt_off, max_open + 1);
    c.take(&B.tile_sum, ntiles);
    c.take(&B.tile_off, ntiles + 1);
    c.take(&B.flags, ntiles * (kTile / 32));
    c.take(&B.scal, 4);
    c.take(&B.lst, 2);
    c.take(&B.meta, B.tcap);
    c.take(&B.cell, B.tcap * 2 * D);
    c.take(&B.box, B.tcap * 2 * D);
    c.take(&B.keys, B.cap * 2 * D);
    c.take(&B.ext, B.cap);
    c.take(&B.mode, B.cap);
    c.take(&B.pstart, B.cap);
    c.take(&B.pend, B.cap);
    c.take(&B.nleft, B.cap);
    c.take(&B.pbase, B.cap);
    c.take(&B.wst, B.cap);
    c.take(&B.frec, B.cap);
    c.take(&B.srec, B.cap * 2);
    c.take(&off_dev, T + 1);
    c.take(&Ldev, CKD_MAX_D);
    c.take(&fctr, 8);
    if (pass == 0) {
      B.arena_bytes = c.off;
      CKD_CUDA(dev_alloc((void**)&B.arena, c.off, s));
    }
  }
  CKD_CUDA(cudaMemsetAsync(B.scal, 0, sizeof(int32_t) * 4, s));

  // the tree's arrays per point
  constexpr int NV = (D + 3) / 4;
  for (int pass = 0; pass < 2; ++pass) {
    Carve c(t->block[0]);
    c.take(&t->pts, (size_t)D * n);
    c.take(&t->ids, n);
    c.take(&t->pts32, (size_t)NV * n);
    c.take(&t->pts64, (size_t)NV * n);
    if (pass == 0) CKD_CUDA(dev_alloc(&t->block[0], c.off, s));
  }

  // trees of a forest: positions off[t] .. off[t+1]-1, root node t
  const std::vector<int64_t>& off = t->tree_off;
  Scratch sc(s);
  CKD_CUDA(cudaMemcpyAsync(off_dev, off.data(), sizeof(int64_t) * (T + 1), cudaMemcpyHostToDevice, s));
  {
    unsigned g = (unsigned)cdiv(n, 256);
    const int64_t* offp = T > 1 ? off_dev : nullptr;
    if (dtype == CKD_F32)
      k_init_points<float><<<g, 256, 0, s>>>((const float*)pts_dev, n, D, B.X[0], B.I[0],
                                             B.NID[0], B.NID[1], offp, T);
    else
      k_init_points<double><<<g, 256, 0, s>>>((const double*)pts_dev, n, D, B.X[0], B.I[0],
                                              B.NID[0], B.NID[1], offp, T);
    CKD_LAUNCH_CHECK();
  }
  CKD_CUDA(cudaMemcpyAsync(Ldev, t->L, sizeof(double) * CKD_MAX_D, cudaMemcpyHostToDevice, s));
  k_root_init<D><<<(unsigned)cdiv(T, 128), 128, 0, s>>>(B.meta, B.cell, B.keys, off_dev, T, Ldev,
                                                        t->periodic);
  CKD_LAUNCH_CHECK();

  // Root bounding boxes: validation (finite, inside the periodic box) and the
  // non-periodic root cells, from the segmented reduction over every point
  // (position p belongs to root NID[p]).
  k_seg_box<D><<<(unsigned)ntiles, kBT, 0, s>>>(B.X[0], B.NID[0], n, n, B.keys);
  CKD_LAUNCH_CHECK();
  std::vector<unsigned long long> rk((size_t)T * 2 * D);
  CKD_CUDA(cudaMemcpyAsync(rk.data(), B.keys, sizeof(unsigned long long) * 2 * D * T,
                           cudaMemcpyDeviceToHost, s));
  CKD_CUDA(cudaStreamSynchronize(s));
  double rlo[CKD_MAX_D], rhi[CKD_MAX_D];
  for (int j = 0; j < D; ++j) {
    rlo[j] = INFINITY;
    rhi[j] = -INFINITY;
  }
  for (int32_t tr = 0; tr < T; ++tr) {
    for (int j = 0; j < D; ++j) {
      auto inv = [](unsigned long long k) {
        unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
        double x;
        std::memcpy(&x, &b, 8);
        return x;
      };
      double lo = inv(rk[(size_t)tr * 2 * D + 2 * j]), hi = inv(rk[(size_t)tr * 2 * D + 2 * j + 1]);
      if (!std::isfinite(lo) || !std::isfinite(hi))
        return fail(CKD_ERR_BAD_ARG, "points contain NaN or infinite coordinates");
      if (t->periodic && (lo < -t->L[j] / 2 || hi > t->L[j] / 2))
        return fail(CKD_ERR_OUT_OF_BOX, "Points outside (-L/2, L/2) range");
      rlo[j] = std::min(rlo[j], lo);
      rhi[j] = std::max(rhi[j], hi);
    }
  }
  if (!t->periodic) {
    k_root_cells<D><<<(unsigned)cdiv(T, 128), 128, 0, s>>>(B.cell, B.keys, T);
    CKD_LAUNCH_CHECK();
  }
  // open roots and the first working set
  std::vector<int32_t> roots;
  std::vector<int32_t> wst0((size_t)T, -1);
  int64_t nw = 0;
  for (int32_t tr = 0; tr < T; ++tr)
    if (off[tr + 1] - off[tr] > leaf) {
      roots.push_back(tr);
      wst0[tr] = (int32_t)nw;
      nw += off[tr + 1] - off[tr];
    }
  int cur = 0;
  if (nw < n) {
    // points of trees that are a single leaf never move: start from the input order
    CKD_CUDA(cudaMemcpyAsync(t->pts, B.X[0], sizeof(double) * D * n, cudaMemcpyDeviceToDevice, s));
    CKD_CUDA(cudaMemcpyAsync(t->ids, B.I[0], sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, s));
  }
  CKD_CUDA(cudaMemcpyAsync(B.wst, wst0.data(), sizeof(int32_t) * T, cudaMemcpyHostToDevice, s));
  if (nw < n && nw > 0) {
    k_compact_roots<D><<<(unsigned)cdiv(n, 256), 256, 0, s>>>(B.X[0], B.I[0], B.NID[0], B.wst,
                                                             off_dev, n, B.X[1], B.I[1], B.NID[1]);
    CKD_LAUNCH_CHECK();
    cur = 1;
  }
  if (!roots.empty())
    CKD_CUDA(cudaMemcpyAsync(B.act[0], roots.data(), sizeof(int32_t) * roots.size(),
                             cudaMemcpyHostToDevice, s));

  // the staged scatter needs 16-byte aligned rows (even stride) and fits D <= 4
  // (<= 72 KB of shared memory per block)
  const bool staged = D <= 4 && (n & 1) == 0;
  if (staged)
    CKD_CUDA(cudaFuncSetAttribute(k_scatter<D, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)scatter_smem(D)));
  // pinned word for the readback of the level state
  static thread_local int4* level_st = nullptr;
  if (!level_st) CKD_CUDA(cudaMallocHost((void**)&level_st, sizeof(int4)));
  // Levels run ahead of the host: a chunk of up to kRunAhead levels is launched
  // with grids sized by bounds known at the last readback (the working set never
  // grows; a level has at most twice the previous level's open nodes and at most
  // nw / (leaf + 1) of them), every kernel reads the exact counts from the
  // device state and idles past them, and the host reads the state once per
  // chunk.  Levels after the last open node are no-ops.
  constexpr int kRunAhead = 6;
  int32_t n_nodes = T;
  int64_t m = (int64_t)roots.size();
  *level_st = make_int4((int32_t)m, (int32_t)nw, n_nodes, 0);
  CKD_CUDA(cudaMemcpyAsync(B.lst, level_st, sizeof(int4), cudaMemcpyHostToDevice, s));
  int depth_levels = 0;
  int par = 0;    // state slot of the next level
  int alist = 0;  // open list buffer of the next level
  int level = 0;  // levels launched
  while (m > 0) {
    if (level >= kMaxLevels)
      return fail(CKD_ERR_DEPTH, "tree depth exceeds the build's level cap (8192 levels)");
    int64_t mb[kRunAhead];
    mb[0] = m;
    int64_t grow = 2 * m;
    int S = 1;
    for (int c = 1; c < kRunAhead && level + c < kMaxLevels; ++c) {
      mb[c] = std::min<int64_t>(2 * mb[c - 1], nw / (leaf + 1));
      if (n_nodes + grow + 2 * mb[c] > B.cap) break;
      grow += 2 * mb[c];
      S = c + 1;
    }
    CKD_TRY(ensure_node_cap(B, (int64_t)n_nodes + grow, s));
    const unsigned ntw = (unsigned)cdiv(nw, kTile);
    for (int c = 0; c < S; ++c, ++level) {
      const int4* st = B.lst + par;
      int4* st_next = B.lst + (1 - par);
      const int32_t* act = B.act[alist];
      const int mbi = (int)std::max<int64_t>(1, mb[c]);
      const unsigned gm = (unsigned)cdiv(mbi, 128);
      if (level > 0) {  // the roots' boxes come from the validation pass
        k_seg_box<D><<<ntw, kBT, 0, s>>>(B.X[cur], B.NID[cur], n, nw, B.keys, st);
        CKD_LAUNCH_CHECK();
      }
      k_decide<D><<<gm, 128, 0, s>>>(act, st, B.meta, B.cell, B.box, B.keys, B.mode, B.ext, B.wst,
                                     B.frec);
      CKD_LAUNCH_CHECK();
      k_flags<<<ntw, kBT, 0, s>>>(B.X[cur], B.NID[cur], B.frec, B.ext, n, st, B.tile_sum,
                                  B.pstart, B.pend, B.flags);
      CKD_LAUNCH_CHECK();
      if (mbi <= kNodesMax && ntw <= kNodesTiles) {
        k_level_nodes<D><<<1, kNodesT, 0, s>>>(act, st, st_next, (int)ntw, B.meta, B.cell,
                                               B.pstart, B.pend, B.tile_sum, B.tile_off, B.wst,
                                               B.mode, B.ext, B.keys, leaf, B.act[1 - alist],
                                               B.srec, B.scal + 1);
        CKD_LAUNCH_CHECK();
      } else {
        CKD_TRY(scan_i32(B.tile_sum, B.tile_off, ntw, s));
        k_children<D><<<gm, 128, 0, s>>>(act, st, mbi, B.meta, B.cell, B.pstart, B.pend,
                                         B.tile_off, B.wst, B.mode, B.ext, B.nleft, B.pbase,
                                         B.keys, leaf, B.nxt_cnt, B.scal + 1);
        CKD_LAUNCH_CHECK();
        CKD_TRY(scan_i64(B.nxt_cnt, B.nxt_off, mbi, s));
        k_next_list<<<gm, 128, 0, s>>>(act, st, st_next, mbi, B.meta, B.nxt_off, leaf, B.mode,
                                       B.ext, B.nleft, B.pbase, B.act[1 - alist], B.wst, B.srec);
        CKD_LAUNCH_CHECK();
      }
      if (staged)
        k_scatter<D, true><<<ntw, kBT, scatter_smem(D), s>>>(
            B.X[cur], B.I[cur], B.NID[cur], B.srec, B.tile_off, B.flags, n, st, B.X[1 - cur],
            B.I[1 - cur], B.NID[1 - cur], t->pts, t->ids, B.scal + 1);
      else
        k_scatter<D, false><<<ntw, kBT, 0, s>>>(B.X[cur], B.I[cur], B.NID[cur], B.srec,
                                                B.tile_off, B.flags, n, st, B.X[1 - cur],
                                                B.I[1 - cur], B.NID[1 - cur], t->pts, t->ids,
                                                B.scal + 1);
      CKD_LAUNCH_CHECK();
      cur = 1 - cur;
      alist = 1 - alist;
      par = 1 - par;
    }
    CKD_CUDA(cudaMemcpyAsync(level_st, B.lst + par, sizeof(int4), cudaMemcpyDeviceToHost, s));
    CKD_CUDA(cudaStreamSynchronize(s));
    m = level_st->x;
    nw = level_st->y;
    n_nodes = level_st->z;
    depth_levels = level_st->w;
  }
  int32_t err = 0;
  CKD_CUDA(cudaMemcpyAsync(&err, B.scal + 1, sizeof(int32_t), cudaMemcpyDeviceToHost, s));

  if (finish) {
    int32_t* const ctr = fctr;
    CKD_CUDA(sc.alloc(&flist, sizeof(int32_t) * 2 * n_nodes));
    int32_t *list = flist, *redo = flist + n_nodes;
    int32_t* const log = B.I[0];  // free after the levels
    int32_t h[6] = {n_nodes, depth_levels, 0, 0, 0, 0};
    CKD_CUDA(cudaMemcpyAsync(ctr, h, sizeof(h), cudaMemcpyHostToDevice, s));
    k_finish_list<<<(unsigned)cdiv(n_nodes, 256), 256, 0, s>>>(B.meta, n_nodes, tree_leaf, list,
                                                               ctr + 4);
    CKD_LAUNCH_CHECK();
    int dev = 0, sms = 148, per_sm = 1;
    CKD_CUDA(cudaGetDevice(&dev));
    CKD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const size_t sm = finish_smem(D, tree_leaf);
    CKD_CUDA(cudaFuncSetAttribute(k_finish<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sm));
    CKD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_finish<D>, kFinT, sm));
    int64_t jobs = n_nodes;
    for (bool resume = false;; resume = true) {
      const int64_t g = std::min<int64_t>(jobs, (int64_t)sms * std::max(1, per_sm));
      k_finish<D><<<(unsigned)g, kFinT, sm, s>>>(
          list, ctr + 4, B.meta, B.cell, B.box, t->pts, t->ids, n, tree_leaf,
          (int32_t)std::min<int64_t>(B.tcap, INT32_MAX), kMaxLevels, ctr, redo, log, resume);
      CKD_LAUNCH_CHECK();
      CKD_CUDA(cudaMemcpyAsync(h, ctr, sizeof(h), cudaMemcpyDeviceToHost, s));
      CKD_CUDA(cudaStreamSynchronize(s));
      if (h[2])
        return fail(CKD_ERR_DEPTH, "tree depth exceeds the build's level cap (8192 levels)");
      if (h[5] == 0) break;
      // More nodes than planned (many equal points, steep clusters): the arrays grow and
      // only the subtrees that found no room are finished again.  At once to the most
      // nodes that a tree can have while these arrays stay small: every launch that runs out
      // of room again costs its deepest subtree's levels (2^22 points of many copies, 27
      // times the planned nodes: 22.8 ms when the tree was built twice, 36.1 when the
      // arrays doubled five times).
      const int64_t most = T + 2 * n;
      ckd_status st = CKD_ERR_OOM;
      if (most * (int64_t)(sizeof(NodeMeta) + 4 * D * sizeof(double)) <= kFinGrowMax)
        st = ensure_tree_cap(B, most, s);
      if (st == CKD_ERR_OOM) {
        cudaGetLastError();
        st = ensure_tree_cap(B, std::max<int64_t>(h[0], B.tcap + 1), s);
      }
      CKD_TRY(st);
      jobs = h[5];
      h[3] = 0;
      h[4] = h[5];
      h[5] = 0;
      CKD_CUDA(cudaMemcpyAsync(ctr, h, sizeof(h), cudaMemcpyHostToDevice, s));
      std::swap(list, redo);
    }
    n_nodes = h[0];
    depth_levels = std::max(depth_levels, (int)h[1]);
  }
  k_leaf_box<D><<<(unsigned)cdiv(n_nodes, 128), 128, 0, s>>>(B.meta, n_nodes, tree_leaf, t->pts, n,
                                                             B.box);
  CKD_LAUNCH_CHECK();
  t->n_nodes = n_nodes;
  t->depth = depth_levels;
  for (int pass = 0; pass < 2; ++pass) {  // the tree's arrays per node
    Carve c(t->block[1]);
    c.take(&t->meta, n_nodes);
    c.take(&t->box, (size_t)2 * D * n_nodes);
    c.take(&t->cell, (size_t)2 * D * n_nodes);
    c.take(&t->box32, (size_t)2 * D * n_nodes);
    c.take(&t->pair, (size_t)pair_f4(D) * n_nodes);
    c.take(&t->cell32, (size_t)2 * D * n_nodes);
    c.take(&t->centre, (size_t)D * n_nodes);
    if (pass == 0) CKD_CUDA(dev_alloc(&t->block[1], c.off, s));
  }
  // FP32 screening copies.  The node-gap slack per axis is 2^-21 * (|q| + B) with
  // B bounding every stored coordinate (and the box side when periodic); the
  // screen is disabled for coordinates near the FP32 range.
  t->screen_ok = true;
  for (int j = 0; j < D; ++j) {
    double b = std::max(std::fabs(rlo[j]), std::fabs(rhi[j])) + (t->periodic ? t->L[j] : 0.0);
    if (!(b < 1e18)) t->screen_ok = false;
    t->slack[j] = (float)(b * (1.0 + 1e-6));
    t->extent[j] = t->periodic ? t->L[j] : rhi[j] - rlo[j];
  }
  k_point_records<D><<<(unsigned)cdiv(n, 256), 256, 0, s>>>(t->pts, n, t->pts64, t->pts32);
  CKD_LAUNCH_CHECK();
  k_node_boxes<<<(unsigned)cdiv((int64_t)n_nodes * 2 * D, 256), 256, 0, s>>>(
      B.box, B.cell, (int64_t)n_nodes * 2 * D, t->box, t->cell, t->box32, t->cell32);
  CKD_LAUNCH_CHECK();
  k_node_records<D><<<(unsigned)cdiv(n_nodes, 128), 128, 0, s>>>(B.meta, n_nodes, B.box, t->meta,
                                                                 t->pair, t->centre);
  CKD_LAUNCH_CHECK();
  CKD_CUDA(cudaStreamSynchronize(s));
  if (err == 3) return fail(CKD_ERR_TIMEOUT, "build: a tile copy into shared memory timed out");
  if (err) return fail(CKD_ERR_CUDA, "internal error: inconsistent partition in build");
  // leaves = (nodes + 1) / 2 for each full binary tree
  t->n_leaves = (n_nodes + T) / 2;
  return CKD_OK;
}

}  // namespace

ckd_status build_dispatch(ckd_tree* t, const void* pts_dev, int dtype, cudaStream_t s) {
  switch (t->d) {
#define CKD_BD(DD) \
  case DD: return build_impl<DD>(t, pts_dev, dtype, s);
    CKD_BD(1) CKD_BD(2) CKD_BD(3) CKD_BD(4) CKD_BD(5) CKD_BD(6) CKD_BD(7) CKD_BD(8)
#undef CKD_BD
  }
  return fail(CKD_ERR_BAD_DIM, "dimensionality must be 1..8");
}

}  // namespace ckd
