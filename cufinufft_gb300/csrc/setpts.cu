// setpts.cu -- bin sort of the nonuniform points (the setpts stage).
//
// The reference sorts in four launches per call (src/2d/spread2d_wrapper.cu:
// 386-613): CalcBinSize_noghost (per-point bin + atomic rank), a Thrust
// exclusive scan, CalcInvertofGlobalSortIdx (scatter of the permutation),
// then CalcSubProb / inclusive scan / MapBintoSubProb for the subproblem
// method and a host readback of their number.  Here:
//   * k_bin_count places every point on the fine grid (place_coord) and ranks
//     it inside its bin -- or directly inside its (bin, bank class), whose
//     counts sum to the bin's -- with one warp-aggregated atomic (one per
//     distinct key in a warp, so clustered points do not serialise on one
//     counter); a few thousand bins or fewer keep their counters a sector
//     apart (kCountStride), or all atomics meet in a handful of L2 sectors,
//     and where many points share a counter blocks count in shared memory
//     first (k_bin_count_crowded);
//   * k_bin_scan turns the counters into bin counts, bin starts and
//     subproblem starts in one pass (two launches beyond 4096 bins);
//   * k_permute (large 3D FP32 sets: k_permute and k_gather_points) writes the
//     sorted structure-of-arrays copy the spread and
//     interp kernels stream -- caller index, first tap and offset per axis --
//     and, in further blocks of the same launch, the subproblem headers (binary
//     search, balanced even when one bin holds most of the points).  Headers
//     are written for the upper bound of their number, the surplus empty; the
//     host learns the number with the one wait that ends setpts (the caller's
//     coordinates are read until the last of these kernels).
// Points come from the caller's coordinates, from the plan's stored first
// taps and offsets (a new layout), or from FP64 coordinates for an FP32 chain
// (placed in FP64, the offset rounded afterwards).
// 1e5 points, 512^2 grid: 12 launches and ~45 us of device time -> 5 launches;
// set_pts and execute together 131 -> 60 us a call in a stream of calls.
#include "device_common.cuh"
#include "kernels.h"

namespace cfg {

constexpr int kPlaceThreads = 256;

// i / bs by a reciprocal: floor(2^32 / bs) + 1 overestimates by at most one
// for i, bs < 2^31 with i bs < 2^33, which the check takes back.
__device__ __forceinline__ int bin_div(int i, int bs, unsigned magic) {
  int q = bs == 1 ? i : (int)__umulhi((unsigned)i, magic);
  if (q * bs > i) --q;
  return q;
}

// First taps and offsets of point i, and its bin.
template <typename T, int SRC>
__device__ __forceinline__ int point_bin(const PlaceArgs<T>& a, int i, int i0[3], T d[3], int lc[3]) {
  int b = 0, mul = 1;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (k < a.dim) {
      if (SRC == kSrcStored) {
        i0[k] = a.src_i0[k][i];
        d[k] = a.src_d[k][i];
      } else if (SRC == kSrcNarrow) {
        double dd;
        place_coord<double>(a.xd[k][i], a.axd[k], i0[k], dd);
        d[k] = (T)dd;
      } else {
        place_coord<T>(a.x[k][i], a.ax[k], i0[k], d[k]);
      }
      const int q = bin_div(i0[k], a.bs[k], a.magic[k]);
      lc[k] = i0[k] - q * a.bs[k];
      b += mul * q;
      mul *= a.nb[k];
    } else {
      lc[k] = 0;
    }
  }
  return b;
}

// Class of a point inside its bin, from its cell inside the bin: its bank
// class (see BankOrder), or the cell (cell order).
__device__ __forceinline__ int order_class(const BankOrder& o, const int* bs, const int lc[3]) {
  if (!o.cell_order) return (lc[0] + o.tx * (lc[1] + o.ty * lc[2])) & (o.ncls - 1);
  return lc[0] + bs[0] * (lc[1] + bs[1] * lc[2]);
}

// Warp-aggregated rank: one atomic per distinct key in the warp.
__device__ __forceinline__ int agg_rank(unsigned act, int key, int* counter) {
  const int lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(act, key);
  const int leader = __ffs(peers) - 1;
  int first = 0;
  if (lane == leader) first = atomicAdd(counter, __popc(peers));
  first = __shfl_sync(peers, first, leader);
  return first + __popc(peers & ((1u << lane) - 1u));
}

// Cell order (BankOrder::cell_order): a bin's points on dense cells (at least
// dense_min points) come first, sorted by cell -- cls_start is the exclusive
// scan of the dense cells' counts only -- then the bin's other points in
// arbitrary order, ranked by the per-bin counter sparse_count.  r is the
// point's rank inside its cell.  Called by the lanes in act together.
__device__ __forceinline__ int cell_position(const BankOrder& o, const int* start, unsigned act, int b,
                                             int c, int r) {
  const long long k0 = (long long)b * o.ncls;
  const int bin0 = o.cls_start[k0];
  const bool dense = o.cls_count[k0 + c] >= o.dense_min;
  const unsigned sparse_lanes = __ballot_sync(act, !dense);
  if (dense) return start[b] + (o.cls_start[k0 + c] - bin0) + r;
  const int sr = agg_rank(sparse_lanes, b, o.sparse_count + b);
  return start[b] + (o.cls_start[k0 + o.ncls] - bin0) + sr;
}

// Position inside its bin of the point ranked r in class c: round-robin over
// the classes, rounds shrinking as classes run out.
__device__ __forceinline__ int interleave_pos(const BankOrder& o, int b, int c, int r) {
  const int4* cnt = reinterpret_cast<const int4*>(o.cls_count + (long long)b * o.ncls);  // ncls 8 or 16
  int pos = 0;
  for (int k = 0; k < o.ncls; k += 4) {
    const int4 v = __ldg(cnt + (k >> 2));
    const int n[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int u = 0; u < 4; ++u) pos += min(n[u], r) + ((k + u < c && n[u] > r) ? 1 : 0);
  }
  return pos;
}

template <typename T, int SRC>
__global__ void __launch_bounds__(kPlaceThreads) k_bin_count(PlaceArgs<T> a) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  // warp-uniform trip count so the warp stays converged for __match_any_sync
  for (long long base = (long long)blockIdx.x * blockDim.x; base < a.M; base += stride) {
    const long long ii = base + threadIdx.x;
    const bool active = ii < a.M;
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (!active) continue;
    const int i = (int)ii;
    int i0[3], lc[3];
    T d[3];
    const int b = point_bin<T, SRC>(a, i, i0, d, lc);
    int r;
    if (a.bank.cls_count) {
      if (a.bank.cell_order == 1) agg_rank(act, b, &a.count[b]);
      const int key = b * a.bank.ncls + order_class(a.bank, a.bs, lc);
      r = agg_rank(act, key, a.bank.cls_count + key);
    } else {
      r = agg_rank(act, b, a.raw + (size_t)b * a.raw_stride);
    }
    a.rank[i] = r;
  }
}

// The same for few counters (crowded_sort): a block ranks its points in shared
// memory, reserves its share of every counter with one atomic, and adds the base it
// got.  Key and rank of a point wait in one register (12 + 13 bits).
template <typename T, int SRC, int U>
__global__ void __launch_bounds__(kPlaceThreads) k_bin_count_crowded(PlaceArgs<T> a) {
  __shared__ int s_count[kCrowdedKeys];
  static_assert(kCrowdedKeys <= 1 << 12 && U * kPlaceThreads <= 1 << 13, "key and rank share an int");
  for (int k = threadIdx.x; k < a.crowded_keys; k += kPlaceThreads) s_count[k] = 0;
  __syncthreads();
  const long long base = (long long)blockIdx.x * (U * kPlaceThreads) + threadIdx.x;
  int at[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = base + u * kPlaceThreads;
    if (i >= a.M) continue;
    int i0[3], lc[3];
    T d[3];
    const int b = point_bin<T, SRC>(a, (int)i, i0, d, lc);
    const int key = a.bank.cls_count ? b * a.bank.ncls + order_class(a.bank, a.bs, lc) : b;
    at[u] = key << 13 | atomicAdd(&s_count[key], 1);
  }
  __syncthreads();
  int* counter = a.bank.cls_count ? a.bank.cls_count : a.raw;
  for (int k = threadIdx.x; k < a.crowded_keys; k += kPlaceThreads)
    if (s_count[k]) s_count[k] = atomicAdd(counter + k, s_count[k]);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const long long i = base + u * kPlaceThreads;
    if (i < a.M) a.rank[i] = s_count[at[u] >> 13] + (at[u] & 0x1fff);
  }
}

// Subproblem headers (a part of k_permute): the subproblem's bin
// by binary search, its point range (subproblem js of bin b: points start[b] +
// js maxsub, at most maxsub of them) and its tile origin (the bin's first
// cell); those past the total, up to the bound that the tables are written for, are
// empty and no later launch reaches them.
__device__ __forceinline__ void write_header(const SubHdrArgs& h, const int* start, const int* count,
                                             const int* bs, const int* nb, int sidx) {
  const int total = h.sub_start[h.nbins];
  SubHdr o;
  o.p0 = o.np = o.ox = o.oy = o.oz = o.pad0 = o.pad1 = o.pad2 = 0;
  int lo = 0;
  if (sidx < total) {
    int hi = h.nbins;  // invariant: sub_start[lo] <= sidx < sub_start[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (h.sub_start[mid] <= sidx) lo = mid;
      else hi = mid;
    }
    const int js = sidx - h.sub_start[lo];
    o.p0 = start[lo] + js * h.maxsub;
    o.np = min(h.maxsub, count[lo] - js * h.maxsub);
    o.ox = (lo % nb[0]) * bs[0];
    o.oy = ((lo / nb[0]) % nb[1]) * bs[1];
    o.oz = (lo / (nb[0] * nb[1])) * bs[2];
  }
  h.sub_to_bin[sidx] = lo;
  h.hdr[sidx] = o;
}

template <typename T, int SRC>
__device__ __forceinline__ void write_point(const PlaceArgs<T>& a, int pos, int idx, const int i0[3], const T d[3]) {
  a.idx[pos] = idx;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (k < a.dim) {
      a.i0[k][pos] = i0[k];
      a.d[k][pos] = d[k];
    }
  }
}

// Blocks [0, pblocks) permute, the others write headers.  WHOLE writes every
// point's sorted copy, seven scattered words in 3D, each a sector of its own; not
// WHOLE writes only where the point came from, and k_gather_points reads the points
// in sorted order and writes the copies in full lines.
template <typename T, int SRC, bool WHOLE>
__global__ void __launch_bounds__(kPlaceThreads) k_permute(PlaceArgs<T> a, SubHdrArgs h, int pblocks) {
  if ((int)blockIdx.x >= pblocks) {
    const int sidx = ((int)blockIdx.x - pblocks) * blockDim.x + threadIdx.x;
    if (sidx < h.nsub) write_header(h, a.start, a.count, a.bs, a.nb, sidx);
    return;
  }
  const long long stride = (long long)pblocks * blockDim.x;
  // warp-uniform trip count: cell order ranks sparse points warp-aggregated
  for (long long base = (long long)blockIdx.x * blockDim.x; base < a.M; base += stride) {
    const long long ii = base + threadIdx.x;
    const bool active = ii < a.M;
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (!active) continue;
    const int i = (int)ii;
    int i0[3], lc[3];
    T d[3];
    const int b = point_bin<T, SRC>(a, i, i0, d, lc);
    const int r = a.rank[i];
    int pos;
    if (!a.bank.cls_count) pos = a.start[b] + r;
    else if (a.bank.cell_order == 2) pos = a.bank.cls_start[(long long)b * a.bank.ncls + order_class(a.bank, a.bs, lc)] + r;
    else if (a.bank.cell_order) pos = cell_position(a.bank, a.start, act, b, order_class(a.bank, a.bs, lc), r);
    else pos = a.start[b] + interleave_pos(a.bank, b, order_class(a.bank, a.bs, lc), r);
    if (WHOLE) write_point<T, SRC>(a, pos, SRC == kSrcStored ? a.src_idx[i] : i, i0, d);
    else a.idx[pos] = i;
  }
}

template <typename T, int SRC>
__global__ void __launch_bounds__(kPlaceThreads) k_gather_points(PlaceArgs<T> a) {
  const int pos = blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= a.M) return;
  const int i = a.idx[pos];
  int i0[3], lc[3];
  T d[3];
  point_bin<T, SRC>(a, i, i0, d, lc);
  write_point<T, SRC>(a, pos, SRC == kSrcStored ? a.src_idx[i] : i, i0, d);
}

// gpu_sort = 0 with method 1 keeps the caller's order (reference "GM",
// TrivialGlobalSortIdx, src/precision_independent.cu:98-105).
template <typename T, int SRC>
__global__ void __launch_bounds__(kPlaceThreads) k_place_unsorted(PlaceArgs<T> a) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.M; i += gridDim.x * blockDim.x) {
    int i0[3], lc[3];
    T d[3];
    point_bin<T, SRC>(a, i, i0, d, lc);
    a.idx[i] = i;
    for (int k = 0; k < 3; ++k) {
      if (k < a.dim) {
        a.i0[k][i] = i0[k];
        a.d[k][i] = d[k];
      }
    }
  }
}

static int place_grid(int M) {
  long long b = ((long long)M + kPlaceThreads - 1) / kPlaceThreads;
  if (b > 152LL * 64) b = 152LL * 64;
  return b < 1 ? 1 : (int)b;
}

static void set_magic(const int bs[3], unsigned magic[3]) {
  for (int k = 0; k < 3; ++k) magic[k] = bs[k] > 1 ? (unsigned)((1ull << 32) / (unsigned)bs[k] + 1) : 0u;
}

// One kernel instance per point source.
#define CFG_SRC_SWITCH(KERNEL, GRID, ...)                                              \
  switch (a.src) {                                                                     \
    case kSrcStored: KERNEL<T, kSrcStored><<<GRID, kPlaceThreads, 0, s>>>(__VA_ARGS__); break; \
    case kSrcNarrow: KERNEL<T, kSrcNarrow><<<GRID, kPlaceThreads, 0, s>>>(__VA_ARGS__); break; \
    default: KERNEL<T, kSrcCoords><<<GRID, kPlaceThreads, 0, s>>>(__VA_ARGS__); break;  \
  }

#define CFG_SRC_SWITCH2(KERNEL, ARG, GRID, ...)                                        \
  switch (a.src) {                                                                     \
    case kSrcStored: KERNEL<T, kSrcStored, ARG><<<GRID, kPlaceThreads, 0, s>>>(__VA_ARGS__); break; \
    case kSrcNarrow: KERNEL<T, kSrcNarrow, ARG><<<GRID, kPlaceThreads, 0, s>>>(__VA_ARGS__); break; \
    default: KERNEL<T, kSrcCoords, ARG><<<GRID, kPlaceThreads, 0, s>>>(__VA_ARGS__); break;  \
  }

template <typename T, int U> static cudaError_t count_crowded(const PlaceArgs<T>& a, cudaStream_t s) {
  CFG_SRC_SWITCH2(k_bin_count_crowded, U, (a.M + U * kPlaceThreads - 1) / (U * kPlaceThreads), a)
  return cudaGetLastError();
}
template <typename T> cudaError_t launch_bin_count(PlaceArgs<T> a, cudaStream_t s) {
  if (a.M == 0) return cudaSuccess;
  set_magic(a.bs, a.magic);
  if (a.crowded_keys > 0) {
    // points per thread: many share a block's counters, few even out the blocks (FP64
    // placement is arithmetic)
    const bool wide = a.M >= 152 * 32 * kPlaceThreads;
    if (sizeof(T) == 8 || a.src == kSrcNarrow) return wide ? count_crowded<T, 8>(a, s) : count_crowded<T, 4>(a, s);
    return wide ? count_crowded<T, 32>(a, s) : count_crowded<T, 8>(a, s);
  }
  CFG_SRC_SWITCH(k_bin_count, place_grid(a.M), a)
  return cudaGetLastError();
}
// 3D FP32 points from which the permutation goes in two steps (one / two, us: 1e6
// points in 64^3 modes 37 / 28, 4e6 195 / 92; 3e5 14.5 / 12.3).  In 2D ordered
// trajectories scatter into few lines anyway (radial, 1e6: 9.6 / 17), and FP64
// points would be placed on the grid once more, which is bound by the FP64 unit
// (1e6: 118 / 219).
constexpr int kGatherPoints = 250000;
template <typename T> cudaError_t launch_permute(PlaceArgs<T> a, const SubHdrArgs& h, cudaStream_t s) {
  if (a.M == 0) return cudaSuccess;
  set_magic(a.bs, a.magic);
  const int pb = place_grid(a.M), hb = (h.nsub + kPlaceThreads - 1) / kPlaceThreads;
  if constexpr (sizeof(T) == 4) {
    if (a.src != kSrcNarrow && a.dim == 3 && a.M >= kGatherPoints) {
      const int gb = (a.M + kPlaceThreads - 1) / kPlaceThreads;
      if (a.src == kSrcStored) {
        k_permute<T, kSrcStored, false><<<pb + hb, kPlaceThreads, 0, s>>>(a, h, pb);
        k_gather_points<T, kSrcStored><<<gb, kPlaceThreads, 0, s>>>(a);
      } else {
        k_permute<T, kSrcCoords, false><<<pb + hb, kPlaceThreads, 0, s>>>(a, h, pb);
        k_gather_points<T, kSrcCoords><<<gb, kPlaceThreads, 0, s>>>(a);
      }
      return cudaGetLastError();
    }
  }
  CFG_SRC_SWITCH2(k_permute, true, pb + hb, a, h, pb)
  return cudaGetLastError();
}
template <typename T> cudaError_t launch_place_unsorted(PlaceArgs<T> a, cudaStream_t s) {
  if (a.M == 0) return cudaSuccess;
  set_magic(a.bs, a.magic);
  CFG_SRC_SWITCH(k_place_unsorted, place_grid(a.M), a)
  return cudaGetLastError();
}

template cudaError_t launch_bin_count<float>(PlaceArgs<float>, cudaStream_t);
template cudaError_t launch_bin_count<double>(PlaceArgs<double>, cudaStream_t);
template cudaError_t launch_permute<float>(PlaceArgs<float>, const SubHdrArgs&, cudaStream_t);
template cudaError_t launch_permute<double>(PlaceArgs<double>, const SubHdrArgs&, cudaStream_t);
template cudaError_t launch_place_unsorted<float>(PlaceArgs<float>, cudaStream_t);
template cudaError_t launch_place_unsorted<double>(PlaceArgs<double>, cudaStream_t);

// ---------------------------------------------------------------------------
// Occupancy counts for the selector's features, over bins a.bs x a.nb, of the
// points of any source (so that a layout can be chosen before the sort).
template <typename T, int SRC>
__global__ void __launch_bounds__(kPlaceThreads) k_feature_count(PlaceArgs<T> a) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long base = (long long)blockIdx.x * blockDim.x; base < a.M; base += stride) {
    const long long ii = base + threadIdx.x;
    const bool active = ii < a.M;
    const unsigned act = __ballot_sync(0xffffffffu, active);
    if (!active) continue;
    int i0[3], lc[3];
    T d[3];
    const int b = point_bin<T, SRC>(a, (int)ii, i0, d, lc);
    const unsigned peers = __match_any_sync(act, b);
    if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&a.count[b], __popc(peers));
  }
}

template <typename T> cudaError_t launch_feature_count(PlaceArgs<T> a, cudaStream_t s) {
  if (a.M == 0) return cudaSuccess;
  set_magic(a.bs, a.magic);
  CFG_SRC_SWITCH(k_feature_count, place_grid(a.M), a)
  return cudaGetLastError();
}
template cudaError_t launch_feature_count<float>(PlaceArgs<float>, cudaStream_t);
template cudaError_t launch_feature_count<double>(PlaceArgs<double>, cudaStream_t);

// ---------------------------------------------------------------------------
// Exclusive scan: 1024 threads x 4 items per block; block totals are scanned
// by one block (up to 4096 blocks, i.e. 16.7M entries), then added back.
constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int kScanMaxBlocks = 4096;

__device__ __forceinline__ int scan_load(const int* in, int i, int n, int mode, int div) {
  if (i >= n) return 0;
  int v = in[i];
  if (mode == 2) return v >= div ? v : 0;  // counts of at least div only
  return mode == 1 ? (v + div - 1) / div : v;
}

// Block-wide exclusive scan of one value per thread; returns the block total.
__device__ __forceinline__ int block_exclusive_scan(int v, int& excl) {
  __shared__ int warp_tot[kScanThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  if (w == 0) {
    int t = lane < (int)(blockDim.x >> 5) ? warp_tot[lane] : 0;
    int ti = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int n = __shfl_up_sync(0xffffffffu, ti, o);
      if (lane >= o) ti += n;
    }
    warp_tot[lane] = ti - t;  // exclusive warp offsets
  }
  __syncthreads();
  excl = warp_tot[w] + incl - v;
  __shared__ int tot;
  if (threadIdx.x == blockDim.x - 1) tot = excl + v;  // inclusive sum of the last thread
  __syncthreads();
  const int total = tot;
  __syncthreads();
  return total;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_partial(const int* in, int n, int mode, int div,
                                                              int* partial) {
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) s += scan_load(in, base + k, n, mode, div);
  int excl;
  int total = block_exclusive_scan(s, excl);
  if (threadIdx.x == 0) partial[blockIdx.x] = total;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_partials(int* partial, int nblocks) {
  // one block: exclusive scan of nblocks (<= 4096) partial sums in place
  int v[kScanItems];
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    int i = threadIdx.x * kScanItems + k;
    v[k] = i < nblocks ? partial[i] : 0;
    s += v[k];
  }
  int excl;
  block_exclusive_scan(s, excl);
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    int i = threadIdx.x * kScanItems + k;
    if (i < nblocks) partial[i] = excl;
    excl += v[k];
  }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_final(const int* in, int n, int mode, int div,
                                                            const int* partial, int* out) {
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int v[kScanItems];
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = scan_load(in, base + k, n, mode, div);
    s += v[k];
  }
  int excl;
  int total = block_exclusive_scan(s, excl);
  excl += partial[blockIdx.x];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) out[base + k] = excl;
    excl += v[k];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = partial[blockIdx.x] + total;
}

int scan_tmp_ints(int n) {
  int nb = (n + kScanTile - 1) / kScanTile;
  return nb < 1 ? 1 : nb;
}

cudaError_t launch_scan(const int* in, int* out, int n, int mode, int div, int* tmp, cudaStream_t s) {
  if (n <= 0) return cudaMemsetAsync(out, 0, sizeof(int), s);
  int nb = scan_tmp_ints(n);
  if (nb > kScanMaxBlocks) return cudaErrorInvalidValue;
  k_scan_partial<<<nb, kScanThreads, 0, s>>>(in, n, mode, div, tmp);
  k_scan_partials<<<1, kScanThreads, 0, s>>>(tmp, nb);
  k_scan_final<<<nb, kScanThreads, 0, s>>>(in, n, mode, div, tmp, out);
  return cudaGetLastError();
}

// Bin counts, bin starts and subproblem starts in one pass: the counters of
// bin b are the `per` ints at raw + b raw_stride (its classes, or itself), a
// bin of c points holds ceil(c / maxsub) subproblems (maxsub 0: none).  Both
// running sums travel in one 64-bit scan, points low, subproblems high.
__device__ __forceinline__ unsigned long long block_exclusive_scan64(unsigned long long v, unsigned long long& excl) {
  __shared__ unsigned long long warp_tot[kScanThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  __syncthreads();
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  unsigned long long before = 0, total = 0;
  for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
    const unsigned long long t = warp_tot[k];
    if (k < w) before += t;
    total += t;
  }
  excl = before + incl - v;
  return total;
}

__device__ __forceinline__ int bin_total(const BinScanArgs& a, int b) {
  if (b >= a.nbins) return 0;
  if (a.cell_start) return a.cell_start[(size_t)(b + 1) * a.ncell] - a.cell_start[(size_t)b * a.ncell];
  const int* c = a.raw + (size_t)b * a.raw_stride;
  int n = 0;
  if ((a.per & 3) == 0) {  // classes: 8 or 16 counters, 16-byte aligned
    for (int k = 0; k < a.per; k += 4) {
      const int4 v = *reinterpret_cast<const int4*>(c + k);
      n += v.x + v.y + v.z + v.w;
    }
    return n;
  }
  return c[0];
}
__device__ __forceinline__ unsigned long long bin_sums(const BinScanArgs& a, int n) {
  const unsigned long long subs = a.maxsub > 0 && n > 0 ? ((unsigned)n - 1u) / (unsigned)a.maxsub + 1u : 0u;
  return (subs << 32) | (unsigned)n;
}

__global__ void __launch_bounds__(kScanThreads) k_bin_sums(BinScanArgs a) {
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  unsigned long long v = 0, excl;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int n = bin_total(a, base + k);
    if (base + k < a.nbins) a.count[base + k] = n;
    v += bin_sums(a, n);
  }
  const unsigned long long total = block_exclusive_scan64(v, excl);
  if (threadIdx.x == 0) a.partial[blockIdx.x] = total;
}

// ONE: the only block, which also sums the counters.
template <bool ONE>
__global__ void __launch_bounds__(kScanThreads) k_bin_scan(BinScanArgs a) {
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int n[kScanItems];
  unsigned long long v = 0, excl, first = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int b = base + k;
    n[k] = ONE ? bin_total(a, b) : (b < a.nbins ? a.count[b] : 0);
    if (ONE && b < a.nbins) a.count[b] = n[k];
    v += bin_sums(a, n[k]);
  }
  if (!ONE) {  // the blocks before this one
    unsigned long long w = 0, unused;
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += blockDim.x) w += a.partial[k];
    first = block_exclusive_scan64(w, unused);
  }
  const unsigned long long total = block_exclusive_scan64(v, excl) + first;
  excl += first;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int b = base + k;
    if (b < a.nbins) {
      a.start[b] = (int)(unsigned)excl;
      a.sub_start[b] = (int)(excl >> 32);
    }
    excl += bin_sums(a, n[k]);
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    a.start[a.nbins] = (int)(unsigned)total;
    a.sub_start[a.nbins] = (int)(total >> 32);
    if (a.total) *a.total = (int)(total >> 32);
  }
}

int bin_scan_partials(int nbins) { return (nbins + kScanTile - 1) / kScanTile; }

cudaError_t launch_bin_scan(const BinScanArgs& a, cudaStream_t s) {
  const int nb = bin_scan_partials(a.nbins);
  if (nb < 1) return cudaErrorInvalidValue;
  if (nb == 1) {
    k_bin_scan<true><<<1, kScanThreads, 0, s>>>(a);
  } else {
    k_bin_sums<<<nb, kScanThreads, 0, s>>>(a);
    k_bin_scan<false><<<nb, kScanThreads, 0, s>>>(a);
  }
  return cudaGetLastError();
}

__global__ void k_classify_subproblems(SubClassArgs a) {
  const int total = a.sub_total[0];
  for (int sidx = blockIdx.x * blockDim.x + threadIdx.x; sidx < a.nsub; sidx += gridDim.x * blockDim.x) {
    if (sidx >= total) {  // past the last subproblem, inside the launch bound
      a.dense[sidx] = 0;
      if (a.ndense) a.ndense[sidx] = 0;
      continue;
    }
    const int b = a.sub_to_bin[sidx];
    const int p0 = a.start[b] + (sidx - a.sub_start[b]) * a.maxsub;
    const int lx = a.i0[0][p0] % a.bs[0];
    const int ly = a.dim > 1 ? a.i0[1][p0] % a.bs[1] : 0;
    const int lz = a.dim > 2 ? a.i0[2][p0] % a.bs[2] : 0;
    const int c = lx + a.bs[0] * (ly + a.bs[1] * lz);
    a.dense[sidx] = a.cls_count[(long long)b * a.ncls + c] >= a.dense_min ? 1 : 0;
    if (a.ndense) {
      const int js = sidx - a.sub_start[b];
      const int np = min(a.maxsub, a.count[b] - js * a.maxsub);
      const int nd = a.cls_start[(long long)(b + 1) * a.ncls] - a.cls_start[(long long)b * a.ncls];
      a.ndense[sidx] = max(0, min(np, nd - js * a.maxsub));
    }
  }
}

cudaError_t launch_classify_subproblems(const SubClassArgs& a, cudaStream_t s) {
  if (a.nsub <= 0) return cudaSuccess;
  int blocks = (a.nsub + 255) / 256;
  if (blocks > 152 * 16) blocks = 152 * 16;
  k_classify_subproblems<<<blocks, 256, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace cfg
