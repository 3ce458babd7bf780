// spread_col.cuh -- 3D FP32 spreading (type 1) by slabs, with the points of a
// column of cells summed in registers (method 2 where cells hold points to
// share).
//
// As in the slab kernel (k_spread_sm_slab) the tile's z-planes are owned, here by
// half as many warps: warp w alone writes the planes z = w and w + NW (mod NS), NW =
// ceil(NS / 2), so it adds every point to two planes with one read of the point's x
// and y values, lanes over the (x, y) taps, R = 32 / NS rows per instruction.  The
// block first orders its points by (column of cells, z) -- a counting sort in
// shared memory, up to kColSort points at a time.  The points of a column meet one
// residue in at most two planes per NS cells of z, so their taps fall on the same
// cells: the warp sums them in registers and goes to the tile (plain loads and
// stores, a __syncwarp between) only where the cells change, which a ballot over
// the chunk's points finds.
//
// Reading and writing the tile for every point was 8 of a point-plane's 14 shared
// wavefronts and bound the slab kernel (115 wavefronts and 404 instructions per
// point at ns 8, shared memory 82% busy); here it is 38 and 147, bound by issue and
// latency (60% of issue slots, 19 warps per SM: the tile's shared memory).  One
// plane per warp took 959 us where two take 803 (4e6 points, 128^3 cells, ns 8);
// a register window over all ns planes above a column, the columns shared out to
// four warps, 2.3 ms: eight warps per SM and a barrier per column.
// Spread stage, slab / this kernel (us), best bins of each: even points, ns 8: 4e6
// in 128^3 cells 1609 / 803, 3.2e7 in 256^3 12284 / 5981; half of them clustered
// 12391 / 6450; 0.5 points per cell 3294 / 2855, 0.2 202 / 239; 1.9 points per cell ns
// 7 1736 / 820, ns 6 1465 / 775, ns 4 616 / 529 (0.5: 175 / 199); the line is
// column_spread's.  Cell-run layout, 3.2e7 half-clustered points 8267 / 5650.
#pragma once

#include "df.cuh"
#include "kernels.h"

namespace cfg {

constexpr int kColChunk = 32;     // points staged at a time
constexpr int kColSort = 1024;    // points ordered at a time
constexpr int kColKeys = 4096;    // cells of a bin at most

// A stage: per point one row of ColRow::bytes -- c kx per tap (complex), kz per
// warp at the two planes that warp adds it to, ky per tap, the two ky of a lane
// that takes two or more rows side by side (slot m R + y: rows 2m R + y and (2m +
// 1) R + y) -- then per warp and point those planes' first cells.  Reads of at
// most 8 bytes: a 16-byte read of a few addresses costs a wavefront per quarter
// warp (values held twice over, ready for packed FMAs: 46 wavefronts a point).
template <int NS> struct ColRow {
  static constexpr int R = 32 / NS, NR = (NS + R - 1) / R, NPR = (NR + 1) / 2, NW = (NS + 1) / 2;
  static constexpr bool kPairs = NR >= 2;
  static constexpr int kz = NS * 8;
  static constexpr int ky = kz + NW * 8;
  static constexpr int used = ky + (kPairs ? NPR * R * 8 : NS * 4);
  static constexpr int bytes = (used + 23) / 16 * 16 + 8;  // 8 (mod 16): rows spread over the banks
  static constexpr int base = kColChunk * bytes;
  static constexpr size_t stage = (base + kColChunk * NW * 8 + 15) / 16 * 16;
};
// Row pitch: one instruction's rows in distinct banks (slab_pitch), but not where
// that would pad the row by more than a sixth: the tile is reached only where the
// cells change, and blocks per SM count more (8^3 bins at ns 8: pitch 15 or 24;
// pitch 16 with the halves of odd rows swapped, no conflicts, was no faster).
__host__ __device__ constexpr int col_pitch(int tx, int ns) {
  return 6 * slab_pitch(tx, ns) <= 7 * tx ? slab_pitch(tx, ns) : tx;
}
// The sort's counters lie where the stages do, which are not in use then.
template <int NS>
size_t col_bytes(const BinTables& bt) {
  const size_t cells = (size_t)col_pitch(bt.bs[0] + NS - 1, NS) * (bt.bs[1] + NS - 1) * (bt.bs[2] + NS - 1);
  const long long keys = (long long)bt.bs[0] * bt.bs[1] * bt.bs[2];
  const size_t count = ((size_t)keys * sizeof(int) + 15) & ~(size_t)15, stages = 2 * ColRow<NS>::stage;
  return ((cells * sizeof(float2) + 15) & ~(size_t)15) + (stages > count ? stages : count) +
         kColSort * sizeof(unsigned short);
}
inline bool col_bins(const BinTables& bt) { return (long long)bt.bs[0] * bt.bs[1] * bt.bs[2] <= kColKeys; }

// Exclusive scan of n shared ints by the block (n <= items * blockDim.x for the
// items each thread takes), in place.
template <int NW>
__device__ __forceinline__ void block_scan_ints(int* v, int n) {
  __shared__ int s_tot[NW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (n + 32 * NW - 1) / (32 * NW), k0 = threadIdx.x * per, k1 = min(n, k0 + per);
  int sum = 0;
  for (int k = k0; k < k1; ++k) sum += v[k];
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) s_tot[warp] = incl;
  __syncthreads();
  int run = incl - sum;
  for (int w = 0; w < warp; ++w) run += s_tot[w];
  for (int k = k0; k < k1; ++k) {
    const int x = v[k];
    v[k] = run;
    run += x;
  }
  __syncthreads();
}

template <int NS>
__global__ void __launch_bounds__(32 * ColRow<NS>::NW, NS <= 8 ? 5 : 2)
k_spread_sm_col(SpreadArgs<float> a, int split) {
  using Row = ColRow<NS>;
  constexpr int HD = horner_degree<float>(NS);
  constexpr int R = Row::R;                  // tile rows per warp instruction
  constexpr int NR = Row::NR;                // instructions per plane
  constexpr int NW = Row::NW;                // warps
  constexpr int CH = kColChunk;
  static_assert(CH == 32, "a lane looks after a point's change of cells");
  constexpr int kPer = (kColSort + 32 * NW - 1) / (32 * NW);
  // cell-run layout: a subproblem that starts on a dense cell leaves its
  // leading dense points to k_spread_sm_run (split) or all of them (not)
  int first = 0;
  if (a.sub_dense && a.sub_dense[blockIdx.x]) {
    if (!split) return;
    first = a.sub_ndense[blockIdx.x];
  }
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const SubTile st = sub_tile_block<3, NS>(a.bins, blockIdx.x);
  if (st.np <= 0) return;  // block-uniform
  if (first >= st.np) return;  // block-uniform
  const int PX = col_pitch(st.TX, NS);
  const int PP = PX * st.TY;                  // plane stride
  const int ncell = PP * st.TZ;
  float2* tile = reinterpret_cast<float2*>(smem_raw);
  unsigned short* s_perm =
      reinterpret_cast<unsigned short*>(smem_raw + (((size_t)ncell * sizeof(float2) + 15) & ~(size_t)15));
  unsigned char* stage0 = reinterpret_cast<unsigned char*>(s_perm + kColSort);  // two stages
  for (int i = threadIdx.x; i < ncell; i += blockDim.x) tile[i] = make_float2(0.f, 0.f);
  const float2* cin = a.c_in + (size_t)blockIdx.y * a.M;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int dx = lane % NS, dyl = lane / NS, yc = min(dyl, R - 1);
  const bool lane_on = lane < R * NS;
  constexpr bool kFullRows = 32 % NS == 0 && (NS * NS) % 32 == 0;  // ns 8, 16: all lanes, rows in range
  const int nkey = a.bins.bs[0] * a.bins.bs[1] * a.bins.bs[2];
  // the sums of the warp's two planes and their first cells (-1: none yet)
  float2 acc0[NR], acc1[NR];
  int cur0 = -1, cur1 = -1;
#pragma unroll
  for (int r = 0; r < NR; ++r) acc0[r] = acc1[r] = make_float2(0.f, 0.f);
  auto flush = [&](int cur, float2* acc) {
    if (cur >= 0) {
      __syncwarp();  // the previous flush's stores
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int dy = r * R + dyl;
        if (kFullRows || (lane_on && dy < NS)) {
          float2* cell = tile + cur + dx + dy * PX;
          *cell = add2(*cell, acc[r]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) acc[r] = make_float2(0.f, 0.f);
  };
  for (int g0 = first; g0 < st.np; g0 += kColSort) {
    const int ng = min(kColSort, st.np - g0);
    __syncthreads();  // every read of the stages and of s_perm is done
    int* s_count = reinterpret_cast<int*>(stage0);
    for (int i = threadIdx.x; i < nkey; i += blockDim.x) s_count[i] = 0;
    __syncthreads();
    int key[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      const int i = u * 32 * NW + threadIdx.x;
      key[u] = -1;
      if (i < ng) {
        const int p = st.p0 + g0 + i;
        const int lx = a.pts.i0[0][p] - st.ox, ly = a.pts.i0[1][p] - st.oy, lz = a.pts.i0[2][p] - st.oz;
        const int k = (ly * a.bins.bs[0] + lx) * a.bins.bs[2] + lz;
        key[u] = k * kColSort + atomicAdd(s_count + k, 1);  // rank < kColSort
      }
    }
    __syncthreads();
    block_scan_ints<NW>(s_count, nkey);
#pragma unroll
    for (int u = 0; u < kPer; ++u)
      if (key[u] >= 0)
        s_perm[s_count[key[u] / kColSort] + key[u] % kColSort] = (unsigned short)(u * 32 * NW + threadIdx.x);
    __syncthreads();
    // thread (q, j) stages taps j and j + NW of a chunk's point q, read while the
    // chunk before it is added
    float2 v = make_float2(0.f, 0.f);
    float d[3] = {0.f, 0.f, 0.f};
    int cell = 0, lz = 0;
    const int q_own = threadIdx.x / NW, j = threadIdx.x - q_own * NW;
    auto load = [&](int c0) {
      if (c0 + q_own >= ng) return;
      const int p = st.p0 + g0 + s_perm[c0 + q_own];
      v = cin[a.pts.idx[p]];
#pragma unroll
      for (int k = 0; k < 3; ++k) d[k] = a.pts.d[k][p];
      lz = a.pts.i0[2][p] - st.oz;
      cell = (a.pts.i0[1][p] - st.oy) * PX + a.pts.i0[0][p] - st.ox;
    };
    load(0);
    for (int c0 = 0, buf = 0; c0 < ng; c0 += CH, buf ^= 1) {
      unsigned char* sb = stage0 + buf * Row::stage;
      const int nq = min(CH, ng - c0);
      if (q_own < nq) {
        unsigned char* row = sb + q_own * Row::bytes;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int jt = j + h * NW;
          float kz = 0.f;
          int base = -1;
          if (jt < NS) {
            reinterpret_cast<float2*>(row)[jt] = mul2(v, dup2(kernel_tap<float, NS, HD>(d[0], jt, a.kc)));
            const float ky = kernel_tap<float, NS, HD>(d[1], jt, a.kc);
            if constexpr (Row::kPairs) {
              const int r = jt / R, y = jt - r * R;  // row instruction and lane row of tap jt
              reinterpret_cast<float*>(row + Row::ky)[((r >> 1) * R + y) * 2 + (r & 1)] = ky;
            } else {
              reinterpret_cast<float*>(row + Row::ky)[jt] = ky;
            }
            int dz = jt - lz % NS;
            dz += dz < 0 ? NS : 0;  // the plane of residue jt
            kz = kernel_tap<float, NS, HD>(d[2], dz, a.kc);
            base = (lz + dz) * PP + cell;
          }
          reinterpret_cast<float*>(row + Row::kz)[2 * j + h] = kz;
          reinterpret_cast<int*>(sb + Row::base)[2 * (j * CH + q_own) + h] = base;
        }
      }
      __syncthreads();  // (also: the tile is zeroed; the other buffer is free)
      load(c0 + CH);
      // lane q: does point q go to other cells than the point before it?
      int2 base = make_int2(-1, -1);
      if (lane < nq) base = reinterpret_cast<const int2*>(sb + Row::base)[warp * CH + lane];
      int before0 = __shfl_up_sync(0xffffffffu, base.x, 1), before1 = __shfl_up_sync(0xffffffffu, base.y, 1);
      if (lane == 0) {
        before0 = cur0;
        before1 = cur1;
      }
      const unsigned moves0 = __ballot_sync(0xffffffffu, lane < nq && base.x != before0);
      const unsigned moves1 = __ballot_sync(0xffffffffu, lane < nq && base.y != before1);
      unsigned moves = moves0 | moves1;
      for (int q = 0;;) {
        const int end = moves ? __ffs(moves) - 1 : nq;
        for (; q < end; ++q) {
          const unsigned char* row = sb + q * Row::bytes;
          const float2 ck = reinterpret_cast<const float2*>(row)[dx];
          const float2 kz = reinterpret_cast<const float2*>(row + Row::kz)[warp];
          const float2 u0 = make_float2(ck.x * kz.x, ck.y * kz.x), u1 = make_float2(ck.x * kz.y, ck.y * kz.y);
          if constexpr (Row::kPairs) {
#pragma unroll
            for (int m = 0; m < Row::NPR; ++m) {
              const float2 k = reinterpret_cast<const float2*>(row + Row::ky)[m * R + yc];
              acc0[2 * m] = fma2(u0, dup2(k.x), acc0[2 * m]);
              acc1[2 * m] = fma2(u1, dup2(k.x), acc1[2 * m]);
              if (2 * m + 1 < NR) {
                acc0[2 * m + 1] = fma2(u0, dup2(k.y), acc0[2 * m + 1]);
                acc1[2 * m + 1] = fma2(u1, dup2(k.y), acc1[2 * m + 1]);
              }
            }
          } else {
            const float2 k = dup2(reinterpret_cast<const float*>(row + Row::ky)[min(dyl, NS - 1)]);
            acc0[0] = fma2(u0, k, acc0[0]);
            acc1[0] = fma2(u1, k, acc1[0]);
          }
        }
        if (q >= nq) break;
        if (moves0 >> q & 1) {
          flush(cur0, acc0);
          cur0 = __shfl_sync(0xffffffffu, base.x, q);
        }
        if (moves1 >> q & 1) {
          flush(cur1, acc1);
          cur1 = __shfl_sync(0xffffffffu, base.y, q);
        }
        moves &= moves - 1;
      }
    }
  }
  flush(cur0, acc0);
  flush(cur1, acc1);
  __syncthreads();
  cplx_flush<float>(tile, a.fw + (size_t)blockIdx.y * a.g.Nf, st, a.g, PX);
}

}  // namespace cfg
