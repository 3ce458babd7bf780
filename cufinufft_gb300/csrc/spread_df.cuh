// spread_df.cuh -- subproblem spreading of FP64 plans in double-float
// arithmetic (SpreadArgs::fp64_df): the slab-owned 3D and private-tile 2D
// kernels of spreadinterp.cuh with tile cells, kernel values and sums as FP32
// pairs, (re hi, im hi, re lo, im lo) in the 16 bytes of an FP64 cell.
//
// Why: an FP64 complex tap is two FMAs, one clock of an SM's FP64 unit; the
// same tap as fifteen packed FP32 instructions (df2_acc_long) is a quarter of that,
// and the kernel rows (FP64 exp and sqrt per value before) become small
// beside the taps.  What bounds it then is the FMA pipe and the 32 bytes of
// shared memory a tap reads and writes, about equally.
//
// Range: a block scales its points' strengths by the power of two that brings
// the largest to [1, 2) and its kernel values by 2^-E per axis (df.cuh); the
// flush undoes both, exactly.
#pragma once

#include "df.cuh"
#include "kernels.h"

namespace cfg {

// The shift that brings the largest finite strength of the block's points to
// [1, 2): high words compare as integers.  smax is zeroed and the block
// synchronised before the call.
__device__ __forceinline__ int strength_shift(const double2* cin, const int* idx, int np, unsigned* smax) {
  unsigned m = 0;
  for (int q = threadIdx.x; q < np; q += blockDim.x) {
    const uint4 v = *reinterpret_cast<const uint4*>(cin + idx[q]);
    const unsigned x = v.y & 0x7fffffffu, y = v.w & 0x7fffffffu;
    if (x < 0x7ff00000u) m = max(m, x);
    if (y < 0x7ff00000u) m = max(m, y);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(smax, m);
  __syncthreads();
  return 1023 - (int)(*smax >> 20);
}

// Flush of a pair tile with row pitch `pitch`; k: the exponent to restore.
__device__ __forceinline__ void df_flush(const float4* tile, double2* grid, const SubTile& st, const GridGeom& g,
                                         int pitch, int k) {
  const int lane = threadIdx.x & 31, nwb = blockDim.x >> 5;
  const int rows = st.TY * st.TZ;
  TileRows rw(threadIdx.x >> 5, st.TY);
  const bool inside = tile_in_grid(st, g);
  for (int r = threadIdx.x >> 5; r < rows; r += nwb, rw.next(nwb, st.TY)) {
    const int gy = inside ? st.oy + rw.iy : wrap3(st.oy + rw.iy, g.nf[1]);
    const int gz = inside ? st.oz + rw.iz : wrap3(st.oz + rw.iz, g.nf[2]);
    double2* dst = grid + ((size_t)gz * g.nf[1] + gy) * g.nf[0];
    const float4* src = tile + (size_t)r * pitch;
    for (int ix = lane; ix < st.TX; ix += 32) {
      const float4 v = src[ix];
      if (v.x == 0.f && v.y == 0.f && v.z == 0.f && v.w == 0.f) continue;
      red_add(dst + (inside ? st.ox + ix : wrap3(st.ox + ix, g.nf[0])), df_widen(v.x, k) + df_widen(v.z, k),
              df_widen(v.y, k) + df_widen(v.w, k));
    }
  }
}

// 3D: planes owned by warps, as k_spread_sm_slab, but with two warps to a
// plane, one for the even tile rows and one for the odd ones: the FP64 tile
// (110 KB at ns 10 with 16x16x2 bins) leaves one block per SM, and with one
// warp per plane the SM had 2.5 warps per scheduler, waiting on their own
// dependent sums (ncu: 37% of cycles issued, FMA pipe 33%, shared memory 40%).
// A chunk of 32 points is staged by one warp per (tap pair, axis), lanes over
// points: with one thread per (point, axis) row three warps worked while the
// others waited at the barrier about as long as the chunk's taps take.  Staged
// values are [tap][point], pitch 33 (conflict-free stores; the lanes of a row
// read distinct banks).  81x96x75 modes, 2e6 points, tol 1e-9: 15.6 ms (FP64)
// -> 6.8 ms (one warp per plane, one thread per row) -> 5.9 ms; now shared
// memory is 69% busy and the FMA pipe 50%.
constexpr int kSlabDfChunk = 32;
constexpr int kSlabDfPitch = kSlabDfChunk + 1;
// tile row pitch: the rows of one instruction are two tile rows apart, so
// 2 pitch = NS (mod 8 cells of 16 bytes) puts its lanes in distinct banks
// (odd widths: NS + 1, one conflict)
__host__ __device__ constexpr int slab_df_pitch(int tx, int ns) {
  return tx + ((((ns + 1) / 2 - tx) % 4) + 4) % 4;
}
__host__ __device__ constexpr int slab_df_instrs(int ns) { return ((ns + 1) / 2 + 32 / ns - 1) / (32 / ns); }
// bytes of one stage buffer: c kx, ky, kz [NS] x pitch, tile offsets
__host__ __device__ constexpr size_t slab_df_stage(int ns) {
  return (size_t)kSlabDfPitch * 3 * ns * sizeof(float4) + kSlabDfChunk * sizeof(int2);
}
// The widest tiles give up the row padding (ns 13 with 16x16x2 bins), then the
// second stage buffer (ns 14), before the kernel is given up.
struct SlabDfShape {
  int pitch, nbuf;
  size_t bytes;
};
inline SlabDfShape slab_df_shape(int ns, const BinTables& bt, size_t limit) {
  const int tx = bt.bs[0] + ns - 1;
  const size_t rows = (size_t)(bt.bs[1] + ns - 1) * (bt.bs[2] + ns - 1) * sizeof(float4), st = slab_df_stage(ns);
  const int pad = slab_df_pitch(tx, ns);
  const SlabDfShape v[3] = {{pad, 2, pad * rows + 2 * st}, {tx, 2, tx * rows + 2 * st}, {tx, 1, tx * rows + st}};
  for (const SlabDfShape& x : v)
    if (x.bytes <= limit) return x;
  return SlabDfShape{0, 0, 0};
}

template <int NS>
__global__ void __launch_bounds__(64 * NS)
k_spread_sm_slab_df(SpreadArgs<double> a, int PX, int nbuf) {
  constexpr int R = 32 / NS;                        // tile rows per warp instruction
  constexpr int NR = slab_df_instrs(NS);            // instructions per half plane
  constexpr int NP = (NS + 1) / 2;                  // tap pairs
  constexpr int CH = kSlabDfChunk, CP = kSlabDfPitch;
  constexpr bool kFullRows = 32 % NS == 0 && NS % 2 == 0 && (NS / 2) % R == 0;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float2 s_tab[64];
  __shared__ unsigned s_max;
  if (threadIdx.x == 0) s_max = 0;
  if (!a.kc.horner) df_table_fill(s_tab, a.kc);
  const SubTile st = sub_tile_block<3, NS>(a.bins, blockIdx.x);  // synchronises
  if (st.np <= 0) return;  // block-uniform
  const int PP = PX * st.TY;  // plane stride
  const int ncell = PP * st.TZ;
  float4* tile = reinterpret_cast<float4*>(smem_raw);
  unsigned char* stage0 = smem_raw + (size_t)ncell * sizeof(float4);
  const int t = blockIdx.y;
  for (int i = threadIdx.x; i < ncell; i += blockDim.x) tile[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  const double2* cin = a.c_in + (size_t)t * a.M;
  const int shift = strength_shift(cin, a.pts.idx + st.p0, st.np, &s_max);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int residue = warp % NS, half = warp / NS;
  const int dx = lane % NS, dyl = min(lane / NS, R - 1);
  const bool lane_on = lane < R * NS;
  for (int c0 = 0, buf = 0; c0 < st.np; c0 += CH, buf ^= 1) {
    if (nbuf == 1) {
      if (c0) __syncthreads();  // the previous chunk's reads of the one buffer
      buf = 0;
    }
    unsigned char* sb = stage0 + buf * slab_df_stage(NS);
    // kernel values duplicated, (h, h, l, l): the packed operands of both
    // components come with one load
    float4* s_ck = reinterpret_cast<float4*>(sb);  // [NS][CP] c kx
    float4* s_ky = s_ck + NS * CP;                 // [NS][CP]
    float4* s_kz = s_ky + NS * CP;                 // [NS][CP]
    int2* s_bl = reinterpret_cast<int2*>(s_kz + NS * CP);      // tile offset, lz mod NS and ly's parity
    const int nq = min(CH, st.np - c0);
    for (int w = warp; w < 3 * NP; w += 2 * NS) {  // warp-uniform (axis, tap pair)
      const int ax = w % 3, tp = w / 3;
      if (lane < nq) {
        const int p = st.p0 + c0 + lane;
        const DF2 k = df_kernel_pair<NS>(a.pts.d[ax][p], tp, a.kc, s_tab);
        if (ax == 0) {
          const double2 v = cin[a.pts.idx[p]];
          const DF re = df_split(v.x, shift), im = df_split(v.y, shift);
          const DF2 c = DF2{make_float2(re.h, im.h), make_float2(re.l, im.l)};
          const DF2 u = df2_mul(c, DF2{dup2(k.h.x), dup2(k.l.x)});
          s_ck[tp * CP + lane] = make_float4(u.h.x, u.h.y, u.l.x, u.l.y);
          if (tp != NS - 1 - tp) {
            const DF2 v2 = df2_mul(c, DF2{dup2(k.h.y), dup2(k.l.y)});
            s_ck[(NS - 1 - tp) * CP + lane] = make_float4(v2.h.x, v2.h.y, v2.l.x, v2.l.y);
          }
          if (tp == 0) {
            const int lx = a.pts.i0[0][p] - st.ox, ly = a.pts.i0[1][p] - st.oy, lz = a.pts.i0[2][p] - st.oz;
            s_bl[lane] = make_int2((lz * st.TY + ly) * PX + lx, 2 * (lz % NS) + (ly & 1));
          }
        } else {
          float4* dst = ax == 1 ? s_ky : s_kz;
          dst[tp * CP + lane] = make_float4(k.h.x, k.h.x, k.l.x, k.l.x);
          dst[(NS - 1 - tp) * CP + lane] = tp == NS - 1 - tp ? make_float4(k.h.x, k.h.x, k.l.x, k.l.x)
                                                              : make_float4(k.h.y, k.h.y, k.l.y, k.l.y);
        }
      }
    }
    __syncthreads();  // (also: the tile is zeroed; the other buffer is free)
    for (int q = 0; q < nq; ++q) {
      const int2 bl = s_bl[q];
      int dz = residue - (bl.y >> 1);
      dz += dz < 0 ? NS : 0;                     // the plane of this warp's residue
      const int dy0 = (half ^ bl.y) & 1;         // its rows: ly + dy = half (mod 2)
      const float4 kz = s_kz[dz * CP + q];
      const float4 ck = s_ck[dx * CP + q];
      const DF2 u = df2_mul(DF2{make_float2(ck.x, ck.y), make_float2(ck.z, ck.w)},
                            DF2{make_float2(kz.x, kz.y), make_float2(kz.z, kz.w)});
      const float2 nuh = neg2(u.h);
      float4* cell = tile + bl.x + dz * PP + dx;
      // lanes without a tap read one of the point's rows all the same and only
      // leave out the store (no divergent branch); just the last instruction
      // can run past the support
      const int d0 = 2 * dyl + dy0, dlast = min(d0 + 2 * (NR - 1) * R, NS - 1);
      float4 v[NR], ky[NR];
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int dy = r == NR - 1 ? dlast : d0 + 2 * r * R;
        ky[r] = s_ky[dy * CP + q];
        v[r] = cell[dy * PX];
      }
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        float2 s = make_float2(v[r].x, v[r].y), e = make_float2(v[r].z, v[r].w);
        df2_acc_long(s, e, u.h, nuh, u.l, make_float2(ky[r].x, ky[r].y), make_float2(ky[r].z, ky[r].w));
        if (kFullRows || (lane_on && (r < NR - 1 || d0 + 2 * r * R < NS)))
          cell[(r == NR - 1 ? dlast : d0 + 2 * r * R) * PX] = make_float4(s.x, s.y, e.x, e.y);
      }
      __syncwarp();  // this point's stores before the next point's loads
    }
  }
  __syncthreads();
  df_flush(tile, a.fw + (size_t)t * a.g.Nf, st, a.g, PX, 3 * df_scale_exp(a.kc.beta) - shift);
}

// 2D: private tile copies, as k_spread_sm_priv.
constexpr int kPrivDfWarps = 4;
__host__ __device__ constexpr size_t priv_df_stage(int ns) {
  return (32 * ((size_t)ns * (sizeof(float4) + sizeof(float2)) + sizeof(int)) + 15) & ~(size_t)15;
}
inline size_t priv_df_bytes(int ns, const BinTables& bt) {
  const size_t px = slab_pitch(bt.bs[0] + ns - 1, ns);
  return kPrivDfWarps * (px * (bt.bs[1] + ns - 1) * sizeof(float4) + priv_df_stage(ns));
}

template <int NS>
__global__ void __launch_bounds__(32 * kPrivDfWarps)
k_spread_sm_priv_df(SpreadArgs<double> a) {
  constexpr int R = 32 / NS;
  constexpr int NR = (NS + R - 1) / R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float2 s_tab[64];
  __shared__ unsigned s_max;
  if (threadIdx.x == 0) s_max = 0;
  if (!a.kc.horner) df_table_fill(s_tab, a.kc);
  const SubTile st = sub_tile_block<2, NS>(a.bins, blockIdx.x);
  if (st.np <= 0) return;  // block-uniform
  const int PX = slab_pitch(st.TX, NS);
  const int ncell = PX * st.TY;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float4* tile0 = reinterpret_cast<float4*>(smem_raw);
  float4* tile = tile0 + (size_t)warp * ncell;
  unsigned char* sb = smem_raw + (size_t)kPrivDfWarps * ncell * sizeof(float4) + warp * priv_df_stage(NS);
  float4* s_ck = reinterpret_cast<float4*>(sb);              // [32][NS]
  float2* s_ky = reinterpret_cast<float2*>(s_ck + 32 * NS);  // [32][NS]
  int* s_base = reinterpret_cast<int*>(s_ky + 32 * NS);
  for (int i = lane; i < ncell; i += 32) tile[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  const int t = blockIdx.y;
  const double2* cin = a.c_in + (size_t)t * a.M;
  const int shift = strength_shift(cin, a.pts.idx + st.p0, st.np, &s_max);
  const int dx = lane % NS, dyl = lane / NS;
  const bool lane_on = lane < R * NS;
  constexpr bool kFullRows = 32 % NS == 0 && (NS * NS) % 32 == 0;
  // warp w takes points [w S, (w + 1) S) of the subproblem
  const int S = (st.np + kPrivDfWarps - 1) / kPrivDfWarps;
  const int beg = warp * S, end = min(st.np, beg + S);
  for (int c0 = beg; c0 < end; c0 += 32) {
    const int nq = min(32, end - c0);
    __syncwarp();  // the previous chunk's reads of the stage are done
    if (lane < nq) {
      const int p = st.p0 + c0 + lane;
      float kh[NS], kl[NS];
#pragma unroll 1
      for (int ax = 1; ax >= 0; --ax) {
        df_kernel_row<NS>(a.pts.d[ax][p], a.kc, s_tab, kh, kl);
        if (ax == 1) {
#pragma unroll
          for (int j = 0; j < NS; ++j) s_ky[lane * NS + j] = make_float2(kh[j], kl[j]);
        }
      }
      const double2 v = cin[a.pts.idx[p]];
      const DF re = df_split(v.x, shift), im = df_split(v.y, shift);
      const DF2 c = DF2{make_float2(re.h, im.h), make_float2(re.l, im.l)};
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        const DF2 w = df2_mul(c, DF2{dup2(kh[j]), dup2(kl[j])});
        s_ck[lane * NS + j] = make_float4(w.h.x, w.h.y, w.l.x, w.l.y);
      }
      s_base[lane] = (a.pts.i0[1][p] - st.oy) * PX + (a.pts.i0[0][p] - st.ox);
    }
    __syncwarp();
    for (int q = 0; q < nq; ++q) {
      const float4 ck = s_ck[q * NS + dx];
      const float2 uh = make_float2(ck.x, ck.y), ul = make_float2(ck.z, ck.w), nuh = neg2(uh);
      float4* cell = tile + s_base[q] + dx;
      // lanes without a tap take the point's last row and leave out the store
      float4 w[NR];
      float2 ky[NR];
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int dy = min(r * R + dyl, NS - 1);
        ky[r] = s_ky[q * NS + dy];
        w[r] = cell[dy * PX];
      }
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int dy = r * R + dyl;
        float2 s = make_float2(w[r].x, w[r].y), e = make_float2(w[r].z, w[r].w);
        df2_acc_long(s, e, uh, nuh, ul, dup2(ky[r].x), dup2(ky[r].y));
        if (kFullRows || (lane_on && dy < NS)) cell[dy * PX] = make_float4(s.x, s.y, e.x, e.y);
      }
      __syncwarp();  // this point's stores before the next point's loads
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ncell; i += blockDim.x) {
    float4 v = tile0[i];
    DF2 sum = DF2{make_float2(v.x, v.y), make_float2(v.z, v.w)};
#pragma unroll
    for (int w = 1; w < kPrivDfWarps; ++w) {
      v = tile0[(size_t)w * ncell + i];
      sum = df2_add(sum, DF2{make_float2(v.x, v.y), make_float2(v.z, v.w)});
    }
    tile0[i] = make_float4(sum.h.x, sum.h.y, sum.l.x, sum.l.y);
  }
  __syncthreads();
  df_flush(tile0, a.fw + (size_t)t * a.g.Nf, st, a.g, PX, 2 * df_scale_exp(a.kc.beta) - shift);
}

}  // namespace cfg
