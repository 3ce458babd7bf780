// spread_win.cuh -- 1D spreading (type 1) with a window of sums in registers.
//
// A point has only ns taps in 1D, so a warp that shares points among its lanes
// spends its time on loads and their latency, and shared atomics of
// neighbouring points meet in the same cells.  Here a thread takes K
// consecutive sorted points and holds the ns tap sums of the current cell in
// registers: a point on the same cell costs ns FMAs per component and no store;
// moving on by s < ns cells adds the s sums left behind to the grid (one vector
// reduction each) and shifts the window.  setpts sorts 1D type-1 points fully by
// cell where cells hold points to share (bank_order), so a thread adds about
// (ns + K / density) sums for K ns taps; in any other order the result is the
// same and a jump adds the whole window.
//
// Bound: the kernel rows (FMA pipe and MUFU) and the gather of the strengths in
// the caller's order.  1e7 ordered points, 1e6 modes, ns 7: spread 87 us (shared
// atomics, lanes over taps: 598 us).
#pragma once

#include "df.cuh"
#include "kernels.h"
#include "spread_df.cuh"

namespace cfg {

// A block stages its points in shared memory with coalesced loads: read where
// they lie, a warp's threads, K points apart, touch 32 sectors per load (110 us of
// the 1e7-point spread).  Thread t's point u sits at slot 17 t + u, so the lanes
// of one read fall in distinct banks.
constexpr int kWinMax = 16;    // points per thread at most (a power of two)
constexpr int kWinPitch = kWinMax + 1;
template <typename T> constexpr int win_threads() { return sizeof(T) == 4 ? 128 : 64; }
// log2 of the points per thread: one wave of threads first (about 1024 per
// SM), then longer runs.
inline int win_log_points(long long points) {
  int lg = 0;
  while ((1 << lg) < kWinMax && (points >> lg) > 152 * 1024) ++lg;
  return lg;
}
__device__ __forceinline__ int win_slot(int i, int lg) { return (i >> lg) * kWinPitch + (i & ((1 << lg) - 1)); }

// A block whose points span at most kWinSpan cells sums them in shared memory
// first: every thread leaves its last window in its own slots, and each cell's sums
// are gathered from them (windows left behind on the way, a few a block, are added
// atomically).  Added to the grid one by one, such sums wait for one another and
// lose bits: 9e6 points in 3750 cells, error 5.7e-7 against 3.9e-7; 8 transforms
// of 2e5 points in 2000 cells 216 us.  FP64 grids sum in FP64 and need no such step
// for their error.
constexpr int kWinSpan = 96;

template <int NS>
__global__ void __launch_bounds__(win_threads<float>())
k_spread_win(SpreadArgs<float> a, int lg) {
  constexpr int HD = horner_degree<float>(NS), NT = win_threads<float>();
  __shared__ int s_cell[NT * kWinPitch];
  __shared__ float s_d[NT * kWinPitch];
  __shared__ float2 s_c[NT * kWinPitch];
  __shared__ float s_sum[2][kWinSpan];
  __shared__ int s_lo[NT / 32], s_hi[NT / 32];
  const int nf0 = a.g.nf[0];
  const long long first = (long long)blockIdx.x * (NT << lg);
  const int np = (int)min((long long)(NT << lg), a.M - first);
  const float2* cin = a.c_in + (size_t)blockIdx.y * a.M;
  float2* grid = a.fw + (size_t)blockIdx.y * a.g.Nf;
  int lo = 0x7fffffff, hi = -1;
#pragma unroll 4
  for (int i = threadIdx.x; i < np; i += NT) {
    const int p = (int)first + i, q = win_slot(i, lg);
    const int cell = a.pts.i0[0][p];
    lo = min(lo, cell);
    hi = max(hi, cell);
    s_cell[q] = cell;
    s_d[q] = a.pts.d[0][p];
    s_c[q] = cin[a.pts.idx[p]];
  }
  for (int i = threadIdx.x; i < kWinSpan; i += NT) s_sum[0][i] = s_sum[1][i] = 0.f;
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if ((threadIdx.x & 31) == 0) {
    s_lo[threadIdx.x >> 5] = lo;
    s_hi[threadIdx.x >> 5] = hi;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) {
    lo = min(lo, s_lo[w]);
    hi = max(hi, s_hi[w]);
  }
  const bool crowded = hi - lo + NS <= kWinSpan;
  const int mine = min(1 << lg, np - (int)(threadIdx.x << lg));
  if (mine > 0) {
    const int q0 = threadIdx.x * kWinPitch;
    float2 acc[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j) acc[j] = make_float2(0.f, 0.f);
    int cur = s_cell[q0];
    auto flush = [&](int j) {
      if (crowded) {
        atomicAdd(&s_sum[0][cur + j - lo], acc[j].x);
        atomicAdd(&s_sum[1][cur + j - lo], acc[j].y);
      } else {
        red_add(grid + wrap_idx(cur + j, nf0), acc[j].x, acc[j].y);
      }
    };
    for (int u = 0; u < mine; ++u) {
      const int cell = s_cell[q0 + u];
      const float2 c = s_c[q0 + u];
      float k[NS];
      kernel_row<float, NS, HD>(s_d[q0 + u], a.kc, k);
      const int s = cell - cur;
      if (s < 0 || s >= NS) {
#pragma unroll
        for (int j = 0; j < NS; ++j) {
          flush(j);
          acc[j] = make_float2(0.f, 0.f);
        }
        cur = cell;
      }
      for (; cur < cell; ++cur) {
        flush(0);
#pragma unroll
        for (int j = 0; j + 1 < NS; ++j) acc[j] = acc[j + 1];
        acc[NS - 1] = make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int j = 0; j < NS; ++j) acc[j] = fma2(c, dup2(k[j]), acc[j]);
    }
#pragma unroll
    for (int j = 0; j < NS; ++j) {
      if (crowded) s_c[q0 + j] = acc[j];  // its own points are done
      else flush(j);
    }
    s_cell[q0] = cur;
  }
  if (!crowded) return;  // block-uniform
  __syncthreads();
  // a quarter of the windows for one cell per thread
  const int windows = (np + (1 << lg) - 1) >> lg;
  for (int i = threadIdx.x; i < 4 * (hi - lo + NS); i += NT) {
    float2 sum = make_float2(0.f, 0.f);
    const int end = min(windows, (i & 3) * (NT / 4) + NT / 4);
    for (int w = (i & 3) * (NT / 4); w < end; ++w) {
      const int j = lo + (i >> 2) - s_cell[w * kWinPitch];
      if (j >= 0 && j < NS) sum = add2(sum, s_c[w * kWinPitch + j]);
    }
    atomicAdd(&s_sum[0][i >> 2], sum.x);
    atomicAdd(&s_sum[1][i >> 2], sum.y);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < hi - lo + NS; i += NT)
    red_add(grid + wrap_idx(lo + i, nf0), s_sum[0][i], s_sum[1][i]);
}

// FP64 plans in double-float (SpreadArgs::fp64_df 1): the window as float pairs,
// a thread's strengths scaled by the power of two of the largest of them.
template <int NS>
__global__ void __launch_bounds__(win_threads<double>())
k_spread_win_df(SpreadArgs<double> a, int lg) {
  constexpr int NT = win_threads<double>();
  __shared__ float2 s_tab[64];
  __shared__ int s_cell[NT * kWinPitch];
  __shared__ double s_d[NT * kWinPitch];
  __shared__ double2 s_c[NT * kWinPitch];
  if (!a.kc.horner) df_table_fill(s_tab, a.kc);
  const int nf0 = a.g.nf[0];
  const long long first = (long long)blockIdx.x * (NT << lg);
  const int np = (int)min((long long)(NT << lg), a.M - first);
  const double2* cin = a.c_in + (size_t)blockIdx.y * a.M;
  double2* grid = a.fw + (size_t)blockIdx.y * a.g.Nf;
#pragma unroll 4
  for (int i = threadIdx.x; i < np; i += NT) {
    const int p = (int)first + i, q = win_slot(i, lg);
    s_cell[q] = a.pts.i0[0][p];
    s_d[q] = a.pts.d[0][p];
    s_c[q] = cin[a.pts.idx[p]];
  }
  __syncthreads();
  const int mine = min(1 << lg, np - (int)(threadIdx.x << lg));
  if (mine <= 0) return;
  const int q0 = threadIdx.x * kWinPitch;
  unsigned m = 0;
  for (int u = 0; u < mine; ++u) {
    const double2 v = s_c[q0 + u];
    const unsigned x = (unsigned)__double2hiint(v.x) & 0x7fffffffu, y = (unsigned)__double2hiint(v.y) & 0x7fffffffu;
    if (x < 0x7ff00000u) m = max(m, x);
    if (y < 0x7ff00000u) m = max(m, y);
  }
  const int shift = 1023 - (int)(m >> 20);
  const int back = df_scale_exp(a.kc.beta) - shift;
  float2 s[NS], e[NS];
#pragma unroll
  for (int j = 0; j < NS; ++j) s[j] = e[j] = make_float2(0.f, 0.f);
  int cur = s_cell[q0];
  auto flush = [&](int j) {
    red_add(grid + wrap_idx(cur + j, nf0), df_widen(s[j].x, back) + df_widen(e[j].x, back),
            df_widen(s[j].y, back) + df_widen(e[j].y, back));
  };
  for (int u = 0; u < mine; ++u) {
    const int cell = s_cell[q0 + u];
    const double2 v = s_c[q0 + u];
    float kh[NS], kl[NS];
    df_kernel_row<NS>(s_d[q0 + u], a.kc, s_tab, kh, kl);
    const int step = cell - cur;
    if (step < 0 || step >= NS) {
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        flush(j);
        s[j] = e[j] = make_float2(0.f, 0.f);
      }
      cur = cell;
    }
    for (; cur < cell; ++cur) {
      flush(0);
#pragma unroll
      for (int j = 0; j + 1 < NS; ++j) {
        s[j] = s[j + 1];
        e[j] = e[j + 1];
      }
      s[NS - 1] = e[NS - 1] = make_float2(0.f, 0.f);
    }
    const DF re = df_split(v.x, shift), im = df_split(v.y, shift);
    const float2 ch = make_float2(re.h, im.h), cl = make_float2(re.l, im.l);
#pragma unroll
    for (int j = 0; j < NS; ++j) df2_acc(s[j], e[j], ch, cl, dup2(kh[j]), dup2(kl[j]));
  }
#pragma unroll
  for (int j = 0; j < NS; ++j) flush(j);
}

template <typename T, int NS>
cudaError_t launch_spread_win(const SpreadArgs<T>& a, cudaStream_t s) {
  const int lg = win_log_points((long long)a.M * a.ntr);
  const long long per = (long long)win_threads<T>() << lg;
  const dim3 grid((unsigned)((a.M + per - 1) / per), a.ntr);
  if constexpr (sizeof(T) == 4) k_spread_win<NS><<<grid, win_threads<T>(), 0, s>>>(a, lg);
  else k_spread_win_df<NS><<<grid, win_threads<T>(), 0, s>>>(a, lg);
  return cudaGetLastError();
}

}  // namespace cfg
