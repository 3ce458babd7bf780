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
// the caller's order.  1e7 ordered points, 1e6 modes, ns 7: spread ~50 us (shared
// atomics, lanes over taps: 598 us).
#pragma once

#include "df.cuh"
#include "kernels.h"
#include "spread_df.cuh"

namespace cfg {

constexpr int kWinThreads = 128;
constexpr int kWinBatch = 4;   // points whose loads are in flight together
constexpr int kWinMax = 16;    // points per thread at most
// One wave of threads first (about 1024 per SM), then longer runs.
inline int win_points(int M) {
  const long long k = ((long long)M + 152 * 1024 - 1) / (152 * 1024);
  return k < 1 ? 1 : (k > kWinMax ? kWinMax : (int)k);
}

template <int NS>
__global__ void __launch_bounds__(kWinThreads)
k_spread_win(SpreadArgs<float> a, int K) {
  constexpr int HD = horner_degree<float>(NS);
  const int nf0 = a.g.nf[0];
  const long long first = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * K;
  if (first >= a.M) return;
  const int beg = (int)first, end = min(a.M, beg + K);
  const float2* cin = a.c_in + (size_t)blockIdx.y * a.M;
  float2* grid = a.fw + (size_t)blockIdx.y * a.g.Nf;
  float2 acc[NS];
#pragma unroll
  for (int j = 0; j < NS; ++j) acc[j] = make_float2(0.f, 0.f);
  int cur = a.pts.i0[0][beg];
  auto flush = [&](int j) { red_add(grid + wrap_idx(cur + j, nf0), acc[j].x, acc[j].y); };
  for (int p0 = beg; p0 < end; p0 += kWinBatch) {
    int cell[kWinBatch];
    float d[kWinBatch];
    float2 c[kWinBatch];
#pragma unroll
    for (int u = 0; u < kWinBatch; ++u) {
      const int p = min(p0 + u, end - 1);
      cell[u] = a.pts.i0[0][p];
      d[u] = a.pts.d[0][p];
      c[u] = cin[a.pts.idx[p]];
    }
#pragma unroll
    for (int u = 0; u < kWinBatch; ++u) {
      if (p0 + u >= end) break;
      float k[NS];
      kernel_row<float, NS, HD>(d[u], a.kc, k);
      const int s = cell[u] - cur;
      if (s < 0 || s >= NS) {
#pragma unroll
        for (int j = 0; j < NS; ++j) {
          flush(j);
          acc[j] = make_float2(0.f, 0.f);
        }
        cur = cell[u];
      }
      for (; cur < cell[u]; ++cur) {
        flush(0);
#pragma unroll
        for (int j = 0; j + 1 < NS; ++j) acc[j] = acc[j + 1];
        acc[NS - 1] = make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int j = 0; j < NS; ++j) acc[j] = fma2(c[u], dup2(k[j]), acc[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < NS; ++j) flush(j);
}

// FP64 plans in double-float (SpreadArgs::fp64_df 1): the window as float pairs,
// a thread's strengths scaled by the power of two of the largest of them.
template <int NS>
__global__ void __launch_bounds__(kWinThreads)
k_spread_win_df(SpreadArgs<double> a, int K) {
  __shared__ float2 s_tab[64];
  if (!a.kc.horner) {
    df_table_fill(s_tab, a.kc);
    __syncthreads();
  }
  const int nf0 = a.g.nf[0];
  const long long first = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * K;
  if (first >= a.M) return;
  const int beg = (int)first, end = min(a.M, beg + K);
  const double2* cin = a.c_in + (size_t)blockIdx.y * a.M;
  double2* grid = a.fw + (size_t)blockIdx.y * a.g.Nf;
  unsigned m = 0;
#pragma unroll 4
  for (int p = beg; p < end; ++p) {
    const double2 v = cin[a.pts.idx[p]];
    const unsigned x = (unsigned)__double2hiint(v.x) & 0x7fffffffu, y = (unsigned)__double2hiint(v.y) & 0x7fffffffu;
    if (x < 0x7ff00000u) m = max(m, x);
    if (y < 0x7ff00000u) m = max(m, y);
  }
  const int shift = 1023 - (int)(m >> 20);
  const int back = df_scale_exp(a.kc.beta) - shift;
  float2 s[NS], e[NS];
#pragma unroll
  for (int j = 0; j < NS; ++j) s[j] = e[j] = make_float2(0.f, 0.f);
  int cur = a.pts.i0[0][beg];
  auto flush = [&](int j) {
    red_add(grid + wrap_idx(cur + j, nf0), df_widen(s[j].x, back) + df_widen(e[j].x, back),
            df_widen(s[j].y, back) + df_widen(e[j].y, back));
  };
  for (int p = beg; p < end; ++p) {
    const int cell = a.pts.i0[0][p];
    const double2 v = cin[a.pts.idx[p]];
    float kh[NS], kl[NS];
    df_kernel_row<NS>(a.pts.d[0][p], a.kc, s_tab, kh, kl);
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
  const int K = win_points(a.M);
  const long long threads = ((long long)a.M + K - 1) / K;
  const dim3 grid((unsigned)((threads + kWinThreads - 1) / kWinThreads), a.ntr);
  if constexpr (sizeof(T) == 4) k_spread_win<NS><<<grid, kWinThreads, 0, s>>>(a, K);
  else k_spread_win_df<NS><<<grid, kWinThreads, 0, s>>>(a, K);
  return cudaGetLastError();
}

}  // namespace cfg
