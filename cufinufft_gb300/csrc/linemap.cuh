// linemap.cuh -- where a line FFT's positions lie in memory (LineSide), shared
// by the line-pass kernels (fftpass.cu, fft_df.cu).
#pragma once

#include "kernels.h"

namespace cfg {

// FFT index w -> mode index i in [0, Np), or -1 for a padding position.
__device__ __forceinline__ int mode_index(int w, int L, int Np) {
  if (w <= (Np - 1) / 2) return w + Np / 2;
  if (w >= L - Np / 2) return w - L + Np / 2;
  return -1;
}
// mode index i -> FFT index
__device__ __forceinline__ int mode_pos(int i, int L, int Np) {
  const int k = i - Np / 2;
  return k >= 0 ? k : L + k;
}

__device__ __forceinline__ long long side_line(const LineSide& s, int la, int lb) {
  const long long ma = s.acorner ? mode_pos(la, s.nfa, s.Na) : la;
  const long long mb = s.bcorner ? mode_pos(lb, s.nfb, s.Nb) : lb;
  return ma * s.sa + mb * s.sb;
}

template <typename T>
__device__ __forceinline__ T line_factor(const LineArgs<T>& a, int la, int lb, int i) {
  T f = T(1);
  if (a.fa) f *= a.fa[la];
  if (a.fb) f *= a.fb[lb];
  if (a.fp && i >= 0) f *= a.fp[i];
  return f;
}

}  // namespace cfg
