// fft_df.cu -- line FFTs of FP64 grids in double-float arithmetic (FP32 pairs).
//
// cuFFT's Z2Z transform is bound by GB300's FP64 unit: a radix-8 butterfly is
// ~10 FP64 instructions per value at a sixty-fourth of the FP32 rate, against
// ~50 packed FP32 instructions here.  A d-dimensional transform is one pass
// per axis over only the lines and positions that carry modes (LineArgs,
// linemap.cuh), with the amplification fused into the first pass of type 2 and
// the deconvolution into the last of type 1: the zero padding is neither
// written, read nor transformed.
//
// A block transforms G lines: every thread holds eight to ten values in
// registers, Stockham passes of radix 8, 4, 2, 5, 3 exchange them through one
// padded shared buffer (read all, wait, write all), the first pass loads from
// global memory and the last stores to it.  Values travel as (re hi, im hi, re
// lo, im lo); the block scales its lines by the power of two that brings the
// largest input to [1, 2), so any FP64 range passes.  Along y and z a block's G
// lines are adjacent, so a row segment of G cells is contiguous.
//
// A 1D transform beyond 4096 points is two such passes, L = L1 L2: columns n2
// of x[n1 L2 + n2], multiplied by W_L^(n2 k1), then rows k1, whose output k2
// lands at k1 + L1 k2.
//
// Measured (FFT with amplification or deconvolution; cuFFT with the mode-row
// kernel before): @@
#include <cuda_runtime.h>

#include "df.cuh"
#include "linemap.cuh"

namespace cfg {
namespace {

constexpr int kDfThreadsMax = 512;
constexpr int kDfValues = 8;  // values per thread (radix 5: 10, radix 3: 9)

using Z = DF2;  // a complex value: h = (re, im), l its low parts

__device__ __forceinline__ Z znorm(Z a) { return fast_two_sum2(a.h, a.l); }
// Sums and products keep their low parts unnormalised (a few ulps) through a
// pass, whose end normalises once.
__device__ __forceinline__ Z zadd(Z a, Z b) { return df2_add(a, b); }
__device__ __forceinline__ Z zsub(Z a, Z b) {
  const float2 s = sub2(a.h, b.h);
  const float2 bb = sub2(s, a.h);
  const float2 e = sub2(sub2(a.h, sub2(s, bb)), add2(b.h, bb));
  return Z{s, add2(e, sub2(a.l, b.l))};
}
// a times the real constant c (as a pair)
#define CFG_DF_CONST(NAME, VALUE)               \
  constexpr float NAME##_h = (float)(VALUE);    \
  constexpr float NAME##_l = (float)((VALUE) - (double)NAME##_h)
__device__ __forceinline__ Z zscale(Z a, float ch, float cl) { return df2_mul(a, Z{dup2(ch), dup2(cl)}); }
// a (dir i)
__device__ __forceinline__ Z zmul_i(Z a, float dir) {
  return Z{make_float2(-dir * a.h.y, dir * a.h.x), make_float2(-dir * a.l.y, dir * a.l.x)};
}
// a w, w = (re hi, im hi, re lo, im lo)
__device__ __forceinline__ Z zmul(Z a, float4 w) {
  const Z p = df2_mul(a, Z{dup2(w.x), dup2(w.z)});
  const Z as = Z{make_float2(a.h.y, a.h.x), make_float2(a.l.y, a.l.x)};
  const Z q = df2_mul(as, Z{make_float2(-w.y, w.y), make_float2(-w.w, w.w)});
  return zadd(p, q);
}

template <int R> struct DftDf;
template <> struct DftDf<2> {
  static __device__ __forceinline__ void run(Z* v, float) {
    const Z a = v[0], b = v[1];
    v[0] = zadd(a, b);
    v[1] = zsub(a, b);
  }
};
template <> struct DftDf<4> {
  static __device__ __forceinline__ void run(Z* v, float dir) {
    const Z s02 = zadd(v[0], v[2]), d02 = zsub(v[0], v[2]);
    const Z s13 = zadd(v[1], v[3]), d13 = zmul_i(zsub(v[1], v[3]), dir);
    v[0] = zadd(s02, s13);
    v[2] = zsub(s02, s13);
    v[1] = zadd(d02, d13);
    v[3] = zsub(d02, d13);
  }
};
template <> struct DftDf<8> {
  static __device__ __forceinline__ void run(Z* v, float dir) {
    CFG_DF_CONST(kH, 0.70710678118654752440);  // 1/sqrt(2)
    Z e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    DftDf<4>::run(e, dir);
    DftDf<4>::run(o, dir);
    // o_m *= exp(dir 2 pi i m / 8): (1 + dir i)/sqrt(2), dir i, (-1 + dir i)/sqrt(2)
    const Z w1 = zscale(zadd(o[1], zmul_i(o[1], dir)), kH_h, kH_l);
    const Z w2 = zmul_i(o[2], dir);
    const Z w3 = zscale(zsub(zmul_i(o[3], dir), o[3]), kH_h, kH_l);
    v[0] = zadd(e[0], o[0]);
    v[4] = zsub(e[0], o[0]);
    v[1] = zadd(e[1], w1);
    v[5] = zsub(e[1], w1);
    v[2] = zadd(e[2], w2);
    v[6] = zsub(e[2], w2);
    v[3] = zadd(e[3], w3);
    v[7] = zsub(e[3], w3);
  }
};
template <> struct DftDf<3> {
  static __device__ __forceinline__ void run(Z* v, float dir) {
    CFG_DF_CONST(kS, 0.86602540378443864676);  // sin(2 pi / 3)
    const Z t = zadd(v[1], v[2]);
    const Z u = zmul_i(zscale(zsub(v[1], v[2]), kS_h, kS_l), dir);
    const Z m = zsub(v[0], Z{mul2(t.h, dup2(0.5f)), mul2(t.l, dup2(0.5f))});
    v[0] = zadd(v[0], t);
    v[1] = zadd(m, u);
    v[2] = zsub(m, u);
  }
};
template <> struct DftDf<5> {
  static __device__ __forceinline__ void run(Z* v, float dir) {
    CFG_DF_CONST(kC1, 0.30901699437494742410);   // cos(2 pi / 5)
    CFG_DF_CONST(kC2, -0.80901699437494742410);  // cos(4 pi / 5)
    CFG_DF_CONST(kS1, 0.95105651629515357212);   // sin(2 pi / 5)
    CFG_DF_CONST(kS2, 0.58778525229247312917);   // sin(4 pi / 5)
    const Z p14 = zadd(v[1], v[4]), m14 = zsub(v[1], v[4]);
    const Z p23 = zadd(v[2], v[3]), m23 = zsub(v[2], v[3]);
    const Z r1 = zadd(v[0], zadd(zscale(p14, kC1_h, kC1_l), zscale(p23, kC2_h, kC2_l)));
    const Z r2 = zadd(v[0], zadd(zscale(p14, kC2_h, kC2_l), zscale(p23, kC1_h, kC1_l)));
    const Z q1 = zmul_i(zadd(zscale(m14, kS1_h, kS1_l), zscale(m23, kS2_h, kS2_l)), dir);
    const Z q2 = zmul_i(zsub(zscale(m14, kS2_h, kS2_l), zscale(m23, kS1_h, kS1_l)), dir);
    v[0] = zadd(v[0], zadd(p14, p23));
    v[1] = zadd(r1, q1);
    v[4] = zsub(r1, q1);
    v[2] = zadd(r2, q2);
    v[3] = zsub(r2, q2);
  }
};

// Shared slot of element i of a line: one spare 16-byte slot every eight (128
// bytes) spreads the strided Stockham writes over the banks.
__device__ __forceinline__ int df_slot(int i) { return i + (i >> 3); }

struct DfCtx {
  const LineDfArgs* d;
  const double2* in;
  double2* out;
  float4* buf;
  int line0, Lp, shift;
  unsigned* smax;
};

// A line on one side: where position w of it lies, and the factor of its modes.
struct DfLine {
  long long base, step;  // index of position 0 (pmode 1: of mode 0), and per position
  double f;
};
// fold 1 and 2: positions lie `line` apart from a multiple of the line count.
__device__ __forceinline__ DfLine df_line(const LineDfArgs& d, const LineSide& s, int line, bool folded, bool factor) {
  const LineArgs<double>& a = d.a;
  DfLine l;
  l.f = 1.0;
  if (folded) {
    l.base = line;
    l.step = a.nlines;
    return l;
  }
  const int lb = a.A == a.nlines ? 0 : line / a.A, la = line - lb * a.A;
  l.base = side_line(s, la, lb);
  l.step = s.sp;
  if (factor) l.f = line_factor(a, la, lb, -1);
  return l;
}
// Index of position w (-1: padding); *mode its mode index (or w).
__device__ __forceinline__ long long df_index(const LineDfArgs& d, const LineSide& s, const DfLine& l, int w,
                                              bool folded, int* mode) {
  *mode = w;
  if (folded) {
    const long long pos = l.base + (long long)w * l.step;
    if (s.pmode == 0) return pos;
    return *mode = mode_index((int)pos, d.Lfull, s.Np);
  }
  if (s.pmode) {
    *mode = mode_index(w, d.a.L, s.Np);
    if (*mode < 0) return -1;
  }
  return l.base + (long long)(s.pmode == 1 ? *mode : w) * l.step;
}

template <int R>
__device__ __forceinline__ void df_pass(DfCtx& c, int Ns, bool first, bool last) {
  constexpr int NB = (kDfValues + R - 1) / R;  // butterflies per thread
  const LineDfArgs& d = *c.d;
  const LineArgs<double>& a = d.a;
  const int L = a.L, G = a.G, nbf = L / R, total = G * nbf;
  const float inv_nbf = 1.f / (float)nbf, inv_Ns = 1.f / (float)Ns;
  const float dir = (float)a.dir;
  // lanes along adjacent lines where those are contiguous in memory
  const bool across = (first && d.in_across) || (last && d.out_across);
  Z v[NB][R];
  int gs[NB], js[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int u = threadIdx.x + b * blockDim.x;
    if (across) {
      gs[b] = u & (G - 1);
      js[b] = u >> a.log2G;
    } else {
      gs[b] = (int)(((float)u + 0.5f) * inv_nbf);
      js[b] = u - gs[b] * nbf;
    }
    if (u >= total) gs[b] = -1;
  }
  if (first) {
    double2 raw[NB][R];
    unsigned m = 0;
    const bool folded = d.fold == 1, per_mode = !a.fac_on_out && a.fp != nullptr && a.si.pmode;
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int line = c.line0 + gs[b];
      const bool on = gs[b] >= 0 && line < a.nlines;
      DfLine l;
      if (on) l = df_line(d, a.si, line, folded, !a.fac_on_out);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        raw[b][r] = make_double2(0.0, 0.0);
        if (!on) continue;
        int mode;
        const long long at = df_index(d, a.si, l, js[b] + r * nbf, folded, &mode);
        if (at < 0) continue;
        raw[b][r] = c.in[at];
        if (per_mode) {
          const double f = l.f * a.fp[mode];
          raw[b][r].x *= f;
          raw[b][r].y *= f;
        }
        const unsigned x = (unsigned)__double2hiint(raw[b][r].x) & 0x7fffffffu;
        const unsigned y = (unsigned)__double2hiint(raw[b][r].y) & 0x7fffffffu;
        if (x < 0x7ff00000u) m = max(m, x);
        if (y < 0x7ff00000u) m = max(m, y);
      }
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(c.smax, m);
    __syncthreads();
    c.shift = 1023 - (int)(*c.smax >> 20);
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const DF re = df_split(raw[b][r].x, c.shift), im = df_split(raw[b][r].y, c.shift);
        v[b][r] = Z{make_float2(re.h, im.h), make_float2(re.l, im.l)};
      }
  } else {
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      if (gs[b] < 0) continue;
      const float4* l = c.buf + gs[b] * c.Lp;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float4 x = l[df_slot(js[b] + r * nbf)];
        v[b][r] = Z{make_float2(x.x, x.y), make_float2(x.z, x.w)};
      }
    }
    __syncthreads();  // every read of this pass is done before any write
  }
  const int tstep = L / (Ns * R);
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    if (gs[b] < 0) continue;
    const int q = (int)(((float)js[b] + 0.5f) * inv_Ns), k = js[b] - q * Ns;
    if (Ns > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[b][r] = zmul(v[b][r], __ldg(d.tw + r * k * tstep));
    }
    DftDf<R>::run(v[b], dir);
#pragma unroll
    for (int r = 0; r < R; ++r) v[b][r] = znorm(v[b][r]);
    const int base = q * Ns * R + k;
    if (!last) {
      float4* l = c.buf + gs[b] * c.Lp;
#pragma unroll
      for (int r = 0; r < R; ++r)
        l[df_slot(base + r * Ns)] = make_float4(v[b][r].h.x, v[b][r].h.y, v[b][r].l.x, v[b][r].l.y);
      continue;
    }
    const int line = c.line0 + gs[b];
    if (line >= a.nlines) continue;
    const bool folded = d.fold != 0, per_mode = a.fac_on_out && a.fp != nullptr && a.so.pmode;
    const DfLine l = df_line(d, a.so, line, folded, a.fac_on_out != 0);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int w = base + r * Ns;
      int mode;
      const long long at = df_index(d, a.so, l, w, folded, &mode);
      if (at < 0) continue;
      Z o = v[b][r];
      if (d.fold == 1) {  // W_L^(line w) as W_L^(1024 a) W_L^b
        const int m = line * w;
        o = zmul(zmul(o, __ldg(d.tw_hi + (m >> 10))), __ldg(d.tw_lo + (m & 1023)));
      }
      double2 x = make_double2(df_widen(o.h.x, -c.shift) + df_widen(o.l.x, -c.shift),
                               df_widen(o.h.y, -c.shift) + df_widen(o.l.y, -c.shift));
      if (per_mode) {
        const double f = l.f * a.fp[mode];
        x.x *= f;
        x.y *= f;
      }
      c.out[at] = x;
    }
  }
  if (!last) __syncthreads();
}

// POW2: radices 8, 4, 2 only (fewer registers)
template <bool POW2>
__global__ void __launch_bounds__(kDfThreadsMax, 1)
k_line_fft_df(const __grid_constant__ LineDfArgs d) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned s_max;
  DfCtx c;
  c.d = &d;
  c.buf = reinterpret_cast<float4*>(smem_raw);
  c.line0 = blockIdx.x * d.a.G;
  c.Lp = d.a.L + (d.a.L >> 3) + 1;
  c.smax = &s_max;
  for (int t = blockIdx.y; t < d.a.ntr; t += gridDim.y) {
    c.in = d.a.in + (long long)t * d.a.si.st;
    c.out = d.a.out + (long long)t * d.a.so.st;
    __syncthreads();  // the previous transform's reads of s_max and the buffer
    if (threadIdx.x == 0) s_max = 0;
    __syncthreads();
    int Ns = 1;
    for (int s = 0; s < d.a.nrad; ++s) {
      const bool first = s == 0, last = s == d.a.nrad - 1;
      switch (d.a.rad[s]) {
        case 8: df_pass<8>(c, Ns, first, last); break;
        case 4: df_pass<4>(c, Ns, first, last); break;
        case 2: df_pass<2>(c, Ns, first, last); break;
        case 5:
          if constexpr (!POW2) df_pass<5>(c, Ns, first, last);
          break;
        default:
          if constexpr (!POW2) df_pass<3>(c, Ns, first, last);
          break;
      }
      Ns *= d.a.rad[s];
    }
  }
}

}  // namespace

int fft_df_cap() { return kDfThreadsMax * kDfValues; }

cudaError_t launch_line_fft_df(LineDfArgs d, cudaStream_t s) {
  if (d.a.nlines <= 0 || d.a.ntr <= 0) return cudaSuccess;
  if (d.a.L > fft_df_cap() || d.a.nrad < 1) return cudaErrorInvalidValue;
  // lines per block: a power of two.  Across lines (y, z, long 1D) four to
  // sixteen adjacent ones -- 64 to 256 contiguous bytes -- while they fit 512
  // threads of eight values; along x as many as give 128 threads.
  const bool across = d.in_across || d.out_across;
  int G = 1, lg = 0;
  while (G < 16 && 2 * G * d.a.L <= fft_df_cap() &&
         (across ? (G < 4 || 2 * G * d.a.L <= 2048) : G * d.a.L < 128 * kDfValues)) {
    G *= 2;
    ++lg;
  }
  // a narrower block where that leaves the chip short of blocks
  while (!across && G > 1 && (long long)((d.a.nlines + G - 1) / G) * d.a.ntr < 2 * 152) {
    G /= 2;
    --lg;
  }
  d.a.G = G;
  d.a.log2G = lg;
  const int threads = ((G * d.a.L + kDfValues - 1) / kDfValues + 31) / 32 * 32;
  const size_t smem = (size_t)G * (d.a.L + d.a.L / 8 + 1) * sizeof(float4);
  const bool pow2 = (d.a.L & (d.a.L - 1)) == 0;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(pow2 ? k_line_fft_df<true> : k_line_fft_df<false>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  dim3 grid((d.a.nlines + G - 1) / G, d.a.ntr < 65535 ? d.a.ntr : 65535);
  if (pow2) k_line_fft_df<true><<<grid, threads, smem, s>>>(d);
  else k_line_fft_df<false><<<grid, threads, smem, s>>>(d);
  return cudaGetLastError();
}

// exp(dir 2 pi i step m / n), m < count, as float pairs: FP64's last bit lies
// below a pair's.
__global__ void k_df_twiddles(float4* out, double dir, long long n, long long step, int count) {
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= count) return;
  double re, im;
  sincospi(2.0 * (double)(step * m % n) / (double)n, &im, &re);
  const DF r = df_from(re), i = df_from(dir * im);
  out[m] = make_float4(r.h, i.h, r.l, i.l);
}

cudaError_t launch_df_twiddles(float4* out, int dir, long long n, long long step, int count, cudaStream_t s) {
  k_df_twiddles<<<(count + 127) / 128, 128, 0, s>>>(out, (double)dir, n, step, count);
  return cudaGetLastError();
}

}  // namespace cfg
