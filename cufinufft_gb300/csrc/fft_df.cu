// fft_df.cu -- line FFTs of FP64 grids in double-float arithmetic (FP32 pairs).
//
// cuFFT's Z2Z transform is bound by GB300's FP64 unit: a butterfly level is
// ~3 FP64 instructions per value at a sixty-fourth of the FP32 rate, against
// ~18 packed FP32 instructions here.  A d-dimensional transform is one pass
// per axis over only the lines and positions that carry modes (LineArgs,
// linemap.cuh), with the amplification fused into the first pass of type 2 and
// the deconvolution into the last of type 1: the zero padding is neither
// written, read nor transformed.
//
// A block transforms G lines in one padded shared buffer by Stockham passes of
// radix 4, 2, 5, 3, every thread holding four to six values in registers
// between reading and writing.  Values travel as (re hi, im hi, re
// lo, im lo); the block scales its lines by the power of two that brings the
// largest input to [1, 2), so any FP64 range passes.  Along y and z a block's G
// lines are adjacent, so a row segment of G cells is contiguous.
//
// A 1D transform beyond 4096 points is two such passes, L = L1 L2: columns n2
// of x[n1 L2 + n2], multiplied by W_L^(n2 k1), then rows k1, whose output k2
// lands at k1 + L1 k2.
//
// Four values per thread and 64 registers (radix 4 at most) rather than eight
// with radix 8 and 128: the chains are latency, and 32 warps per SM hide more of
// it than one exchange less saves (256^3: 0.87 against 0.99 ms; 2048^2: 0.277
// against 0.275).  What bounds it now: instruction issue and latency, 30-40% of
// cycles issued; the FMA pipe would allow a quarter of the time.
//
// Measured (FFT with amplification or deconvolution; cuFFT, or the unpruned 2D
// double-float form, with the mode-row kernel before): 2048^2 type 2 403 -> 277
// us, 256^3 type 2 3.71 -> 0.87 ms, 150x192x162 type 1 1.03 -> 0.41 ms, 405000
// points type 2 672 -> 89 us.
#include <cuda_runtime.h>

#include "df.cuh"
#include "linemap.cuh"

namespace cfg {
namespace {

constexpr int kDfThreadsMax = 1024;
constexpr int kDfValues = 4;  // values per thread (radix 5: 5, radix 3: 6)

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

// One Stockham pass of radix R over the block's G lines in shared memory:
// every thread reads its butterflies, waits, and writes them back in order.
// The first pass reads FP64 values and splits them.
template <int R>
__device__ __forceinline__ void df_pass(const LineDfArgs& d, float4* buf, int Lp, int Ns, bool first, int shift) {
  constexpr int NB = (kDfValues + R - 1) / R;  // butterflies per thread
  const int L = d.a.L, nbf = L / R, total = d.a.G * nbf;
  const float inv_nbf = 1.f / (float)nbf, inv_Ns = 1.f / (float)Ns;
  const float dir = (float)d.a.dir;
  Z v[NB][R];
  int at[NB], js[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int u = threadIdx.x + b * blockDim.x;
    const int g = (int)(((float)u + 0.5f) * inv_nbf);
    js[b] = u - g * nbf;
    at[b] = g * Lp;
    if (u >= total) {
      at[b] = -1;
      continue;
    }
    const float4* l = buf + at[b];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float4 x = l[df_slot(js[b] + r * nbf)];
      if (first) {
        const double2 y = make_double2(__hiloint2double(__float_as_int(x.y), __float_as_int(x.x)),
                                       __hiloint2double(__float_as_int(x.w), __float_as_int(x.z)));
        const DF re = df_split(y.x, shift), im = df_split(y.y, shift);
        v[b][r] = Z{make_float2(re.h, im.h), make_float2(re.l, im.l)};
      } else {
        v[b][r] = Z{make_float2(x.x, x.y), make_float2(x.z, x.w)};
      }
    }
  }
  __syncthreads();  // every read of this pass is done before any write
  const int tstep = L / (Ns * R);
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    if (at[b] < 0) continue;
    const int q = (int)(((float)js[b] + 0.5f) * inv_Ns), k = js[b] - q * Ns;
    if (!first) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[b][r] = zmul(v[b][r], __ldg(d.tw + r * k * tstep));
    }
    DftDf<R>::run(v[b], dir);
    const int base = q * Ns * R + k;
    float4* l = buf + at[b];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const Z o = znorm(v[b][r]);
      l[df_slot(base + r * Ns)] = make_float4(o.h.x, o.h.y, o.l.x, o.l.y);
    }
  }
  __syncthreads();
}

// POW2: radices 4 and 2 only (fewer registers).  Load, passes and store each
// go through shared memory: the index and factor arithmetic of the pruned lines
// stays out of the butterflies, whose registers decide the occupancy.
template <bool POW2>
__global__ void __launch_bounds__(kDfThreadsMax, 1)
k_line_fft_df(const __grid_constant__ LineDfArgs d) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned s_max;
  const LineArgs<double>& a = d.a;
  float4* buf = reinterpret_cast<float4*>(smem_raw);
  const int line0 = blockIdx.x * a.G, L = a.L, total = a.G * L, Lp = L + (L >> 3) + 1;
  const float inv_L = 1.f / (float)L;
  for (int t = blockIdx.y; t < a.ntr; t += gridDim.y) {
    __syncthreads();  // the previous transform's reads
    if (threadIdx.x == 0) s_max = 0;
    __syncthreads();
    unsigned m = 0;
    {
      const double2* in = a.in + (long long)t * a.si.st;
      const bool folded = d.fold == 1, per_mode = !a.fac_on_out && a.fp != nullptr && a.si.pmode;
#pragma unroll 4
      for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int g = d.in_across ? e & (a.G - 1) : (int)(((float)e + 0.5f) * inv_L);
        const int w = d.in_across ? e >> a.log2G : e - g * L;
        double2 v = make_double2(0.0, 0.0);
        if (line0 + g < a.nlines) {
          const DfLine l = df_line(d, a.si, line0 + g, folded, per_mode);
          int mode;
          const long long at = df_index(d, a.si, l, w, folded, &mode);
          if (at >= 0) {
            v = in[at];
            if (per_mode) {
              const double f = l.f * a.fp[mode];
              v.x *= f;
              v.y *= f;
            }
          }
        }
        const unsigned x = (unsigned)__double2hiint(v.x) & 0x7fffffffu, y = (unsigned)__double2hiint(v.y) & 0x7fffffffu;
        if (x < 0x7ff00000u) m = max(m, x);
        if (y < 0x7ff00000u) m = max(m, y);
        reinterpret_cast<double2*>(buf)[g * Lp + df_slot(w)] = v;
      }
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_max, m);
    __syncthreads();
    const int shift = 1023 - (int)(s_max >> 20);
    int Ns = 1;
    for (int s = 0; s < a.nrad; ++s) {
      const bool first = s == 0;
      switch (a.rad[s]) {
        case 4: df_pass<4>(d, buf, Lp, Ns, first, shift); break;
        case 2: df_pass<2>(d, buf, Lp, Ns, first, shift); break;
        case 5:
          if constexpr (!POW2) df_pass<5>(d, buf, Lp, Ns, first, shift);
          break;
        default:
          if constexpr (!POW2) df_pass<3>(d, buf, Lp, Ns, first, shift);
          break;
      }
      Ns *= a.rad[s];
    }
    double2* out = a.out + (long long)t * a.so.st;
    const bool folded = d.fold != 0, per_mode = a.fac_on_out && a.fp != nullptr && a.so.pmode;
#pragma unroll 4
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      const int g = d.out_across ? e & (a.G - 1) : (int)(((float)e + 0.5f) * inv_L);
      const int w = d.out_across ? e >> a.log2G : e - g * L;
      if (line0 + g >= a.nlines) continue;
      const DfLine l = df_line(d, a.so, line0 + g, folded, per_mode);
      int mode;
      const long long at = df_index(d, a.so, l, w, folded, &mode);
      if (at < 0) continue;
      const float4 x = buf[g * Lp + df_slot(w)];
      Z o = Z{make_float2(x.x, x.y), make_float2(x.z, x.w)};
      if (d.fold == 1) {  // W_L^(line w) as W_L^(1024 a) W_L^b
        const int k = (line0 + g) * w;
        o = zmul(zmul(o, __ldg(d.tw_hi + (k >> 10))), __ldg(d.tw_lo + (k & 1023)));
      }
      double2 y = make_double2(df_widen(o.h.x, -shift) + df_widen(o.l.x, -shift),
                               df_widen(o.h.y, -shift) + df_widen(o.l.y, -shift));
      if (per_mode) {
        const double f = l.f * a.fp[mode];
        y.x *= f;
        y.y *= f;
      }
      out[at] = y;
    }
  }
}

}  // namespace

int fft_df_cap() { return kDfThreadsMax * kDfValues; }

cudaError_t launch_line_fft_df(LineDfArgs d, cudaStream_t s) {
  if (d.a.nlines <= 0 || d.a.ntr <= 0) return cudaSuccess;
  if (d.a.L > fft_df_cap() || d.a.nrad < 1) return cudaErrorInvalidValue;
  // lines per block: a power of two.  Across lines (y, z, long 1D) four to
  // sixteen adjacent ones -- 64 to 256 contiguous bytes -- while they fit a
  // block; along x as many as give 128 threads.
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
  if (smem > 47 * 1024) {
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
