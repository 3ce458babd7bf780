// df.cuh -- double-float arithmetic on packed pairs: two independent FP32
// pairs (re and im of a complex value, or two kernel taps) per float2, every
// step one f32x2 instruction on both halves, each half an IEEE operation.
// Used by the kernels of FP64 plans that stay off GB300's FP64 units (about
// 2 FMAs per clock and SM, a sixty-fourth of the FP32 rate).
#pragma once

#include "device_common.cuh"

namespace cfg {

__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
// a - b, rounded once (the product with -1 is exact)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// Two unevaluated sums h + l (lanes x and y).
struct DF2 {
  float2 h, l;
};
__device__ __forceinline__ DF2 df2_dup(DF a) { return DF2{dup2(a.h), dup2(a.l)}; }
// s + e = a + b exactly (Knuth); fast_two_sum2 needs |a| >= |b| (Dekker)
__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2& s, float2& e) {
  s = add2(a, b);
  const float2 bb = sub2(s, a);
  e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}
__device__ __forceinline__ DF2 fast_two_sum2(float2 a, float2 b) {
  DF2 r;
  r.h = add2(a, b);
  r.l = sub2(b, sub2(r.h, a));
  return r;
}
// a * b to ~2^-46 relative, h the rounded product (not renormalised: |l| a
// few ulps of h)
__device__ __forceinline__ DF2 df2_mul(DF2 a, DF2 b) {
  DF2 r;
  r.h = mul2(a.h, b.h);
  r.l = fma2(a.h, b.h, neg2(r.h));
  r.l = fma2(a.h, b.l, r.l);
  r.l = fma2(a.l, b.h, r.l);
  return r;
}
__device__ __forceinline__ DF2 df2_add(DF2 a, DF2 b) {
  float2 s, e;
  two_sum2(a.h, b.h, s, e);
  return DF2{s, add2(e, add2(a.l, b.l))};
}
// (s, t) += a * b: the sum's rounding errors and the product's low parts
// collect in t (twelve instructions)
__device__ __forceinline__ void df2_acc(float2& s, float2& t, float2 ah, float2 al, float2 bh, float2 bl) {
  const float2 p = mul2(ah, bh);
  float2 pe = fma2(ah, bh, neg2(p));
  pe = fma2(ah, bl, pe);
  pe = fma2(al, bh, pe);
  float2 n, e;
  two_sum2(s, p, n, e);
  s = n;
  t = add2(t, add2(e, pe));
}
// The same for long sums (a tile cell under up to a subproblem's points):
// renormalised, so that the low part -- and its rounding -- stays below an ulp
// of the sum instead of growing with the number of terms (1000 points on one
// cell: 2e-13 -> 4e-14 relative).  nah = -ah, so that no step needs a negated
// operand (fifteen instructions).
__device__ __forceinline__ void df2_acc_long(float2& s, float2& t, float2 ah, float2 nah, float2 al, float2 bh,
                                             float2 bl) {
  const float2 np = mul2(nah, bh);
  float2 pe = fma2(ah, bh, np);
  pe = fma2(ah, bl, pe);
  pe = fma2(al, bh, pe);
  const float2 n = sub2(s, np);
  const float2 bb = sub2(n, s);
  const float2 e = sub2(sub2(s, sub2(n, bb)), add2(np, bb));
  const float2 low = add2(t, add2(e, pe));
  s = add2(n, low);
  t = sub2(low, sub2(s, n));
}
// (s, t, u) += a * b where s starts at a power of two of at least twice any
// partial sum of the products: then s - (s + ab) is exact (no branch, no
// two-sum), so one FMA rounds the sum, one recovers its error, and t, u
// collect errors and low parts (six instructions; absolute error ~2^-48 of
// that power per product).
__device__ __forceinline__ void df2_acc_biased(float2& s, float2& t, float2& u, float2 ah, float2 al, float2 bh,
                                               float2 bl) {
  const float2 n = fma2(ah, bh, s);
  t = add2(t, fma2(ah, bh, sub2(s, n)));
  u = fma2(ah, bl, u);
  u = fma2(al, bh, u);
  s = n;
}
// The least power of two that is at least twice b (b > 0, far from the ends
// of the exponent range).
__device__ __forceinline__ float bias_for(float b) {
  return __int_as_float((__float_as_int(b) & 0x7f800000) + (2 << 23));
}

// v 2^shift as an FP32 pair, by integer operations on the exponent and
// mantissa fields (a conversion, a subtraction and a second conversion would
// each occupy the FP64 unit): h the top 24 bits rounded to nearest, l the
// signed rest of 29 bits rounded to 24.  Below 2^-126 (and for FP64 subnormals)
// the result is zero; infinities and NaNs give NaN.
__device__ __forceinline__ DF df_split(double v, int shift) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const unsigned hi = (unsigned)(b >> 32), lo = (unsigned)b;
  const int ef = (int)((hi >> 20) & 0x7ffu);
  const int e = ef - 896 + shift;  // FP32 exponent field of v 2^shift
  const unsigned sign = hi & 0x80000000u;
  // exponent and mantissa of |v|, half a unit of h added: a carry may reach
  // the exponent, as it should
  const unsigned long long up = (b & 0x7fffffffffffffffull) + 0x10000000ull;
  DF r;
  r.h = __uint_as_float(sign | ((unsigned)(up >> 29) + ((unsigned)(shift - 896) << 23)));
  const float ls = __uint_as_float(sign | ((unsigned)(e > 52 ? e - 52 : 0) << 23));
  r.l = __int2float_rn((int)(lo << 3) >> 3) * ls;
  if (ef == 0 || e <= 0) r.h = r.l = 0.f;
  if (ef == 0x7ff || e >= 254) r.h = __uint_as_float(0x7fc00000u);
  return r;
}

// (h + l) 2^k as double by widening h and l through their exponent fields (an
// FP64 addition is left; conversions would take the same narrow unit).
__device__ __forceinline__ double df_widen(float v, int k) {
  const unsigned b = __float_as_uint(v);
  const int ef = (int)((b >> 23) & 0xffu);
  const int e = ef + 896 + k;
  if (ef == 0xff) return __longlong_as_double(((long long)((b & 0x80000000u) | 0x7ff80000u)) << 32);
  if (ef == 0 || e <= 0) return 0.0;  // below 2^-126 of the block's largest, or of FP64's range
  const unsigned hi = e >= 2047 ? 0x7ff00000u : ((unsigned)e << 20) | ((b >> 3) & 0xfffffu);
  const unsigned lo = e >= 2047 ? 0u : b << 29;
  return __longlong_as_double(((long long)((b & 0x80000000u) | hi) << 32) | lo);
}

// ---- ES kernel rows in double-float ---------------------------------------
// kh[j] + kl[j] = phi(d - NS/2 + j) 2^-E, E = round(beta log2 e), to ~2^-46
// of the peak.
//
// Fitted polynomials (kerevalmeth 1): taps j and NS-1-j are mirror images,
// p_{NS-1-j}(z) = p_j(-z), so one Horner chain in z^2 on the pair (even
// part, odd part) gives both: half the steps of two chains, packed.
//
// z = 2 d - 1 and z^2 of a point's offset.
__device__ __forceinline__ void df_poly_arg(double d, DF& z, DF& w) {
  const DF d0 = df_split(d, 1);  // 2 d
  float zh, ze;
  two_sum(-1.f, d0.h, zh, ze);
  z = df_renorm(zh, __fadd_rn(ze, d0.l));
  w = df_mul(z, z);
}
// taps p (lane x) and NS-1-p (lane y)
template <int NS>
__device__ __forceinline__ DF2 df_poly_pair(DF z, DF w1, int p, const DFCoef<double>& c) {
  constexpr int HD = horner_degree<double>(NS), NP = (NS + 1) / 2, NK = HD / 2;
  const DF2 w = df2_dup(w1);
  DF2 v = DF2{c.ph[p], c.pl[p]};
#pragma unroll
  for (int k = 1; k <= NK; ++k) v = df2_add(df2_mul(v, w), DF2{c.ph[k * NP + p], c.pl[k * NP + p]});
  // even + z odd, even - z odd
  const DF o = df_mul(DF{v.h.y, v.l.y}, z);
  const DF2 r = df2_add(DF2{dup2(v.h.x), dup2(v.l.x)}, DF2{make_float2(o.h, -o.h), make_float2(o.l, -o.l)});
  return fast_two_sum2(r.h, r.l);
}
template <int NS>
__device__ __forceinline__ void df_poly_row(double d, const DFCoef<double>& c, float* kh, float* kl) {
  DF z, w;
  df_poly_arg(d, z, w);
#pragma unroll
  for (int p = 0; p < (NS + 1) / 2; ++p) {
    const DF2 q = df_poly_pair<NS>(z, w, p, c);
    kh[p] = q.h.x;
    kl[p] = q.l.x;
    kh[NS - 1 - p] = p == NS - 1 - p ? q.h.x : q.h.y;
    kl[NS - 1 - p] = p == NS - 1 - p ? q.l.x : q.l.y;
  }
}

// exp form: phi / e^beta = 2^y, y = -(beta log2 e) z / (1 + sqrt(1 - z)),
// z = c x^2 (see es_value_fast: the exponent is small where phi is large,
// so ~2^-46 relative in y stays ~2^-47 of the peak in phi).  sqrt and the
// quotient: the hardware approximation and one Newton step on the exact
// residual.  2^y = 2^n 2^(k/64) e^g: an integer, a table (which carries
// e^beta 2^-E) and a short series, |g| <= ln 2 / 128, its terms from g^3 on
// in FP32 (< 3e-8, so 2^-24 of that is below 2^-48).  Taps at x0 + d0 (lane x) and x1 + d0 (lane y)
__device__ __forceinline__ DF2 df_exp_pair(DF d0, float x0, float x1, const DFCoef<double>& c, const float2* tab) {
  const float2 one = dup2(1.f);
  const DF2 cc = DF2{dup2(c.c_h), dup2(c.c_l)}, mb = DF2{dup2(-c.b_h), dup2(-c.b_l)};
  const DF2 ln2 = DF2{dup2(0.693147182464599609375f), dup2(-1.904654323148236e-09f)};
  float2 s, e;
  two_sum2(make_float2(x0, x1), dup2(d0.h), s, e);
  const DF2 x = fast_two_sum2(s, add2(e, dup2(d0.l)));
  DF2 z = df2_mul(x, x);
  z = df2_mul(cc, z);
  z = fast_two_sum2(z.h, z.l);
  // u = 1 - z >= 0, s = sqrt(u)
  DF2 u = fast_two_sum2(one, neg2(z.h));
  u = fast_two_sum2(u.h, sub2(u.l, z.l));
  const bool in0 = u.h.x > 0.f, in1 = u.h.y > 0.f;  // outside the support the kernel is zero
  u.h = make_float2(fmaxf(u.h.x, 1e-30f), fmaxf(u.h.y, 1e-30f));
  const float2 r = make_float2(rsqrt_approx(u.h.x), rsqrt_approx(u.h.y));
  const float2 s0 = mul2(u.h, r);
  const float2 res = add2(fma2(neg2(s0), s0, u.h), u.l);
  DF2 q = fast_two_sum2(one, s0);                   // 1 + sqrt(u)
  q.l = fma2(mul2(res, dup2(0.5f)), r, q.l);
  // v = z / q
  const float2 rq = make_float2(rcp_approx(q.h.x), rcp_approx(q.h.y));
  const float2 v0 = mul2(z.h, rq);
  float2 rem = fma2(neg2(v0), q.h, z.h);
  rem = fma2(neg2(v0), q.l, add2(rem, z.l));
  const DF2 v = fast_two_sum2(v0, mul2(rem, rq));
  const DF2 y = df2_mul(mb, v);
  // n + k/64 nearest y (the added constant leaves its integer in the mantissa)
  const float2 magic = dup2(12582912.f);
  const float2 m = __ffma2_rn(y.h, dup2(64.f), magic);
  const int i0 = __float_as_int(m.x) - 0x4b400000, i1 = __float_as_int(m.y) - 0x4b400000;
  const float2 f0 = __ffma2_rn(sub2(m, magic), dup2(-0.015625f), y.h);
  two_sum2(f0, y.l, s, e);
  const DF2 g = df2_mul(DF2{s, e}, ln2);
  // e^g - 1 = g + g^2/2 + g^3 (1/6 + g/24 + g^2/120)
  const float2 hg = mul2(g.h, dup2(0.5f));
  const float2 sq = mul2(g.h, hg);
  float2 lo = fma2(g.h, hg, neg2(sq));
  lo = fma2(g.h, g.l, lo);
  float2 p = fma2(g.h, dup2(1.f / 120.f), dup2(1.f / 24.f));
  p = fma2(p, g.h, dup2(1.f / 6.f));
  lo = fma2(mul2(mul2(sq, g.h), dup2(2.f)), p, lo);
  two_sum2(g.h, sq, s, e);
  const DF2 em = DF2{s, add2(e, add2(g.l, lo))};
  const float2 t0 = tab[i0 & 63], t1 = tab[i1 & 63];
  const DF2 t = DF2{make_float2(t0.x, t1.x), make_float2(t0.y, t1.y)};
  const DF2 pr = df2_mul(t, em);
  DF2 w = fast_two_sum2(t.h, pr.h);
  w = fast_two_sum2(w.h, add2(w.l, add2(t.l, pr.l)));
  const float2 sc = make_float2(__int_as_float(((i0 >> 6) + 127) << 23), __int_as_float(((i1 >> 6) + 127) << 23));
  const float2 in = make_float2(in0 ? sc.x : 0.f, in1 ? sc.y : 0.f);
  return DF2{mul2(w.h, in), mul2(w.l, in)};
}
template <int NS>
__device__ __forceinline__ void df_exp_row(double d, const DFCoef<double>& c, const float2* tab, float* kh,
                                           float* kl) {
  const DF d0 = df_split(d, 0);
#pragma unroll
  for (int p = 0; p < (NS + 1) / 2; ++p) {
  const DF2 q = df_exp_pair(d0, float(p) - 0.5f * NS, float(NS - 1 - p) - 0.5f * NS, c, tab);
  kh[p] = q.h.x;
  kl[p] = q.l.x;
  kh[NS - 1 - p] = p == NS - 1 - p ? q.h.x : q.h.y;
  kl[NS - 1 - p] = p == NS - 1 - p ? q.l.x : q.l.y;
  }
}

template <int NS>
__device__ __forceinline__ void df_kernel_row(double d, const KernelCoeffs<double>& kc, const float2* tab, float* kh,
                                              float* kl) {
  if (kc.horner) df_poly_row<NS>(d, kc.df, kh, kl);
  else df_exp_row<NS>(d, kc.df, tab, kh, kl);
}

// Taps p (lane x) and NS-1-p (lane y) alone: a block whose threads share a
// point's row evaluates it pair by pair.
template <int NS>
__device__ __forceinline__ DF2 df_kernel_pair(double d, int p, const KernelCoeffs<double>& kc, const float2* tab) {
  if (kc.horner) {
    DF z, w;
    df_poly_arg(d, z, w);
    return df_poly_pair<NS>(z, w, p, kc.df);
  }
  return df_exp_pair(df_split(d, 0), float(p) - 0.5f * NS, float(NS - 1 - p) - 0.5f * NS, kc.df, tab);
}

// The block's copy of the 2^(k/64) table (64 entries; the caller syncs).
__device__ __forceinline__ void df_table_fill(float2* tab, const KernelCoeffs<double>& kc) {
  for (int i = threadIdx.x; i < 64; i += blockDim.x) tab[i] = kc.df.exp2_tab[i];
}

}  // namespace cfg
