// gbf_pair.cuh — FP32-pair arithmetic, logarithm and exponential for the
// FP64 step (gbf_f64_pair.cuh).
//
// A pair (h, l) is the unevaluated sum of two FP32 numbers, about 48
// significant bits. The operations are the error-free transformations TwoSum
// (Knuth, TAOCP vol. 2, sec. 4.2.2), FastTwoSum and TwoProduct through FMA
// (Dekker 1971), every one of them with an explicit rounding, so that the
// compiler can neither fuse nor reorder them. GB300 issues FP32 at 58 times
// its FP64 rate: a pair product is 7 instructions, about 1/8 of a DFMA's cost.
#pragma once

#include <math.h>

#include "gbf_internal.h"

struct GbfPf {
  float h, l;
};
// Exact double -> pair for host-side constants (48 bits kept).
__host__ __device__ __forceinline__ GbfPf pf_const(double d) {
  const float h = (float)d;
  return {h, (float)(d - (double)h)};
}

__device__ __forceinline__ GbfPf pf_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
// |a| >= |b|, or a = 0
__device__ __forceinline__ GbfPf pf_fast(float a, float b) {
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ GbfPf pf_neg(GbfPf a) { return {-a.h, -a.l}; }
__device__ __forceinline__ GbfPf pf_add(GbfPf a, GbfPf b) {
  const GbfPf s = pf_two_sum(a.h, b.h);
  return pf_fast(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ GbfPf pf_sub(GbfPf a, GbfPf b) { return pf_add(a, pf_neg(b)); }
__device__ __forceinline__ GbfPf pf_addf(GbfPf a, float b) {
  const GbfPf s = pf_two_sum(a.h, b);
  return pf_fast(s.h, __fadd_rn(s.l, a.l));
}
// a product, its parts not renormalised (|l| up to about 2^-22 |h|)
__device__ __forceinline__ GbfPf pf_mul_raw(GbfPf a, GbfPf b) {
  const float p = __fmul_rn(a.h, b.h);
  return {p, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.l, __fmaf_rn(a.h, b.h, -p)))};
}
__device__ __forceinline__ GbfPf pf_mul(GbfPf a, GbfPf b) {
  const GbfPf p = pf_mul_raw(a, b);
  return pf_fast(p.h, p.l);
}
__device__ __forceinline__ GbfPf pf_mulf_raw(GbfPf a, float b) {
  const float p = __fmul_rn(a.h, b);
  return {p, __fmaf_rn(a.l, b, __fmaf_rn(a.h, b, -p))};
}
__device__ __forceinline__ GbfPf pf_mulf(GbfPf a, float b) {
  const GbfPf p = pf_mulf_raw(a, b);
  return pf_fast(p.h, p.l);
}
__device__ __forceinline__ float pf_rcp(float x) {  // about 1 ulp (PTX rcp.approx)
#ifdef __CUDACC__
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return 1.f / x;  // the tests' build for the CPU
#endif
}
// a / b
__device__ __forceinline__ GbfPf pf_div(GbfPf a, GbfPf b) {
  const float rc = pf_rcp(b.h), q = __fmul_rn(a.h, rc);
  const float rem = __fadd_rn(__fmaf_rn(-q, b.h, a.h), __fmaf_rn(-q, b.l, a.l));
  return pf_fast(q, __fmul_rn(rem, rc));
}

// ------------------------------------------- FP64 <-> FP32 on integer units
// FP64 <-> FP32 conversions run on GB300's FP64 unit, at the rate of a DFMA
// (1.9 lanes a clock and SM measured; integer operations 53 and more), and so
// does a conversion that is predicated off: the forms below are integer
// operations on the bit fields for every input, with no instruction kept for
// the rare ones.
__device__ __forceinline__ bool gbf_is_zero(double d) {
  return (((unsigned)__double2hiint(d) << 1) | (unsigned)__double2loint(d)) == 0u;
}
__device__ __forceinline__ bool gbf_is_finite(double d) { return ((unsigned)__double2hiint(d) & 0x7ff00000u) != 0x7ff00000u; }

// (double)f, exact; subnormal f gives 0.
__device__ __forceinline__ double gbf_f2d(float f) {
  const unsigned b = __float_as_uint(f), u = b & 0x7fffffffu;
  const unsigned hi = (u >> 3) + (u >= 0x7f800000u ? 0x70000000u : 0x38000000u);
  const bool zero = u < 0x00800000u;
  return __hiloint2double((int)((b & 0x80000000u) | (zero ? 0u : hi)), (int)(zero ? 0u : u << 29));
}
// The pair nearest to d: |d - (h + l)| <= 2^-48 |d| for |d| in [2^-74, 2^128);
// below, the 24 leading bits (below 2^-126: 0).
__device__ __forceinline__ GbfPf pf_from_double(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const unsigned a = hi & 0x7fffffffu, sg = hi & 0x80000000u;
  // h: the leading 24 bits; l: the 29 bits below them, rounded to 24: their
  // leading 23 and last 6 bits as FP32 integers (2^23 + n, minus 2^23)
  const unsigned r = lo & 0x1fffffffu;
  unsigned h = ((a - (896u << 20)) << 3) | (lo >> 29);
  unsigned sc = ((a >> 20) - 948u) << 23;
  if (a < (897u << 20)) h = 0u;
  if (a < (949u << 20)) sc = 0u;
  if (a >= (1151u << 20)) {
    h = a > 0x7ff00000u || (a == 0x7ff00000u && lo != 0u) ? 0x7fffffffu : 0x7f800000u;
    sc = 0u;
  }
  const float n = __fmaf_rn(__fsub_rn(__uint_as_float(0x4b000000u + (r >> 6)), 8388608.f), 64.f,
                            __fsub_rn(__uint_as_float(0x4b000000u + (r & 63u)), 8388608.f));
  const float l = __fmul_rn(n, __uint_as_float(sg | sc)), hf = __uint_as_float(sg | h);
  const float s = __fadd_rn(hf, l);
  return {s, __fsub_rn(l, __fsub_rn(s, hf))};
}
__device__ __forceinline__ double pf_to_double(GbfPf a) { return __dadd_rn(gbf_f2d(a.h), gbf_f2d(a.l)); }

// The conversions with every input's exact result. (float)d, and (double)(float)d in fd.
static __device__ __noinline__ float gbf_d2f_general(double d, double* fd) {
  const float f = (float)d;
  *fd = (double)f;
  return f;
}
__device__ __forceinline__ float gbf_d2f(double d, double& fd) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const unsigned a = hi & 0x7fffffffu;
  if (a - (897u << 20) < (253u << 20)) {  // a normal result, whichever way it rounds
    // round the 53-bit number to 24 bits, ties to even, carrying into the exponent
    const unsigned t = lo + 0x0fffffffu + ((lo >> 29) & 1u);
    const unsigned h = hi + (t < lo ? 1u : 0u);
    fd = __hiloint2double((int)h, (int)(t & 0xe0000000u));
    return __uint_as_float((hi & 0x80000000u) | (((h & 0x7fffffffu) - (896u << 20)) << 3) | (t >> 29));
  }
  if ((a | lo) == 0u) {
    fd = d;
    return __uint_as_float(hi);
  }
  return gbf_d2f_general(d, &fd);
}
// d as an FP32 pair, h = (float)d, l = (float)(d - h) (gbf_df_from_double).
static __device__ __noinline__ float2 gbf_d2f2_general(double d) {
  const float h = (float)d;
  return make_float2(h, (float)(d - (double)h));
}
__device__ __forceinline__ float2 gbf_d2f2(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const unsigned a = hi & 0x7fffffffu;
  if (a - (960u << 20) < (190u << 20)) {  // both parts normal
    double fd;
    const float h = gbf_d2f(d, fd);
    // d - h in units of d's last place, a signed 29-bit integer: its leading
    // 23 and last 6 bits as FP32 integers, their sum rounded once
    const int n = (int)lo - __double2loint(fd);
    const float n1 = __fsub_rn(__uint_as_float(0x4b400000u + (unsigned)(n >> 6)), 12582912.f);
    const float n2 = __fsub_rn(__uint_as_float(0x4b000000u + ((unsigned)n & 63u)), 8388608.f);
    const unsigned sc = ((a >> 20) - 948u) << 23;
    return make_float2(h, __fmul_rn(__fmaf_rn(n1, 64.f, n2), __uint_as_float((hi & 0x80000000u) | sc)));
  }
  if ((a | lo) == 0u) return make_float2(__uint_as_float(hi), 0.f);
  return gbf_d2f2_general(d);
}
// (double)f
__device__ __forceinline__ double gbf_f2d_all(float f) {
  const unsigned b = __float_as_uint(f), u = b & 0x7fffffffu;
  unsigned m = u, e = u >= 0x7f800000u ? 0x70000000u : 0x38000000u;
  if (u < 0x00800000u && u != 0u) {  // subnormal: normalised
    const int n = __clz((int)u) - 8;
    m = (u << n) & 0x007fffffu;
    e = (unsigned)(897 - n) << 20;
  }
  return __hiloint2double((int)((b & 0x80000000u) | (u == 0u ? 0u : (m >> 3) + e)), (int)(m << 29));
}

// ------------------------------------------------------ ln and 2^x tables
// Table-driven in the manner of Tang (ACM TOMS 15, 1989; 16, 1990), the
// reduced argument and the last sums in FP64, the polynomials (the part below
// 2^-20 of ln, below 2^-9 of 2^x) in FP32 pairs: five FP64 instructions a
// function where CUDA's log and exp take about 27 each (55 for the pair at
// the measured 10.9e9 a second). The entries are computed at compile time
// from the series of atanh and exp. 512 and 256 entries: the cubic terms are
// then below 2^-31 of the result's scale, within a pair's reach, and the
// tables (14 KB) stay in L1.
constexpr int kPfLnBits = 9, kPfExpBits = 8;
constexpr unsigned kPfLnOff = 0x3f300000u;  // 0.6875: ln's reduced argument lies in [0.6875, 1.375)
constexpr double kPfLn2 = 0.693147180559945309417232121458;
struct GbfLnEntry {
  float ic, icm1;  // 1 / c in 11 bits, 1 / c - 1 (exact)
  double lnc;
};
struct GbfPfTables {
  GbfLnEntry ln[1 << kPfLnBits];
  double ex[1 << kPfExpBits];    // 2^(i / 256)
  float2 exp_pf[1 << kPfExpBits];  // the same as a pair
};
// Sums of two FP64 numbers, for entries rounded once: error-free product by
// Dekker's splitting, products of two of them to about 2^-104.
struct GbfDd {
  double h, l;
};
constexpr GbfDd dd_fast(double a, double b) {
  const double s = a + b;
  return {s, b - (s - a)};
}
constexpr double dd_top(double a) {
  const double t = 134217729.0 * a;
  return t - (t - a);
}
constexpr GbfDd dd_prod(double a, double b) {
  const double p = a * b, ah = dd_top(a), al = a - ah, bh = dd_top(b), bl = b - bh;
  return {p, ((ah * bh - p) + ah * bl + al * bh) + al * bl};
}
constexpr GbfDd dd_mul(GbfDd a, GbfDd b) {
  const GbfDd p = dd_prod(a.h, b.h);
  return dd_fast(p.h, p.l + (a.h * b.l + a.l * b.h));
}
constexpr GbfDd dd_div(double a, double b) {
  const double q = a / b;
  const GbfDd p = dd_prod(q, b);
  return dd_fast(q, ((a - p.h) - p.l) / b);
}
// 2 atanh(z), z = (c - 1) / (c + 1), |z| < 0.19: 2 z (1 + z^2 (1/3 + z^2 t)), t
// in plain FP64 (z^4 < 2^-9). c in 11 bits.
constexpr double pf_cx_ln(double c) {
  const GbfDd z = dd_div(c - 1.0, c + 1.0), z2 = dd_mul(z, z);
  double t = 0.0;
  for (int k = 41; k >= 5; k -= 2) t = t * z2.h + 1.0 / k;
  const GbfDd third = dd_div(1.0, 3.0), zt = dd_mul(z2, GbfDd{t, 0.0});
  const GbfDd u = dd_mul(z2, dd_fast(third.h, third.l + zt.h + zt.l));
  const GbfDd s = dd_mul(z, dd_fast(1.0, u.h + u.l));
  return 2.0 * s.h;
}
constexpr double pf_cx_exp(double x) {
  double s = 1.0;
  for (int k = 22; k >= 1; k--) s = 1.0 + s * x / k;
  return s;
}
constexpr GbfPfTables pf_make_tables() {
  GbfPfTables t = {};
  for (int i = 0; i < (1 << kPfLnBits); i++) {
    // interval i of [0.6875, 1.375): FP32 numbers with these 9 bits above kPfLnOff's
    const bool up = i >= 320;  // [0.6875, 1): steps of 2^-10; [1, 1.375): steps of 2^-9
    const double x0 = up ? 1.0 + (i - 320) / 512.0 : 0.6875 + i / 1024.0, w = up ? 1.0 / 512.0 : 1.0 / 1024.0;
    double ic = (double)(long long)(1024.0 / (x0 + 0.5 * w) + 0.5) / 1024.0;
    if (i == 319 || i == 320) ic = 1.0;  // both sides of 1: ln c = 0, so ln is relatively accurate there
    t.ln[i].ic = (float)ic;
    t.ln[i].icm1 = (float)(ic - 1.0);
    t.ln[i].lnc = -pf_cx_ln(ic);
  }
  for (int i = 0; i < (1 << kPfExpBits); i++) {
    const double e = pf_cx_exp(kPfLn2 * i / 256.0);
    t.ex[i] = e;
    t.exp_pf[i].x = (float)e;
    t.exp_pf[i].y = (float)(e - (double)(float)e);
  }
  return t;
}
static __device__ const GbfPfTables g_pf_tab = pf_make_tables();

// x^2 and x^3 f of a pair x.
struct GbfPfPowers {
  float p, pe;  // x^2
  float c, ce;  // x^3 f
};
__device__ __forceinline__ GbfPfPowers pf_powers(GbfPf x, GbfPf f) {
  GbfPfPowers w;
  w.p = __fmul_rn(x.h, x.h);
  w.pe = __fmaf_rn(__fadd_rn(x.h, x.h), x.l, __fmaf_rn(x.h, x.h, -w.p));
  const GbfPf x3 = pf_mul_raw(GbfPf{w.p, w.pe}, x), c = pf_mul_raw(x3, f);
  w.c = c.h;
  w.ce = c.l;
  return w;
}

// ln(1 - om) for 1 - om in (2^-12, 1.37); omf: om in FP32. Error below 2^-51 of
// ln (the entry, r and two sums rounded, the entry up to 1.5 ln; 2^-50.7 for om in
// (-2^-9, 0), where r is twice as long), in the mean 2^-53.7. 1 - om = 2^k m, m in
// [0.6875, 1.375).
template <bool LOW>
__device__ __forceinline__ double pf_ln1m_k(double om, unsigned tmp) {
  const GbfLnEntry* t = &g_pf_tab.ln[(int)(tmp >> (23 - kPfLnBits)) & ((1 << kPfLnBits) - 1)];
  float2 ic = __ldg(reinterpret_cast<const float2*>(t));
  double lnc = __ldg(&t->lnc);
  if (LOW) {
    const int k = (int)tmp >> 23;
    ic.x = __fmul_rn(ic.x, __uint_as_float((unsigned)(127 - k) << 23));
    ic.y = __fsub_rn(ic.x, 1.f);  // exact: 11 bits times at most 2^12
    lnc = __fma_rn((double)k, kPfLn2, lnc);
  }
  const double r = __fma_rn(-gbf_f2d(ic.x), om, gbf_f2d(ic.y));  // m / c - 1: nothing cancels as om -> 0
  const GbfPf x = pf_from_double(r);
  // x^3 (1/3 - x/4 + x^2/5 - x^3/6), the terms beyond 1/3 in the pair's low part
  const GbfPfPowers w = pf_powers(x, GbfPf{0.333333343f, __fmaf_rn(x.h, __fmaf_rn(x.h, __fmaf_rn(x.h, -0.166666672f, 0.2f), -0.25f),
                                                                   -9.93410776e-9f)});
  const GbfPf s = pf_fast(__fmul_rn(-0.5f, w.p), w.c);
  const double corr = pf_to_double(GbfPf{s.h, __fadd_rn(s.l, __fmaf_rn(-0.5f, w.pe, w.ce))});
  return __dadd_rn(__dadd_rn(lnc, r), corr);
}
static __device__ __noinline__ double pf_ln1m_low(double om, unsigned tmp) { return pf_ln1m_k<true>(om, tmp); }
__device__ __forceinline__ double gbf_ln1m(double om, float omf) {
  const unsigned tmp = __float_as_uint(__fsub_rn(1.f, omf)) - kPfLnOff;
  return tmp >> 23 ? pf_ln1m_low(om, tmp) : pf_ln1m_k<false>(om, tmp);
}

// The reduced exponential of 2^u, |u| < 1000 (2^u a normal number): 2^u = 2^(n / 256) (1 + e), |e| < 2^-9.5.
struct GbfPfExp {
  GbfPf e;
  int n;
};
__device__ __forceinline__ int pf_exp_index(float u, float& n256) {
  const float v = __fadd_rn(u, 49152.f);  // 1.5 2^15: the nearest multiple of 1 / 256 in the low mantissa bits
  n256 = __fsub_rn(v, 49152.f);
  return (int)(__float_as_uint(v) & 0x7fffffu) - 0x400000;
}
__device__ __forceinline__ GbfPf pf_exp_poly(GbfPf f) {  // 2^f - 1, |f| <= 2^-9 or little more
  const GbfPf t = pf_mul_raw(f, GbfPf{0.693147182f, -1.90465421e-9f});
  const GbfPfPowers w = pf_powers(t, GbfPf{0.166666672f, -4.96705388e-9f});
  const float q = __fmul_rn(__fmul_rn(w.p, w.p), __fmaf_rn(t.h, 8.33333377e-3f, 4.16666679e-2f));
  const GbfPf s = pf_fast(t.h, __fmul_rn(0.5f, w.p)), z = pf_fast(s.h, w.c);
  return pf_fast(z.h, __fadd_rn(__fadd_rn(z.l, s.l), __fadd_rn(t.l, __fadd_rn(__fmaf_rn(0.5f, w.pe, w.ce), q))));
}
__device__ __forceinline__ GbfPfExp pf_exp2_reduce(double u, float uf) {
  float n256;
  GbfPfExp x;
  x.n = pf_exp_index(uf, n256);
  x.e = pf_exp_poly(pf_from_double(__dsub_rn(u, gbf_f2d(n256))));
  return x;
}
// 2^(n / 256) in FP64
__device__ __forceinline__ double pf_exp2_scale(int n) {
  const double T = __ldg(&g_pf_tab.ex[n & 255]);
  return __hiloint2double(__double2hiint(T) + (n >> 8) * (1 << 20), __double2loint(T));
}
// 2^u and 1 - 2^u in FP64; 2^u as a pair: 2^-46 and its argument's rounding, |u|
// 2^-48 (-100 < u < 127: P_k's u is above -0.33 / lambda and below 11 / lambda <= 88).
__device__ __forceinline__ double gbf_exp2(double u, float uf) {
  const GbfPfExp x = pf_exp2_reduce(u, uf);
  const double T = pf_exp2_scale(x.n);
  return __fma_rn(T, pf_to_double(x.e), T);
}
__device__ __forceinline__ double gbf_one_minus_exp2(double u, float uf) {
  const GbfPfExp x = pf_exp2_reduce(u, uf);
  const double T = pf_exp2_scale(x.n);
  return __fma_rn(-T, pf_to_double(x.e), __dsub_rn(1.0, T));  // 1 - T is exact for T in [1/2, 2]
}
__device__ __forceinline__ GbfPf pf_exp2(GbfPf u) {
  float n256;
  const int n = pf_exp_index(u.h, n256);
  const GbfPf e = pf_exp_poly(pf_fast(__fsub_rn(u.h, n256), u.l));
  const float2 T = __ldg(&g_pf_tab.exp_pf[n & 255]);
  const float m = __fmul_rn(T.x, e.h), me = __fmaf_rn(T.x, e.h, -m);
  const GbfPf s = pf_fast(T.x, m);
  const GbfPf r = pf_fast(s.h, __fadd_rn(s.l, __fadd_rn(T.y, __fmaf_rn(T.y, e.h, __fmaf_rn(T.x, e.l, me)))));
  const float sc = __uint_as_float((unsigned)((n >> 8) + 127) << 23);
  return {__fmul_rn(r.h, sc), __fmul_rn(r.l, sc)};
}
