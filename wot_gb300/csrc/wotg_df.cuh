// wotg_df.cuh — sums and logarithms of half-steps as FP32 pairs.
//
// An FP64 instruction holds its SM sub-partition's FP64 unit for 64 cycles on
// this part, for one active lane as for 32 (measured: DADD, DMUL, DFMA and the
// F32 <-> F64 conversions 64 cycles each, log2(double) 2190, exp(double) 1080).
// A half-step ends in one merge and one logarithm per row, which in FP64 took
// longer than the row's exponentials at the sizes of a day pair. Here the merge
// runs on unevaluated FP32 pairs (h, l), value h + l, of 46 to 48 significant
// bits, against the 22 bits of the exponentials that are summed; the error-free
// transformations are Dekker's and Knuth's (T. J. Dekker, Numer. Math. 18, 1971;
// D. E. Knuth, TAOCP 2, 4.2.2).
#pragma once

#include "wotg_common.cuh"

namespace wotg {

// a + b = s + e exactly.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
// The same for |a| >= |b|.
__device__ __forceinline__ void fast_two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  e = __fsub_rn(b, __fsub_rn(s, a));
}
// (h, l) *= f
__device__ __forceinline__ void df_scale(float& h, float& l, float f) {
  const float p = __fmul_rn(h, f);
  l = __fmaf_rn(l, f, __fmaf_rn(h, f, -p));
  h = p;
}
// (h, l) += (h2, l2)
__device__ __forceinline__ void df_add(float& h, float& l, float h2, float l2) {
  float s, e;
  two_sum(h, h2, s, e);
  fast_two_sum(s, __fadd_rn(e, __fadd_rn(l, l2)), h, l);
}

// Merge of base-2 partials (m, h + l) over the lanes that differ in the bits of
// `FROM` .. `TO` (powers of two): every lane ends with the group's total. The
// scale factors are the FP32 ex2 (2 ulp).
template <int FROM, int TO>
__device__ __forceinline__ void df_merge_lanes(float& m, float& h, float& l) {
#pragma unroll
  for (int o = FROM; o >= TO; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o);
    float h2 = __shfl_xor_sync(0xffffffffu, h, o);
    float l2 = __shfl_xor_sync(0xffffffffu, l, o);
    const float mn = fmaxf(m, m2);
    df_scale(h, l, ex2(m - mn));
    df_scale(h2, l2, ex2(m2 - mn));
    df_add(h, l, h2, l2);
    m = mn;
  }
}

// Table of log2_pair: entry i holds 1 / c and -log2 of it as a pair, for the
// centre c of [1 + i/128, 1 + (i + 1)/128).
constexpr int kLogTable = 128;
__device__ __forceinline__ float4 log_table_entry(int i) {
  const float rc = (float)(1.0 / (1.0 + ((double)i + 0.5) / kLogTable));
  const double t = -log2((double)rc);
  const float th = (float)t;
  return make_float4(rc, th, (float)(t - (double)th), 0.f);
}

// log2(h + l) = c + d + f for h in [2^-100, 2^100]: table-driven (P. T. P. Tang, ACM
// TOMS 16, 1990): h + l = 2^e mant, r = mant / c - 1 with |r| < 1/255, the series
// of log(1 + r) with its first two terms as pairs. Absolute error about 2^-48 (as a
// pair, c + d rounded, it was 2^-44: enough to move a weight's low part, of 2^-39
// units, in every fourth iteration, and with it single FP32 exponents).
__device__ __forceinline__ void log2_pair(float h, float l, const float4* tab, float& c, float& d, float& f) {
  const int b = __float_as_int(h);
  const int e = (b >> 23) - 127;
  const float scale = __int_as_float((127 - e) << 23);
  const float mh = __int_as_float((b & 0x7FFFFF) | 0x3F800000), ml = __fmul_rn(l, scale);
  const float4 t = tab[(b >> 16) & 127];
  const float p = __fmul_rn(mh, t.x);
  float rh, rl;
  fast_two_sum(__fsub_rn(p, 1.f), __fmaf_rn(ml, t.x, __fmaf_rn(mh, t.x, -p)), rh, rl);
  const float q = __fmul_rn(rh, rh);
  const float ql = __fmaf_rn(__fmul_rn(2.f, rh), rl, __fmaf_rn(rh, rh, -q));
  float g = __fmaf_rn(rh, -1.f / 6.f, 0.2f);
  g = __fmaf_rn(rh, g, -0.25f);
  g = __fmaf_rn(rh, g, 1.f / 3.f);
  float a, bl;                                            // log(1 + r)
  fast_two_sum(rh, __fmul_rn(-0.5f, q), a, bl);
  bl = __fadd_rn(bl, __fadd_rn(rl, __fmaf_rn(__fmul_rn(q, rh), g, __fmul_rn(-0.5f, ql))));
  constexpr float kH = 1.44269502f, kL = 1.92596295e-8f;  // log2 e
  float x = __fmul_rn(a, kH);
  float xl = __fmaf_rn(a, kL, __fmaf_rn(bl, kH, __fmaf_rn(a, kH, -x)));
  float s, sl, u, ul;
  two_sum(t.y, x, s, sl);
  two_sum((float)e, s, u, ul);
  c = u;
  float v, vl;
  two_sum(ul, sl, v, vl);
  fast_two_sum(v, __fadd_rn(vl, __fadd_rn(t.z, xl)), d, f);
}

// Base-2 log-sum-exp o + m + log2(h + l) in FP64.
__device__ __forceinline__ double lse2_pair(float o, float m, float h, float l, const float4* tab) {
  if (!(h >= 0x1p-100f && h <= 0x1p100f)) return (double)o + (double)m + log2((double)h + (double)l);
  float c, d, f;
  log2_pair(h, l, tab, c, d, f);
  return ((double)o + (double)m) + ((double)c + ((double)d + (double)f));
}

}  // namespace wotg
