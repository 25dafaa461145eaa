// wotg_state.cuh — state of one transport solve on the device and the
// element arithmetic of the streamed (materialised) half-steps, shared by the
// persistent solver kernel (wotg_persist.cuh), the on-the-fly form and the
// standalone half-step.
#pragma once

#include <stdint.h>

#include "wotg_coef.cuh"
#include "wotg_common.cuh"

namespace wotg {

// Per-solve vectors in the caller's workspace.
struct Vecs {
  double* u;       // I   absorbed potential (reference u)
  double* v;       // J
  double* la;      // I   log a
  double* lb;      // J   log b
  double* la_old;  // I   log a at the start of the last iteration (stage-exit test)
  double* lb_old;  // J
  double* logp;    // I   log p (p = G of this growth iteration)
  double* p;       // I
  double* Lrow;    // I   log sum_j exp(v_j/eps + lb_j - kappa C_ij)
  double* Lcol;    // J   log sum_i exp(u_i/eps + la_i - kappa C_ij)
  float* wrow;     // I   (u_i/eps + la_i) * log2(e), FP32 operand of the column pass (hi part, see split_weight)
  float* wcol;     // ldc (v_j/eps + lb_j) * log2(e), zero in padding columns (hi part)
  float* wrow_lo;  // I   remainders of the weights (lo parts)
  float* wcol_lo;  // ldc
  float4* rowc;    // I   per-row constants of the dense coupling (coupling_rows_kernel)
  float2* part;    // nrb x ldc column-pass partials (m, s) in base 2
  unsigned long long* maxslot;  // 2 slots of max(a, b) bits, alternating per iteration
  double* red;     // kRedBlocks x kNq reduction partials
  double* scal;    // kNq final sums + misc scalars
  int* counters;   // [0] absorptions
};

constexpr int kNq = 8;
constexpr int kRedBlocks = 296;

struct Geom {
  int64_t I, J, ldc;
  int row_grid;             // standalone row pass: CTAs
  int ncb, nrb;             // column pass: blocks of 1024 columns x row blocks
  int64_t rows_per;         // rows per row block
};

// exp(la) as the absorption test needs it: the test only compares the largest
// exp(la) with tau, so away from log(tau) the value is 0 (below) or +inf
// (above) with the same outcome, and the FP64 exp (slow on this part) is formed
// only within 1e-9 of log(tau). NaN stays NaN.
__device__ __forceinline__ double absorb_key(double la, const Coef& c) {
  if (la < c.ltau_lo) return 0.0;
  if (la > c.ltau_hi) return INFINITY;
  return exp(la);
}

// Exponent of one element: plain (w - k2 C, one rounding) or precise (relative
// to the grid offset o with the weight's and kappa2's low parts, see
// split_weight).
template <bool PREC>
__device__ __forceinline__ float expo(float cc, float w, float wl, float o, float k2, float k2l) {
  if (PREC) return fmaf(-k2, cc, w - o) + fmaf(-k2l, cc, wl);
  return fmaf(-k2, cc, w);
}

// One step of an online base-2 LSE: the partial (m, s) (with PREC the sum
// compensated, s - cmp) takes in the four exponents x.
template <bool PREC>
__device__ __forceinline__ void lse_step(float x0, float x1, float x2, float x3, float& m, float& s, float& cmp) {
  const float mn = fmaxf(m, fmaxf(fmaxf(x0, x1), fmaxf(x2, x3)));
  const float r = ex2(m - mn);
  const float v = (ex2(x0 - mn) + ex2(x1 - mn)) + (ex2(x2 - mn) + ex2(x3 - mn));
  if (PREC) {
    s = __fmul_rn(s, r);
    cmp = __fmul_rn(cmp, r);
    kahan_add(s, cmp, v);
  } else {
    s = s * r + v;
  }
  m = mn;
}

// One lane's share of a row's online base-2 LSE: float4 columns lane, lane + 32,
// ... < nv, in order; (m, s) as partial s 2^m, with PREC the sum compensated,
// s - cmp. cost(k), w(k), wl(k) load float4 k of the row, the weights and their
// low parts (from global or shared memory).
template <bool PREC, class Cost, class W, class Wl>
__device__ __forceinline__ void row_lse(const Cost& cost, const W& w, const Wl& wl, int nv, int lane, float o, float k2,
                                        float k2l, float& m, float& s, float& cmp) {
  m = kNegBig;
  s = 0.f;
  cmp = 0.f;
  auto step = [&](const float4& cc, const float4& ww, const float4& wlo) {
    lse_step<PREC>(expo<PREC>(cc.x, ww.x, wlo.x, o, k2, k2l), expo<PREC>(cc.y, ww.y, wlo.y, o, k2, k2l),
                   expo<PREC>(cc.z, ww.z, wlo.z, o, k2, k2l), expo<PREC>(cc.w, ww.w, wlo.w, o, k2, k2l), m, s, cmp);
  };
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  // the cost loads of the next 128-float4 chunk are issued before this
  // chunk's arithmetic (two chunks of loads in flight per lane)
  float4 cn[4];
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (lane + 32 * t < nv) cn[t] = cost(lane + 32 * t);
  int k = lane;
  const int full = nv & ~127;   // whole chunks; the last, partial one follows
  for (; k < full; k += 128) {
    float4 cc[4], ww[4], wlo[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) cc[t] = cn[t];
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (k + 128 + 32 * t < nv) cn[t] = cost(k + 128 + 32 * t);
#pragma unroll
    for (int t = 0; t < 4; ++t) ww[t] = w(k + 32 * t);
#pragma unroll
    for (int t = 0; t < 4; ++t) wlo[t] = PREC ? wl(k + 32 * t) : zero;
#pragma unroll
    for (int t = 0; t < 4; ++t) step(cc[t], ww[t], wlo[t]);
  }
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (k + 32 * t < nv) step(cn[t], w(k + 32 * t), PREC ? wl(k + 32 * t) : zero);
}

// One thread's share of a column pass: the online base-2 LSE of 4 columns over
// rows [r0, r1), in chunks of kColRowChunk rows. cost(i) loads the columns'
// float4 of row i, w(i) and wl(i) the row's weight; o the columns' offsets (PREC).
constexpr int kColRowChunk = 4;

template <bool PREC, class I, class Cost, class W, class Wl>
__device__ __forceinline__ void col_lse(const Cost& cost, const W& w, const Wl& wl, I r0, I r1, const float (&o)[4],
                                        float k2, float k2l, float (&m)[4], float (&s)[4]) {
  float cmp[4] = {0.f, 0.f, 0.f, 0.f};   // PREC: compensated sums s - cmp
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    m[q] = kNegBig;
    s[q] = 0.f;
  }
  I i = r0;
  // the next chunk's cost loads are issued before this chunk's arithmetic
  float4 cn[kColRowChunk];
  if (i + kColRowChunk <= r1) {
#pragma unroll
    for (int t = 0; t < kColRowChunk; ++t) cn[t] = cost(i + t);
  }
  for (; i + kColRowChunk <= r1; i += kColRowChunk) {
    float4 cc[kColRowChunk];
    float ww[kColRowChunk], wlo[kColRowChunk];
#pragma unroll
    for (int t = 0; t < kColRowChunk; ++t) cc[t] = cn[t];
    if (i + 2 * kColRowChunk <= r1) {
#pragma unroll
      for (int t = 0; t < kColRowChunk; ++t) cn[t] = cost(i + kColRowChunk + t);
    }
#pragma unroll
    for (int t = 0; t < kColRowChunk; ++t) ww[t] = w(i + t);
#pragma unroll
    for (int t = 0; t < kColRowChunk; ++t) wlo[t] = PREC ? wl(i + t) : 0.f;
    float x[4][kColRowChunk];
#pragma unroll
    for (int t = 0; t < kColRowChunk; ++t) {
      x[0][t] = expo<PREC>(cc[t].x, ww[t], wlo[t], o[0], k2, k2l);
      x[1][t] = expo<PREC>(cc[t].y, ww[t], wlo[t], o[1], k2, k2l);
      x[2][t] = expo<PREC>(cc[t].z, ww[t], wlo[t], o[2], k2, k2l);
      x[3][t] = expo<PREC>(cc[t].w, ww[t], wlo[t], o[3], k2, k2l);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float mx = x[q][0];
#pragma unroll
      for (int t = 1; t < kColRowChunk; ++t) mx = fmaxf(mx, x[q][t]);
      const float mn = fmaxf(m[q], mx);
      const float r = ex2(m[q] - mn);
      float v = 0.f;
#pragma unroll
      for (int t = 0; t < kColRowChunk; ++t) v += ex2(x[q][t] - mn);
      if (PREC) {
        s[q] = __fmul_rn(s[q], r);
        cmp[q] = __fmul_rn(cmp[q], r);
        kahan_add(s[q], cmp[q], v);
      } else {
        s[q] = s[q] * r + v;
      }
      m[q] = mn;
    }
  }
  for (; i < r1; ++i) {
    const float4 cc = cost(i);
    const float ww = w(i);
    const float wlo = PREC ? wl(i) : 0.f;
    const float xs[4] = {expo<PREC>(cc.x, ww, wlo, o[0], k2, k2l), expo<PREC>(cc.y, ww, wlo, o[1], k2, k2l),
                         expo<PREC>(cc.z, ww, wlo, o[2], k2, k2l), expo<PREC>(cc.w, ww, wlo, o[3], k2, k2l)};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float mn = fmaxf(m[q], xs[q]);
      const float r = ex2(m[q] - mn);
      if (PREC) {
        s[q] = __fmul_rn(s[q], r);
        cmp[q] = __fmul_rn(cmp[q], r);
        kahan_add(s[q], cmp[q], ex2(xs[q] - mn));
      } else {
        s[q] = s[q] * r + ex2(xs[q] - mn);
      }
      m[q] = mn;
    }
  }
  if (PREC) {
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] -= cmp[q];
  }
}

// The gap terms of one point: x = exp(t) its marginal sum (t = log x), p its
// target, the scaling a~ = exp(la) exp(u/eps) evaluated as the reference does.
// Where nothing overflows or underflows, log(x / p) = t - log p and
// log a~ = la + u/eps (to an ulp), which saves four of the six FP64
// transcendentals per point (slow on this part); at the edges the reference's
// own expressions run, so overflow, 0 log 0 and NaN behave as in the reference.
__device__ __forceinline__ void gap_terms(double t, double la, double ue, double p, double logp, double lambda,
                                          double eps, double* x_out, double* f_out, double* conj_out) {
  const double x = exp(t);
  double f, conj;
  if (x > 0.0 && fabs(t) < 700.0 && fabs(la) < 700.0 && fabs(ue) < 700.0 && fabs(la + ue) < 700.0 && p > 0.0) {
    f = x * (t - logp) - x + p;
    conj = lambda * p * (exp(-eps * (la + ue) / lambda) - 1.0);
  } else {
    const double at = exp(la) * exp(ue);
    f = x * log(x / p) - x + p;
    conj = lambda * p * (exp(-eps * log(at) / lambda) - 1.0);
  }
  *x_out = x;
  *f_out = f;
  *conj_out = conj;
}

}  // namespace wotg
