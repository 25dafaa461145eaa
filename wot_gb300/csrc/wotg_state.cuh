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
  double* red;     // kRedBlocks x kNq reduction partials
  double* scal;    // kNq final sums + misc scalars
};

constexpr int kNq = 8;
constexpr int kRedBlocks = 296;

struct Geom {
  int64_t I, J, ldc;
  int row_grid;             // standalone row pass: CTAs
  int ncb, nrb;             // column pass: blocks of 1024 columns x row blocks
  int64_t rows_per;         // rows per row block
};

// Exponents of two elements: plain (w - k2 C, one rounding) or precise (relative
// to the grid offset o with the weight's and kappa2's low parts, see split_weight),
// from -o, -k2 and -k2l. As packed FP32 pairs: the passes are bound by instruction
// issue (24 instructions per element in scalar form, of which the exponential is one).
template <bool PREC>
__device__ __forceinline__ float2 expo2(float2 cc, float2 w, float2 wl, float2 no, float2 nk2, float2 nk2l) {
  if (PREC) return __fadd2_rn(__ffma2_rn(nk2, cc, __fadd2_rn(w, no)), __ffma2_rn(nk2l, cc, wl));
  return __ffma2_rn(nk2, cc, w);
}
__device__ __forceinline__ float2 pair_of(float x) { return make_float2(x, x); }
// a - b of pairs (the product by -1 is exact; a negated pair costs two instructions)
__device__ __forceinline__ float2 sub2_rn(float2 a, float2 b) { return __ffma2_rn(b, pair_of(-1.f), a); }

// One step of an online base-2 LSE: the partial (m, s) (with PREC the sum
// compensated, s - cmp) takes in four columns of a row.
template <bool PREC>
__device__ __forceinline__ void lse_step(const float4& cc, const float4& w, const float4& wl, float2 no, float2 nk2,
                                         float2 nk2l, float& m, float& s, float& cmp) {
  const float2 x01 = expo2<PREC>(make_float2(cc.x, cc.y), make_float2(w.x, w.y), make_float2(wl.x, wl.y), no, nk2, nk2l);
  const float2 x23 = expo2<PREC>(make_float2(cc.z, cc.w), make_float2(w.z, w.w), make_float2(wl.z, wl.w), no, nk2, nk2l);
  const float mn = fmaxf(m, fmaxf(fmaxf(x01.x, x01.y), fmaxf(x23.x, x23.y)));
  const float r = ex2(m - mn);
  const float2 z01 = sub2_rn(x01, pair_of(mn)), z23 = sub2_rn(x23, pair_of(mn));
  // (e0 + e1) + (e2 + e3)
  const float2 e = __fadd2_rn(make_float2(ex2(z01.x), ex2(z23.x)), make_float2(ex2(z01.y), ex2(z23.y)));
  const float v = e.x + e.y;
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
// low parts (from global or shared memory); ahead(k) is told each whole chunk's first
// float4 (of 128).
struct NoAhead {
  __device__ __forceinline__ void operator()(int) const {}
};
template <bool PREC, class Cost, class W, class Wl, class Ahead = NoAhead>
__device__ __forceinline__ void row_lse(const Cost& cost, const W& w, const Wl& wl, int nv, int lane, float o, float k2,
                                        float k2l, float& m, float& s, float& cmp, const Ahead& ahead = Ahead()) {
  m = kNegBig;
  s = 0.f;
  cmp = 0.f;
  const float2 no = pair_of(-o), nk2 = pair_of(-k2), nk2l = pair_of(-k2l);
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
    ahead(k - lane);
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
    for (int t = 0; t < 4; ++t) lse_step<PREC>(cc[t], ww[t], wlo[t], no, nk2, nk2l, m, s, cmp);
  }
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (k + 32 * t < nv) lse_step<PREC>(cn[t], w(k + 32 * t), PREC ? wl(k + 32 * t) : zero, no, nk2, nk2l, m, s, cmp);
}

// One thread's share of a column pass: the online base-2 LSE (m, s) of 4 columns (as
// two pairs), with PREC compensated by cmp, over rows.
constexpr int kColRowChunk = 4;
struct ColSums {
  float2 m[2], s[2], cmp[2];
};
__device__ __forceinline__ void col_clear(ColSums& c) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    c.m[q] = pair_of(kNegBig);
    c.s[q] = c.cmp[q] = pair_of(0.f);
  }
}
// Takes v, the sum of the new exponentials against the new maximum mn, into pair q.
template <bool PREC>
__device__ __forceinline__ void col_take(ColSums& c, int q, float2 mn, float2 v) {
  const float2 d = sub2_rn(c.m[q], mn);
  const float2 r = make_float2(ex2(d.x), ex2(d.y));
  if (PREC) {
    // kahan_add of both columns
    const float2 s = __fmul2_rn(c.s[q], r), cm = __fmul2_rn(c.cmp[q], r);
    const float2 y = sub2_rn(v, cm), t = __fadd2_rn(s, y);
    c.cmp[q] = sub2_rn(sub2_rn(t, s), y);
    c.s[q] = t;
  } else {
    c.s[q] = __ffma2_rn(c.s[q], r, v);
  }
  c.m[q] = mn;
}
// NR rows of costs cc with their weights; no the columns' -offsets (PREC).
template <bool PREC, int NR>
__device__ __forceinline__ void col_rows(const float4 (&cc)[NR], const float (&ww)[NR], const float (&wlo)[NR],
                                         const float2 (&no)[2], float2 nk2, float2 nk2l, ColSums& c) {
  float2 x[2][NR];
#pragma unroll
  for (int t = 0; t < NR; ++t) {
    x[0][t] = expo2<PREC>(make_float2(cc[t].x, cc[t].y), pair_of(ww[t]), pair_of(wlo[t]), no[0], nk2, nk2l);
    x[1][t] = expo2<PREC>(make_float2(cc[t].z, cc[t].w), pair_of(ww[t]), pair_of(wlo[t]), no[1], nk2, nk2l);
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    float2 mn = c.m[q];
#pragma unroll
    for (int t = 0; t < NR; ++t) mn = make_float2(fmaxf(mn.x, x[q][t].x), fmaxf(mn.y, x[q][t].y));
    float2 v = pair_of(0.f);
#pragma unroll
    for (int t = 0; t < NR; ++t) {
      const float2 z = sub2_rn(x[q][t], mn);
      const float2 e = make_float2(ex2(z.x), ex2(z.y));
      v = t == 0 ? e : __fadd2_rn(v, e);
    }
    col_take<PREC>(c, q, mn, v);
  }
}

template <bool PREC>
__device__ __forceinline__ void col_result(const ColSums& c, float (&m)[4], float (&s)[4]) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    m[2 * q] = c.m[q].x;
    m[2 * q + 1] = c.m[q].y;
    s[2 * q] = PREC ? c.s[q].x - c.cmp[q].x : c.s[q].x;
    s[2 * q + 1] = PREC ? c.s[q].y - c.cmp[q].y : c.s[q].y;
  }
}

// The same over rows [r0, r1): cost(i) loads the columns' float4 of row i, w(i) and
// wl(i) the row's weight; o the columns' offsets (PREC); ahead(i) is told each whole
// chunk's first row.
template <bool PREC, class I, class Cost, class W, class Wl, class Ahead = NoAhead>
__device__ __forceinline__ void col_lse(const Cost& cost, const W& w, const Wl& wl, I r0, I r1, const float (&o)[4],
                                        float k2, float k2l, float (&m)[4], float (&s)[4], const Ahead& ahead = Ahead()) {
  ColSums c;
  col_clear(c);
  const float2 no[2] = {make_float2(-o[0], -o[1]), make_float2(-o[2], -o[3])};
  const float2 nk2 = pair_of(-k2), nk2l = pair_of(-k2l);
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
    ahead((int)i);
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
    col_rows<PREC, kColRowChunk>(cc, ww, wlo, no, nk2, nk2l, c);
  }
  for (; i < r1; ++i) {
    const float4 cc[1] = {cost(i)};
    const float ww[1] = {w(i)}, wlo[1] = {PREC ? wl(i) : 0.f};
    col_rows<PREC, 1>(cc, ww, wlo, no, nk2, nk2l, c);
  }
  col_result<PREC>(c, m, s);
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
