// wotg_resident.cuh — the persistent solver for costs that fit in the SMs' shared
// memory. A CTA takes whole row blocks, so that a few blocks more than SMs double the
// rows of its plan: costs of up to some 3.5e6 entries fit, of squarish ones about
// 70 % at 4e6, 40 % at 4.5e6 and 20 % at 5e6 (2000 x 2500, with 167 blocks of 12 rows,
// does not); the others run streamed or on the fly.
//
// A CTA owns whole row blocks of the column pass and keeps their rows of C, its
// FP64 state and the column weights in shared memory, so the row weights never
// leave it: an iteration is
//   row phase     a warp per owned row, then a thread per row (log2, a-update)
//   column phase  a warp per (row block, 128 columns): partials to the owners
//                 of the columns                                    | exchange
//   merge phase   a warp per owned float4 column, b-update: weights to every
//                 CTA                                               | exchange
// with two exchanges in place of three grid barriers. An exchange carries its
// own flags: a consumer polls the data words themselves until they show the
// iteration's tag (a value and its tag are one 64-bit word, so no fence is
// needed), which takes one trip to L2 and back after the write instead of the
// 2300 cycles of a grid barrier (fence, atomic, poll). Overwriting is safe
// without more: weights of iteration e are written by a CTA that holds the
// partials of e of every row block, i.e. after every CTA has read all weights of
// e - 1; partials of e are written after all weights of e - 1 were read, i.e.
// after every merge of e - 1. Grid barriers remain where sums are tested.
//
// What bounds it: a chain of latencies (about 8 us an iteration with grid
// barriers at 1237 x 1511, of which the element arithmetic is 1.3): L2 round
// trips, and FP64 instructions at 64 cycles each. The per-point coefficients of
// the updates are therefore folded once per stage (A, W: one FP64 FMA each), and
// the grid roundings of weights and offsets read the integer that the magic
// addition leaves in the low word.
#pragma once

#include "wotg_persist.cuh"

namespace wotg {

constexpr int kResidentThreads = 384;     // 12 warps: the rows of a usual block, 168 registers each
constexpr int kResidentWarps = kResidentThreads / 32;
constexpr int kResidentMaxBlocks = 256;   // row blocks a merge holds in registers (16 per lane)
constexpr int kMergeSteps = kResidentMaxBlocks / 16;
constexpr uint32_t kPollTries = 6000000;     // polls of some 0.4 us

// Sizes of a CTA's share: the most rows, rounded-up float4 columns, and bytes.
struct ResidentPlan {
  int grid, rows, cols4;
  size_t bytes;
};

inline ResidentPlan resident_plan(const Geom& g, int sms) {
  ResidentPlan p;
  p.grid = (int)(g.nrb < sms ? g.nrb : sms);
  if (p.grid < 1) p.grid = 1;
  const int64_t blocks = (g.nrb + p.grid - 1) / p.grid;
  p.rows = (int)(blocks * g.rows_per < g.I ? blocks * g.rows_per : g.I);
  const int64_t nv = g.ldc >> 2;
  p.cols4 = (int)((nv + p.grid - 1) / p.grid);
  const size_t rows = (size_t)p.rows, cols = (size_t)p.cols4 * 4;
  p.bytes = kMergeHeaderBytes + rows * g.ldc * 4 + (size_t)g.ldc * 12 + (rows + cols) * ((7 + 4) * 8 + 16 + 4) + rows * 8;
  return p;
}
inline bool resident_fits(const ResidentPlan& p, const Geom& g, size_t smem_limit) {
  return g.nrb <= kResidentMaxBlocks && p.rows <= kPersistBlk / 2 && p.cols4 * 4 <= kPersistBlk / 2 && p.bytes <= smem_limit;
}

__device__ __forceinline__ void st_words(void* p, uint64_t a, uint64_t b) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_words(const void* p, uint64_t& a, uint64_t& b) {
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ uint64_t ld_word(const uint64_t* p) {
  uint64_t a;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
  return a;
}
__device__ __forceinline__ uint64_t word(float v, uint32_t tag) {
  return (uint64_t)__float_as_uint(v) | ((uint64_t)tag << 32);
}

// A partial (m, s) as one word: s is a non-negative sum below 2^64, so s 2^-64
// leaves the sign (the iteration's parity) and the top exponent bit (a row of the
// block has a > tau) free. A non-finite s travels as m = NaN.
__device__ __forceinline__ uint64_t pack_partial(float m, float s, uint32_t parity, bool over) {
  if (!(s < 0x1p64f)) {
    m = __int_as_float(0x7FC00000);
    s = 0.f;
  }
  const uint32_t b = __float_as_uint(__fmul_rn(s, 0x1p-64f)) | (parity << 31) | ((over ? 1u : 0u) << 30);
  return (uint64_t)__float_as_uint(m) | ((uint64_t)b << 32);
}

// A column offset (on the 2^-14 grid) as one word: its grid integer and the low
// bits of the iteration; kFarOffset for an offset beyond +-1024, which is then
// in wcol_lo.
constexpr int kFarOffset = -(1 << 24);
__device__ __forceinline__ uint32_t offset_word(int n, uint32_t epoch) { return ((uint32_t)n << 7) | (epoch & 127u); }

struct Resident : PersistBase {
  // Shared memory by offset (float and double indexes kept in sh().off), so that
  // every access is a shared-memory one with a 32-bit address and no register
  // holds an array's place.
  enum : int { kWhi, kWlo, kOcols, kRhi, kRlo,                                                  // floats (C is at kC4)
               kPr, kPc,                                                                      // float4 points
               kU, kLa, kLao, kLogp, kAr, kWr, kKr, kV, kLb, kLbo, kAc, kWc, kKc, kLc, kEx };   // doubles
  static_assert(kEx < 22, "sh().off[22 .. 30] hold the CTA's share");
  enum : int { kRp = 32, kCp = 33 };   // floats: the points' third parts
  static constexpr int kC4 = (int)(kMergeHeaderBytes / 16);   // the owned rows of C, in float4s
  static constexpr int kLr = kLao;   // the old scalings are dead in the final stage, where a check keeps its row sums

  __device__ static __forceinline__ float& F(int i) { return reinterpret_cast<float*>(persist_smem)[i]; }
  __device__ static __forceinline__ float4& F4(int i) { return reinterpret_cast<float4*>(persist_smem)[i]; }
  __device__ static __forceinline__ double& D(int i) { return reinterpret_cast<double*>(persist_smem)[i]; }
  __device__ static __forceinline__ float& F(int array, int t) { return F(sh().off[array] + t); }
  __device__ static __forceinline__ double& D(int array, int t) { return D(sh().off[array] + t); }
  // A row's (column's) point: offset o on the grid; P = W + (A - alpha o ln 2) log2 e as
  // grid value and remainder (a third part, below the remainder's 2^-39 units, in kRp
  // and kCp), so that its next weight is P - alpha (L2 - o); W.
  __device__ static __forceinline__ float4& pr(int t) { return F4(sh().off[kPr] + t); }
  __device__ static __forceinline__ float4& pc(int t) { return F4(sh().off[kPc] + t); }

  // Owned row blocks [b0, b1), rows [r0, r0 + nr), float4 columns [c0, c1), columns [j0, j0 + nc).
  __device__ static __forceinline__ int r0() { return sh().off[22]; }
  __device__ static __forceinline__ int nr() { return sh().off[23]; }
  __device__ static __forceinline__ int nc() { return sh().off[24]; }
  __device__ static __forceinline__ int b0() { return sh().off[25]; }
  __device__ static __forceinline__ int b1() { return sh().off[26]; }
  __device__ static __forceinline__ int c0() { return sh().off[27]; }
  __device__ static __forceinline__ int c1() { return sh().off[28]; }
  __device__ static __forceinline__ int j0() { return sh().off[29]; }
  __device__ static __forceinline__ int nv() { return sh().off[30]; }
  // {hi | tag, lo | tag} of each column (lb_old's and Lcol's memory), the columns'
  // offset words (wcol's memory), partials at (c4 nrb + r) 4 + q
  __device__ static __forceinline__ uint64_t* wl() { return reinterpret_cast<uint64_t*>(A().V.lb_old); }
  __device__ static __forceinline__ uint32_t* ol() { return reinterpret_cast<uint32_t*>(A().V.wcol); }
  __device__ static __forceinline__ uint64_t* part() { return reinterpret_cast<uint64_t*>(A().V.part); }

  __device__ Resident(int rows_cap, int cols_cap) {
    fill_table();
    if (threadIdx.x == 0) {
      int at = 4 * kC4 + rows_cap * (int)A().g.ldc;   // floats, a multiple of 4 up to the doubles
      for (int k = kWhi; k <= kOcols; ++k) {
        sh().off[k] = at;
        at += (int)A().g.ldc;
      }
      sh().off[kPr] = at >> 2;
      at += 4 * rows_cap;
      sh().off[kPc] = at >> 2;
      at += 4 * cols_cap;
      at >>= 1;                           // doubles
      for (int k = kU; k <= kLc; ++k) {
        sh().off[k] = at;
        at += k <= kKr ? rows_cap : cols_cap;
      }
      sh().off[kEx] = at;
      at += 4 * (rows_cap + cols_cap);
      at <<= 1;                           // floats
      sh().off[kRhi] = at;
      sh().off[kRlo] = at + rows_cap;
      sh().off[kRp] = at + 2 * rows_cap;
      sh().off[kCp] = at + 3 * rows_cap;
      const int nv = (int)(A().g.ldc >> 2), n = gridDim.x, b = blockIdx.x;
      const int b0 = (int)((int64_t)A().g.nrb * b / n), b1 = (int)((int64_t)A().g.nrb * (b + 1) / n);
      const int c0 = (int)((int64_t)nv * b / n), c1 = (int)((int64_t)nv * (b + 1) / n);
      const int r0 = (int)(b0 * A().g.rows_per);
      sh().off[22] = r0;
      sh().off[23] = (int)min(A().g.I, b1 * A().g.rows_per) - r0;
      sh().off[24] = max(0, (int)min((int64_t)c1 * 4, A().g.J) - c0 * 4);
      sh().off[25] = b0;
      sh().off[26] = b1;
      sh().off[27] = c0;
      sh().off[28] = c1;
      sh().off[29] = c0 * 4;
      sh().off[30] = nv;
    }
    __syncthreads();
    const int r0 = Resident::r0(), nr = Resident::nr(), j0 = Resident::j0(), nc = Resident::nc(), nv = Resident::nv(), b0 = Resident::b0();
    const int started = A().ctl->started;
    if (threadIdx.x == 0) {
      sh().epoch = (uint32_t)A().ctl->epoch;
      sh().row_over = 0;
    }
    const float* o_row = reinterpret_cast<const float*>(A().V.rowc);
    for (int t = threadIdx.x; t < nr; t += kResidentThreads) {
      const int i = r0 + t;
      D(kU, t) = A().V.u[i];
      D(kLa, t) = A().V.la[i];
      D(kLogp, t) = A().V.logp[i];
      D(kLr, t) = started && A().ctl->lrow_valid ? A().V.Lrow[i] * kLog2e : D(kLa, t);
      pr(t).x = started ? o_row[i] : 0.f;
    }
    for (int t = threadIdx.x; t < nc; t += kResidentThreads) {
      D(kV, t) = A().V.v[j0 + t];
      D(kLb, t) = A().V.lb[j0 + t];
      D(kLbo, t) = D(kLb, t);
      const int n = started ? (int)ol()[j0 + t] >> 7 : 0;
      pc(t).x = n == kFarOffset ? A().V.wcol_lo[j0 + t] : (float)n * 0x1p-14f;
    }
    for (int t = threadIdx.x; t < A().g.ldc; t += kResidentThreads)
      if (t >= A().g.J) F(kWhi, t) = F(kWlo, t) = F(kOcols, t) = 0.f;
    const float4* C4 = reinterpret_cast<const float4*>(A().C + (int64_t)r0 * A().g.ldc);
    for (int64_t k = threadIdx.x; k < (int64_t)nr * nv; k += kResidentThreads) F4(kC4 + (int)k) = ld_stream(C4 + k);
    if (!started)   // own partials of "iteration 0", so that iteration 1's parity is new
      for (int64_t k = threadIdx.x; k < (int64_t)(b1() - b0) * nv; k += kResidentThreads) {
        uint64_t* e = part() + ((k % nv) * A().g.nrb + b0 + k / nv) * 4;
        st_words(e, 0, 0);
        st_words(e + 2, 0, 0);
      }
    __syncthreads();
  }

  // 2^-14-grid roundings by the magic addition: the float on the grid is the
  // integer in the low word of the sum.
  __device__ static __forceinline__ double near(double x, float* f) {
    if (below_1024(x)) {
      const double t = x + kGridMagic;
      *f = (float)__double2loint(t) * 0x1p-14f;
      return t - kGridMagic;
    }
    *f = grid_value(x);
    return (double)*f;
  }
  __device__ static __forceinline__ float2 split(double w) {
    if (below_1024(w)) {
      float hi;
      const double h = near(w, &hi);
      return make_float2(hi, (float)(w - h));
    }
    return split_pair(w);
  }
  // Base-2 log-sum-exp o + m + log2(h + l) in FP64.
  __device__ static __forceinline__ double lse2_own(float o, const float4& r) {
    if (!(r.y >= 0x1p-100f && r.y <= 0x1p100f)) return (double)o + (double)r.x + log2((double)r.y + (double)r.z);
    float c, d, f, a, b;
    log2_pair(r.y, r.z, mg().tab, c, d, f);
    two_sum(r.x, c, a, b);
    return (double)o + ((double)a + ((double)b + ((double)d + (double)f)));
  }
  // P of a point whose offset is now o (see pr), from K = W + A log2 e; its third part.
  __device__ static __forceinline__ void point_at(float4& p, float& third, float o, double K, double alpha) {
    const double x = fma(-alpha, (double)o, K);
    const float2 w = split(x);
    p.x = o;
    p.y = w.x;
    p.z = w.y;
    third = (float)((x - (double)w.x) - (double)w.y);
  }
  // Coefficients folded per stage: log a = A - alpha ln 2 L2, weight = W + log a log2 e = K - alpha L2.
  __device__ static __forceinline__ void fold_row(int t) {
    const double a = fma(sh().c.alpha1, D(kLogp, t), fma(D(kU, t), sh().ku, sh().a1logj)), w = D(kU, t) * sh().iel2;
    D(kAr, t) = a;
    D(kWr, t) = w;
    D(kKr, t) = fma(a, kLog2e, w);
    pr(t).w = (float)w;
    point_at(pr(t), F(kRp, t), pr(t).x, D(kKr, t), sh().c.alpha1);
  }
  __device__ static __forceinline__ void fold_col(int t) {
    const double a = fma(D(kV, t), sh().kv, sh().bconst), w = D(kV, t) * sh().iel2;
    D(kAc, t) = a;
    D(kWc, t) = w;
    D(kKc, t) = fma(a, kLog2e, w);
    pc(t).w = (float)w;
    point_at(pc(t), F(kCp, t), pc(t).x, D(kKc, t), sh().c.alpha2);
  }
  __device__ static __noinline__ void fold_all() {
    for (int t = threadIdx.x; t < nr(); t += kResidentThreads) fold_row(t);
    for (int t = threadIdx.x; t < nc(); t += kResidentThreads) fold_col(t);
  }

  // The weight and the new offset of a point from its merged sum r = (m, h, l), on
  // FP32 pairs: delta = m + log2(h + l) = L2 - o, weight = P - alpha delta. This is
  // the critical path of the exchange; the FP64 state follows beside it (settle).
  // False where the FP64 path has to decide: sums or values out of range, or a
  // scaling within 1e-3 of tau. On success r becomes (delta, flag, old offset).
  __device__ static __forceinline__ bool quick(const float4& p, float third, float4& r, float ah, float al, float& o, float& hi, float& lo,
                                        bool& over) {
    if (!(r.y >= 0x1p-100f && r.y <= 0x1p100f)) return false;
    float c, d, f, a, b, e;
    log2_pair(r.y, r.z, mg().tab, c, d, f);
    two_sum(r.x, c, a, b);
    two_sum(b, d, b, e);
    two_sum(a, b, a, b);
    fast_two_sum(a, __fadd_rn(b, __fadd_rn(e, f)), a, b);
    float n = rintf(a * 0x1p14f);
    n += rintf(__fmaf_rn(b, 0x1p14f, __fmaf_rn(a, 0x1p14f, -n)));
    o = __fmaf_rn(n, 0x1p-14f, p.x);
    const float z = __fmul_rn(ah, a);
    const float ze = __fmaf_rn(ah, a, -z) + __fmaf_rn(ah, b, __fmul_rn(al, a));
    float q, ql;
    two_sum(p.z, -z, q, ql);
    fast_two_sum(q, __fadd_rn(__fsub_rn(ql, ze), third), q, ql);
    float k = rintf(q * 0x1p14f);
    k += rintf(__fmaf_rn(ql, 0x1p14f, __fmaf_rn(q, 0x1p14f, -k)));
    hi = __fmaf_rn(k, 0x1p-14f, p.y);
    lo = __fadd_rn(__fmaf_rn(k, -0x1p-14f, q), ql);
    const float la = (hi - p.w) * (float)kLn2, t = la - (float)sh().consts[3];
    over = t > 0.f;
    if (!(fabsf(a) < 500.f && fabsf(z) < 500.f && fabsf(p.y) < 512.f && fabsf(o) < 1023.f && fabsf(hi) < 1023.f &&
          fabsf(p.w) < 4096.f && fabsf(t) > 1e-3f))
      return false;
    r = make_float4(a, b, 1.f, p.x);
    return true;
  }
  // FP64 state of a point after quick(): L2, log a and P at the new offset.
  __device__ static __forceinline__ void settle_row(int t) {
    const float4 r = mg().res[t];
    if (r.z != 1.f) return;
    const double L2 = (double)r.w + ((double)r.x + (double)r.y);
    D(kLao, t) = D(kLa, t);
    D(kLa, t) = fma(-sh().a1ln2, L2, D(kAr, t));
    point_at(pr(t), F(kRp, t), pr(t).x, D(kKr, t), sh().c.alpha1);
  }
  __device__ static __forceinline__ void settle_col(int t) {
    const float4 r = mg().res[kPersistBlk / 2 + t];
    if (r.z != 1.f) return;
    const double L2 = (double)r.w + ((double)r.x + (double)r.y);
    D(kLc, t) = L2;
    D(kLbo, t) = D(kLb, t);
    D(kLb, t) = fma(-sh().a2ln2, L2, D(kAc, t));
    point_at(pc(t), F(kCp, t), pc(t).x, D(kKc, t), sh().c.alpha2);
  }

  __device__ static __forceinline__ bool update_row(int t, double L2) {
    const double x = fma(-sh().a1ln2, L2, D(kAr, t));
    D(kLao, t) = D(kLa, t);
    D(kLa, t) = x;
    const float2 w = split(fma(x, kLog2e, D(kWr, t)));
    F(kRhi, t) = w.x;
    F(kRlo, t) = w.y;
    return over_tau(x);
  }
  // Column t's weight and offset o (on the grid) to every CTA.
  __device__ static __forceinline__ void publish(int t, float hi, float lo, float o, bool over) {
    const uint32_t tag = (sh().epoch << 1) | (over ? 1u : 0u);
    const int j = j0() + t;
    int n = kFarOffset;
    if (fabsf(o) < 1024.f) {
      n = (int)(o * 0x1p14f);
    } else {
      A().V.wcol_lo[j] = o;
      __threadfence();
    }
    asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(ol() + j), "r"(offset_word(n, sh().epoch)) : "memory");
    st_words(wl() + 2 * (int64_t)j, word(hi, tag), word(lo, tag));
  }

  // All weights and offsets of iteration `epoch` into shared memory; *over when
  // any a or b was above tau.
  __device__ static __noinline__ bool stage_weights(bool* over) {
    bool ov = false, fail = false;
    const uint32_t want = sh().epoch & 0x7FFFFFFFu, want_o = sh().epoch & 127u;
    const int J = (int)A().g.J;
    constexpr int kAtOnce = 4;
    for (int j = threadIdx.x; j < J && !fail; j += kAtOnce * kResidentThreads) {
      uint64_t a[kAtOnce], b[kAtOnce];
      uint32_t o[kAtOnce];
      for (uint32_t t = 0;; ++t) {
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k) {
          const int jk = j + k * kResidentThreads;
          if (jk < J) {
            ld_words(wl() + 2 * (int64_t)jk, a[k], b[k]);
            asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(o[k]) : "l"(ol() + jk) : "memory");
          }
        }
        bool ready = true;
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k)
          if (j + k * kResidentThreads < J)
            ready = ready && (uint32_t)(a[k] >> 33) == want && (uint32_t)(b[k] >> 33) == want &&
                    (o[k] & 127u) == want_o;
        if (ready) break;
        if (t >= kPollTries || ((t & 255) == 255 && *(volatile int*)&A().ctl->err)) {
          fail = true;
          break;
        }
      }
#pragma unroll
      for (int k = 0; k < kAtOnce; ++k) {
        const int jk = j + k * kResidentThreads;
        if (jk < J) {
          F(kWhi, jk) = __uint_as_float((uint32_t)a[k]);
          F(kWlo, jk) = __uint_as_float((uint32_t)b[k]);
          const int n = (int)o[k] >> 7;
          if (n == kFarOffset) {
            __threadfence();
            F(kOcols, jk) = *(volatile float*)(A().V.wcol_lo + jk);
          } else {
            F(kOcols, jk) = (float)n * 0x1p-14f;
          }
          ov |= (a[k] >> 32) & 1;
        }
      }
    }
    if (fail) {
      atomicExch(&A().ctl->err, 1);
      sh().ok = 0;
    }
    const int any = __syncthreads_or(ov ? 1 : 0);
    if (over) *over = any != 0;
    return sh().ok != 0;
  }

  template <bool FRESH>
  __device__ static __noinline__ void row_phase() {
    const int lane = threadIdx.x & 31;
    const int w4 = sh().off[kWhi] >> 2, wl4 = sh().off[kWlo] >> 2, nv = Resident::nv(), nr = Resident::nr(), p4 = sh().off[kPr];
    for (int t = threadIdx.x >> 5; t < nr; t += kResidentWarps) {
      float m, s, cmp, h, l;
      const int row = kC4 + t * nv;
      row_lse<true>([row](int k) { return F4(row + k); }, [w4](int k) { return F4(w4 + k); },
                    [wl4](int k) { return F4(wl4 + k); }, nv, lane, F4(p4 + t).x, sh().c.kappa2, sh().c.kappa2_lo, m, s,
                    cmp);
      two_sum(s, -cmp, h, l);
      df_merge_lanes<16, 1>(m, h, l);
      if (lane == 0) mg().res[t] = make_float4(m, h, l, 0.f);
    }
    __syncthreads();
    bool over = false;
    for (int t = threadIdx.x; t < nr; t += kResidentThreads) {
      float4 r = mg().res[t], p = F4(p4 + t);
      if (FRESH) {
        const double L2 = lse2_own(p.x, r);
        D(kLr, t) = L2;
        A().V.Lrow[r0() + t] = L2 * kLn2;
        float o;
        near(L2, &o);
        point_at(F4(p4 + t), F(kRp, t), o, D(kKr, t), sh().c.alpha1);
      } else {
        float o, hi, lo;
        bool ov;
        if (quick(p, F(kRp, t), r, sh().a1h, sh().a1l, o, hi, lo, ov)) {
          F(kRhi, t) = hi;
          F(kRlo, t) = lo;
          F4(p4 + t).x = o;
          mg().res[t] = r;
          over |= ov;
        } else {
          const double L2 = lse2_own(p.x, r);
          over |= update_row(t, L2);
          near(L2, &o);
          point_at(F4(p4 + t), F(kRp, t), o, D(kKr, t), sh().c.alpha1);
          mg().res[t].z = 0.f;
        }
      }
    }
    if (FRESH)
      __syncthreads();
    else
      sh().row_over = __syncthreads_or(over ? 1 : 0) != 0;
  }

  __device__ static __noinline__ void row_update_cached() {
    bool over = false;
    for (int t = threadIdx.x; t < nr(); t += kResidentThreads) {
      over |= update_row(t, D(kLr, t));
      mg().res[t].z = 0.f;   // nothing to settle
    }
    sh().row_over = __syncthreads_or(over ? 1 : 0) != 0;
  }

  __device__ static __noinline__ void col_phase() {
    const int lane = threadIdx.x & 31;
    const int nv = Resident::nv(), b0 = Resident::b0();
    const int ncg = (nv + 31) >> 5, units = ncg * (b1() - b0);
    const uint32_t parity = sh().epoch & 1;
    const bool over = sh().row_over != 0;
    for (int un = threadIdx.x >> 5; un < units; un += kResidentWarps) {
      const int r = un / ncg, c4 = (un % ncg) * 32 + lane;
      if (c4 >= nv) continue;
      const int a = r * (int)A().g.rows_per, e = min(nr(), a + (int)A().g.rows_per);
      float o[4], m[4], s[4];
      const float4 ov = F4((sh().off[kOcols] >> 2) + c4);
      o[0] = ov.x;
      o[1] = ov.y;
      o[2] = ov.z;
      o[3] = ov.w;
      const int wr = sh().off[kRhi], wrl = sh().off[kRlo];
      col_lse<true>([c4, nv](int i) { return F4(kC4 + i * nv + c4); }, [wr](int i) { return F(wr + i); },
                    [wrl](int i) { return F(wrl + i); }, a, e, o, sh().c.kappa2, sh().c.kappa2_lo, m, s);
      uint64_t* out = part() + ((int64_t)c4 * A().g.nrb + b0 + r) * 4;
      st_words(out, pack_partial(m[0], s[0], parity, over), pack_partial(m[1], s[1], parity, over));
      st_words(out + 2, pack_partial(m[2], s[2], parity, over), pack_partial(m[3], s[3], parity, over));
    }
  }

  // A warp per two owned columns: lane (rl, q) polls the words of column q's row
  // blocks rl, rl + 16, ... and keeps them, so that the maximum comes first.
  template <int STEPS>
  __device__ static __noinline__ void merge_phase() {
    const int lane = threadIdx.x & 31, rl = lane >> 1;
    const uint32_t parity = sh().epoch & 1;
    const int nrb = A().g.nrb;
    // rows first: their FP64 state, by the four warps with the fewest columns
    if (threadIdx.x >= kResidentThreads - 128)
      for (int t = threadIdx.x - (kResidentThreads - 128); t < nr(); t += 128) settle_row(t);
    const int c2_end = c1() * 2;
    for (int c2 = c0() * 2 + (threadIdx.x >> 5); c2 < c2_end; c2 += kResidentWarps) {
      const int col = c2 * 2 + (lane & 1);
      const uint64_t* p = part() + ((int64_t)(c2 >> 1) * nrb + rl) * 4 + (col & 3);
      uint64_t w[STEPS];
      bool ready = false;
      for (uint32_t t = 0; !ready; ++t) {
        bool mine = true;
#pragma unroll
        for (int k = 0; k < STEPS; ++k)
          w[k] = rl + k * 16 < nrb ? ld_word(p + k * 64) : 0;
#pragma unroll
        for (int k = 0; k < STEPS; ++k)
          mine = mine && (rl + k * 16 >= nrb || (uint32_t)(w[k] >> 63) == parity);
        ready = __all_sync(0xffffffffu, mine);
        if (!ready && (t >= kPollTries || ((t & 255) == 255 && *(volatile int*)&A().ctl->err))) {
          atomicExch(&A().ctl->err, 1);
          sh().ok = 0;
          break;
        }
      }
      float m = kNegBig;
      bool over = false;
#pragma unroll
      for (int k = 0; k < STEPS; ++k)
        if (rl + k * 16 < nrb) {
          m = fmaxf(m, __uint_as_float((uint32_t)w[k]));
          over |= (w[k] >> 62) & 1;
        }
#pragma unroll
      for (int o = 16; o >= 2; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      float h = 0.f, l = 0.f;
#pragma unroll
      for (int k = 0; k < STEPS; ++k)
        if (rl + k * 16 < nrb) {
          const float s = __fmul_rn(__uint_as_float((uint32_t)(w[k] >> 32) & 0x3FFFFFFFu), 0x1p64f);
          const float f = ex2(__uint_as_float((uint32_t)w[k]) - m);
          const float x = __fmul_rn(s, f);
          float e;
          two_sum(h, x, h, e);
          l = __fadd_rn(l, __fadd_rn(e, __fmaf_rn(s, f, -x)));
        }
#pragma unroll
      for (int o = 16; o >= 2; o >>= 1) {
        const float h2 = __shfl_xor_sync(0xffffffffu, h, o), l2 = __shfl_xor_sync(0xffffffffu, l, o);
        df_add(h, l, h2, l2);
      }
      over = __any_sync(0xffffffffu, over);
      const int t = col - j0();
      if (rl == 0 && t < nc()) mg().res[kPersistBlk / 2 + t] = make_float4(m, h, l, over ? 1.f : 0.f);
    }
    __syncthreads();
    // a thread per column: weights and offsets first, the FP64 state by other warps
    const int nc = Resident::nc(), p4 = sh().off[kPc];
    for (int t = threadIdx.x; t < nc; t += kResidentThreads) {
      float4 r = mg().res[kPersistBlk / 2 + t], p = F4(p4 + t);
      const bool row_flag = r.w != 0.f;
      float o, hi, lo;
      bool ov;
      if (quick(p, F(kCp, t), r, sh().a2h, sh().a2l, o, hi, lo, ov)) {
        publish(t, hi, lo, o, ov || row_flag);
        F4(p4 + t).x = o;
        mg().res[kPersistBlk / 2 + t] = r;
      } else {
        const double L2 = lse2_own(p.x, r);
        near(L2, &o);
        const double x = fma(-sh().a2ln2, L2, D(kAc, t));
        const float2 wv = split(fma(x, kLog2e, D(kWc, t)));
        publish(t, wv.x, wv.y, o, row_flag || over_tau(x));
        D(kLc, t) = L2;
        D(kLbo, t) = D(kLb, t);
        D(kLb, t) = x;
        point_at(F4(p4 + t), F(kCp, t), o, D(kKc, t), sh().c.alpha2);
        mg().res[kPersistBlk / 2 + t].z = 0.f;
      }
    }
    // settled by the last four warps while the weights travel (one thread still
    // handles one column; res is complete after the barrier)
    __syncthreads();
    if (threadIdx.x >= kResidentThreads - 128)
      for (int t = threadIdx.x - (kResidentThreads - 128); t < nc; t += 128) settle_col(t);
  }

  __device__ static bool iterate(bool lrow_valid, bool* over) {
    if (threadIdx.x == 0) ++sh().epoch;
    __syncthreads();
    if (lrow_valid)
      row_update_cached();
    else
      row_phase<false>();
    col_phase();
    if (A().g.nrb <= 64)
      merge_phase<4>();
    else if (A().g.nrb <= 128)
      merge_phase<8>();
    else
      merge_phase<kMergeSteps>();
    return stage_weights(over);
  }
  __device__ static bool fresh() {
    row_phase<true>();
    return true;
  }

  // u += eps log a, a = 1 (and for v, b); weights at the current epsilon,
  // published again under the same tag (`over` kept for CTAs that have not seen
  // it yet); a grid barrier separates them from the next staging.
  template <bool RESCALE>
  __device__ static __noinline__ bool absorb(double eps_old) {
    for (int t = threadIdx.x; t < nr(); t += kResidentThreads) {
      const double un = D(kU, t) + eps_old * D(kLa, t);
      D(kU, t) = un;
      D(kLa, t) = 0.0;
      if (RESCALE) D(kLao, t) = 0.0;
      fold_row(t);
    }
    for (int t = threadIdx.x; t < nc(); t += kResidentThreads) {
      const double vn = D(kV, t) + eps_old * D(kLb, t);
      D(kV, t) = vn;
      D(kLb, t) = 0.0;
      if (RESCALE) D(kLbo, t) = 0.0;
      fold_col(t);
      float2 w;
      split_weight(vn * sh().c.inv_eps * kLog2e, &w.x, &w.y, 0);
      publish(t, w.x, w.y, pc(t).x, !RESCALE);
    }
    return sync() && stage_weights(nullptr);
  }
  __device__ static bool start_stage(double eps_old, double eps) {
    set_coef(eps);
    reset_gap();
    return absorb<true>(eps_old);
  }
  __device__ static bool absorb_now(double eps) { return absorb<false>(eps); }
  __device__ static bool start_refine(double eps) {
    set_coef(eps);
    fold_all();
    for (int t = threadIdx.x; t < nc(); t += kResidentThreads)
      publish(t, A().V.wcol[j0() + t], A().V.wcol_lo[j0() + t], 0.f, false);
    return sync() && stage_weights(nullptr);
  }
  __device__ static bool resume(double eps) {
    set_coef(eps);
    fold_all();
    return stage_weights(nullptr);
  }
  // State of the rows and columns for the next launch, or for the outputs.
  __device__ static __noinline__ bool save(bool done) {
    __syncthreads();
    for (int t = threadIdx.x; t < nr(); t += kResidentThreads) {
      A().V.u[r0() + t] = D(kU, t);
      A().V.la[r0() + t] = D(kLa, t);
      reinterpret_cast<float*>(A().V.rowc)[r0() + t] = pr(t).x;
    }
    for (int t = threadIdx.x; t < nc(); t += kResidentThreads) {
      A().V.v[j0() + t] = D(kV, t);
      A().V.lb[j0() + t] = D(kLb, t);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) A().ctl->epoch = (int)sh().epoch;
    if (!done) return true;
    if (!sync()) return false;   // nobody polls the offset words any more
    for (int t = threadIdx.x; t < nc(); t += kResidentThreads) {
      A().V.wcol[j0() + t] = F(kWhi, j0() + t);
      A().V.wcol_lo[j0() + t] = F(kWlo, j0() + t);
    }
    return true;
  }

  // Sums over D(kEx, 4 t + k) of the rows (warps with rows(w)) or columns into this
  // CTA's place in V.red; ex holds rows first.
  template <int NQ>
  __device__ static void cta_sums(const int (&slot)[NQ], const bool (&of_rows)[NQ]) {
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < NQ; ++q)
      if (w == q) {
        double t = 0.0;
        const int a = of_rows[q] ? 0 : nr(), e = of_rows[q] ? nr() : nr() + nc();
        for (int k = a + lane; k < e; k += 32) t += D(kEx, 4 * k + slot[q]);
        t = warp_sum(t);
        if (lane == 0) A().V.red[blockIdx.x * kNq + q] = t;
      }
  }

  // The exponentials of all owned points one per thread: their FP64 chains run
  // side by side.
  __device__ static __noinline__ bool stage_test(bool* go_on) {
    const int n = nr() + nc();
    for (int k = threadIdx.x; k < 3 * n; k += kResidentThreads) {
      const int p = k / 3, f = k % 3;
      const bool row = p < nr();
      const int t = row ? p : p - nr();
      const double x = f == 0 ? (row ? D(kU, t) : D(kV, t)) * sh().c.inv_eps
                              : f == 1 ? (row ? D(kLa, t) : D(kLb, t)) : (row ? D(kLao, t) : D(kLbo, t));
      D(kEx, 4 * p + f) = exp(x);
    }
    __syncthreads();
    for (int p = threadIdx.x; p < n; p += kResidentThreads) {
      const double e = D(kEx, 4 * p), ta = D(kEx, 4 * p + 1) * e, d = ta - D(kEx, 4 * p + 2) * e;
      D(kEx, 4 * p) = d * d;
      D(kEx, 4 * p + 1) = ta * ta;
    }
    cta_sums<4>({0, 1, 0, 1}, {true, true, false, false});
    if (!reduce_ctas<4>()) return false;
    return stage_decision(go_on);
  }

  __device__ static __noinline__ bool gap_test(double sumk, bool* go_on, bool* nan) {
    const Coef& c = sh().c;
    const int n = nr() + nc();
    auto point = [&](int p, double* t, double* la_, double* ue) {
      if (p < nr()) {
        *la_ = D(kLa, p);
        *ue = D(kU, p) * c.inv_eps;
        *t = *la_ + *ue + D(kLr, p) * kLn2 - c.logJ;
      } else {
        *la_ = D(kLb, p - nr());
        *ue = D(kV, p - nr()) * c.inv_eps;
        *t = *la_ + *ue + D(kLc, p - nr()) * kLn2 - c.logI;
      }
    };
    for (int k = threadIdx.x; k < 2 * n; k += kResidentThreads) {
      const int p = k >> 1;
      double t, l, ue;
      point(p, &t, &l, &ue);
      D(kEx, 4 * p + (k & 1)) = exp(k & 1 ? -c.eps * (l + ue) / (p < nr() ? c.lambda1 : c.lambda2) : t);
    }
    __syncthreads();
    for (int p = threadIdx.x; p < n; p += kResidentThreads) {
      const bool row = p < nr();
      double t, l, ue, x, f, conj;
      point(p, &t, &l, &ue);
      const double pp = row ? A().V.p[r0() + p] : c.q, lp = row ? D(kLogp, p) : c.logq, lam = row ? c.lambda1 : c.lambda2;
      x = D(kEx, 4 * p);
      if (x > 0.0 && fabs(t) < 700.0 && fabs(l) < 700.0 && fabs(ue) < 700.0 && fabs(l + ue) < 700.0 && pp > 0.0) {
        f = x * (t - lp) - x + pp;
        conj = lam * pp * (D(kEx, 4 * p + 1) - 1.0);
      } else {
        gap_terms(t, l, ue, pp, lp, lam, c.eps, &x, &f, &conj);
      }
      const double ub = (row ? D(kU, p) : D(kV, p - nr())) + c.eps * l;
      D(kEx, 4 * p) = lam * f + conj + ub * x;
      D(kEx, 4 * p + 1) = f;
      D(kEx, 4 * p + 2) = ub * x;
      D(kEx, 4 * p + 3) = x;
    }
    cta_sums<7>({0, 0, 1, 1, 2, 2, 3}, {true, false, true, false, true, false, true});
    if (!reduce_ctas<7>()) return false;
    return gap_decision(sumk, go_on, nan);
  }

  __device__ static __noinline__ bool sum_exp(double* out) {
    float h = 0.f, l = 0.f;
    for (int64_t k = threadIdx.x; k < (int64_t)nr() * nv(); k += kResidentThreads) {
      const float4 cc = F4(kC4 + (int)k);
      const float k2 = sh().c.kappa2;
      df_add(h, l, (ex2(-k2 * cc.x) + ex2(-k2 * cc.y)) + (ex2(-k2 * cc.z) + ex2(-k2 * cc.w)), 0.f);
    }
    return total_pairs(h, l, out);
  }

  __device__ static __noinline__ bool mean_growth() {
    for (int t = threadIdx.x; t < nr(); t += kResidentThreads) D(kEx, 4 * t) = A().V.p[r0() + t];
    cta_sums<1>({0}, {true});
    if (!reduce_ctas<1>()) return false;
    return publish_mean();
  }
};

template <bool GAP>
__global__ void __launch_bounds__(kResidentThreads, 1) resident_kernel(const __grid_constant__ PersistArgs A, int rows_cap, int cols_cap) {
  PersistBase::begin(A);
  Resident p(rows_cap, cols_cap);
  persist_run<GAP>(p);
}

}  // namespace wotg
