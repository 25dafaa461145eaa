// wotg_persist.cuh — a whole materialised-cost solve in one persistent kernel.
//
// Every CTA owns a contiguous block of rows and of columns (their FP64 state,
// merges and updates) and takes its share of the column pass; an iteration is
//   row phase      a warp per owned row: the online LSE of the row (row_lse),
//                  merged as FP32 pairs; then a thread per row: log2 and the
//                  FP64 a-update                                        | grid barrier
//   column phase   a warp per (128 columns, row block): col_lse partials  | grid barrier
//   merge phase    a warp per owned float4 column: its row blocks' partials
//                  merged as FP32 pairs; then a thread per column: log2 and
//                  the FP64 b-update                                    | grid barrier
// and the stages, batches, absorptions, stage-exit tests and duality-gap tests
// of the reference run in the same kernel: every CTA sums the same partial sums
// in the same order and so takes the same decisions.
//
// What bounds it. At the sizes of a day pair (up to a few 1e7 entries, C in L2)
// an iteration used to be four launches of 2 to 37 us each, and most of that was
// FP64: one instruction holds a sub-partition's FP64 unit 64 cycles
// (wotg_df.cuh), and a row's merge and update took some 85 of them on one lane.
// Here the merges are FP32 pairs, the updates take one instruction for up to 32
// rows, and a grid barrier (2300 cycles) stands where a launch did.
//
// The element arithmetic, its order within a lane and the row blocks of the
// column pass are those of the standalone passes, so the sums of exponentials
// are the same bits whatever the grid.
//
// Barriers: one CTA per SM, launched cooperatively, so that all are resident;
// each wait is bounded and a CTA that gives up raises *err, on which the others
// give up as well. A launch runs at most `budget` iterations and leaves its
// state in PersistCtl, so that no launch is long.
#pragma once

#include <stddef.h>

#include "wotg_barrier.cuh"
#include "wotg_df.cuh"
#include "wotg_state.cuh"

namespace wotg {

constexpr int kPersistThreads = 512;
constexpr int kPersistWarps = kPersistThreads / 32;
constexpr int kPersistBlk = 512;      // rows (columns) of a CTA merged per round
constexpr int kScalings = 5;          // n_scalings of the duality-gap solver (optimal_transport.py:105)
constexpr uint32_t kBarrierTries = 10000000;  // polls of about 0.3 us

enum PersistMode : int { kModeGap = 0, kModeFixed = 1, kModeRefine = 2 };
enum PersistStatus : int { kRunning = 0, kConverged = 1, kMaxIter = 2, kNonfinite = 3 };

struct PersistCtl {
  double eps, q, sumk;            // current epsilon, mean(p), sum exp(-C/eps) / (I J) at the final stage
  double gap_num, gap_den;        // the last relative gap as a quotient
  long long it, checks, absorptions;
  int stage, status, lrow_valid, started, since, index, epoch;
  int batch;                      // iterations done of a batch that the launch ended in
  unsigned long long bar;         // grid barrier: arrivals and flags (PersistBase::sync); zeroed per launch
  int err, pad2_;                 // zeroed per launch
};

struct PersistArgs {
  const float* C;
  Geom g;
  Vecs V;
  PersistCtl* ctl;
  double epsilon, lambda1, lambda2, epsilon0, tau, tolerance, max_iter, cost_scale;
  double scale_factor;            // exp(-log(epsilon) / kScalings)
  int batch_size, scaling_iter, inner_iter_max, extra_iter, n_iter, mode;
  long long budget;               // iterations of this launch
  int wfloats;                    // streamed: floats of a weight vector kept in shared memory, 0: none are
};

// The solver's control state during a launch; thread 0 of every CTA keeps the
// same copy in shared memory (in registers it would crowd out the passes).
struct RunState {
  double eps, sumk;
  long long it, checks, absorptions, used;
  int stage, status, lrow_valid, since, index, stage_done, batch;
};

// A virtual CTA's tiles in a tensor-core half-step (wotg_tc_persist.cuh).
struct TcStretch {
  int n, t, q, nseg, nq;
};

// A CTA's working state, at the start of its dynamic shared memory (hdr()). The
// variants are stateless: what they keep between phases is here, and not in an
// object on the stack, because the phases are functions of their own and a
// stack access after a grid barrier (whose acquire empties L1) is a trip to L2.
struct PersistShared {
  float2 pairs[32];               // a pair sum per warp
  double sums[8][kNq];
  double tot[kNq];
  Coef c;
  double a1ln2, a1logj, ku, a2ln2, bconst, kv, iel2;   // folded update coefficients
  double consts[4];               // log I, log J, log q, log tau
  double dx, dy;                  // 1 / I, 1 / J
  float a1h, a1l, a2h, a2l;       // alpha1, alpha2 as pairs
  RunState rs;
  BarrierSeen seen;               // its flags: absorption; rows to recompute
  int flagged, flagged2;          // raised at the last barrier that took them
  int ok, decision, ticket;
  int r0, r1, j0, j1, c0, c1;     // owned rows, columns, float4 columns
  int row_flag, over_flag;        // a row to recompute / a scaling above tau, since the half-step began
  int row_ok, col_ok;             // on-the-fly: offsets of the side exist for this epsilon
  int jbase[2], segbase[2];       // on-the-fly, per half: tiles and segments of the half-steps before
  int copied[2], copied_seg[2];   // and the producer's own count
  TcStretch stretch[2][2];        // on-the-fly: of either side, per half
  unsigned int epoch;             // resident: the iteration
  int row_over;                   // resident: an owned row is above tau
  int off[34];                    // resident: its arrays' places
};

// What the variants that merge sums themselves keep beside it.
struct MergeShared {
  float4 tab[kLogTable];          // log2_pair's table
  float4 res[kPersistBlk];        // merged (m, h, l) per row or column of a round
};

// The header of dynamic shared memory: the state, a copy of the kernel's arguments
// (a parameter reached by reference from a function would be a load through L2)
// and, where a variant merges, MergeShared.
constexpr int kPersistArgBytes = 640;
struct PersistHeader {
  PersistShared sh;
  alignas(16) unsigned char args[kPersistArgBytes];
  alignas(16) MergeShared mg;     // streamed and resident variants only
};
constexpr size_t kMergeHeaderBytes = (sizeof(PersistHeader) + 1023) & ~size_t(1023);
constexpr size_t kPlainHeaderBytes = (offsetof(PersistHeader, mg) + 1023) & ~size_t(1023);

extern __shared__ __align__(1024) unsigned char persist_smem[];
__device__ __forceinline__ PersistHeader& persist_hdr() { return *reinterpret_cast<PersistHeader*>(persist_smem); }

// Weight and offset of a point from FP64: as split_weight / grid_value, with the
// rounding to the 2^-14 grid by one FP64 addition of 1.5 * 2^38 (the same
// nearest-even value) for |w| < 2^10.
__device__ __forceinline__ bool below_1024(double w) { return (__double2hiint(w) & 0x7FFFFFFF) < 0x40900000; }
constexpr double kGridMagic = 412316860416.0;   // 1.5 * 2^38: ulp 2^-14

__device__ __forceinline__ float2 split_pair(double w) {
  if (below_1024(w)) {
    const double h = (w + kGridMagic) - kGridMagic;
    return make_float2((float)h, (float)(w - h));
  }
  float2 r;
  split_weight(w, &r.x, &r.y, 0);
  return r;
}
__device__ __forceinline__ float grid_near(double x) {
  return below_1024(x) ? (float)((x + kGridMagic) - kGridMagic) : grid_value(x);
}

struct PersistBase {
  __device__ static __forceinline__ PersistShared& sh() { return persist_hdr().sh; }
  __device__ static __forceinline__ MergeShared& mg() { return persist_hdr().mg; }
  __device__ static __forceinline__ const PersistArgs& A() {
    return *reinterpret_cast<const PersistArgs*>(persist_hdr().args);
  }

  // Copies the arguments, resets the state; a CTA's shares of rows and columns.
  template <class Args>
  __device__ static void begin(const Args& args) {
    static_assert(sizeof(Args) % 4 == 0 && sizeof(Args) <= kPersistArgBytes, "copied by words into the header");
    for (int k = threadIdx.x; k < (int)(sizeof(Args) / 4); k += blockDim.x)
      reinterpret_cast<uint32_t*>(persist_hdr().args)[k] = reinterpret_cast<const uint32_t*>(&args)[k];
    __syncthreads();
    if (threadIdx.x == 0) {
      PersistShared& s = sh();
      const Geom& g = A().g;
      const int n = gridDim.x, b = blockIdx.x;
      s.seen = BarrierSeen{(unsigned int)n, 0, 0};
      s.ok = 1;
      s.r0 = (int)(g.I * b / n);
      s.r1 = (int)(g.I * (b + 1) / n);
      s.j0 = (int)(g.J * b / n);
      s.j1 = (int)(g.J * (b + 1) / n);
      s.jbase[0] = s.jbase[1] = s.segbase[0] = s.segbase[1] = 0;
      s.copied[0] = s.copied[1] = s.copied_seg[0] = s.copied_seg[1] = 0;
    }
    __syncthreads();
  }
  __device__ static void fill_table() {
    for (int i = threadIdx.x; i < kLogTable; i += blockDim.x) mg().tab[i] = log_table_entry(i);
  }

  // All CTAs arrive; with `take`, `flag` and `flag2` are or-ed over the CTAs into
  // sh().flagged and sh().flagged2 (wotg_barrier.cuh). The counts last a launch: its
  // budget keeps the flags below 2^20 (barriers that take flags: one per iteration
  // streamed, up to four on the fly), and the arrivals, at most nine barriers per
  // iteration with its tests, below 2^24.
  __device__ static __noinline__ bool barrier(bool flag, bool flag2, bool take) {
    __syncthreads();
    if (threadIdx.x == 0) {
      PersistShared& s = sh();
      PersistCtl* ctl = A().ctl;
      asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&ctl->bar), "l"(barrier_arrival(flag, flag2))
                   : "memory");
      unsigned long long v = 0;
      bool done = false;
      for (uint32_t t = 0; t < kBarrierTries; ++t) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(&ctl->bar) : "memory");
        if (barrier_complete(v, s.seen)) {
          done = true;
          break;
        }
        if ((t & 255) == 255 && *(volatile int*)&ctl->err) break;
      }
      if (!done) {
        atomicExch(&ctl->err, 1);
        s.ok = 0;
      }
      bool f, f2;
      barrier_pass(v, gridDim.x, take, s.seen, &f, &f2);
      s.flagged = f;
      s.flagged2 = f2;
    }
    __syncthreads();
    return sh().ok != 0;
  }
  // A barrier without flags.
  __device__ static __forceinline__ bool sync() { return barrier(false, false, false); }
  // One whose flags are taken. No two in a row, but where the second only adds to the
  // first's `flagged` (TcPersist::side).
  __device__ static __forceinline__ bool sync(bool flag, bool* flagged, bool flag2 = false, bool* flagged2 = nullptr) {
    const bool ok = barrier(flag, flag2, true);
    *flagged = sh().flagged != 0;
    if (flagged2) *flagged2 = sh().flagged2 != 0;
    return ok;
  }

  // Coefficients of the updates at `eps` (make_coef's, its divisions one per lane).
  __device__ static void set_coef(double eps) {
    __syncthreads();
    if (threadIdx.x < 32) {
      const int l = threadIdx.x;
      const double num = l == 1 ? A().lambda1 : l == 2 ? A().lambda2 : l == 5 ? A().cost_scale : 1.0;
      const double den = l == 1 || l == 3 ? A().lambda1 + eps : l == 2 || l == 4 ? A().lambda2 + eps : eps;
      const double x = num / den;
      Coef c;
      c.eps = eps;
      c.inv_eps = __shfl_sync(0xffffffffu, x, 0);
      c.alpha1 = __shfl_sync(0xffffffffu, x, 1);
      c.alpha2 = __shfl_sync(0xffffffffu, x, 2);
      c.inv_l1e = __shfl_sync(0xffffffffu, x, 3);
      c.inv_l2e = __shfl_sync(0xffffffffu, x, 4);
      c.kappa = __shfl_sync(0xffffffffu, x, 5);
      if (l == 0) {
        c.lambda1 = A().lambda1;
        c.lambda2 = A().lambda2;
        c.logI = sh().consts[0];
        c.logJ = sh().consts[1];
        c.logq = sh().consts[2];
        c.q = A().ctl->q;
        coef_kappa2(c);
        c.ltau_lo = sh().consts[3] - 1e-9;
        c.ltau_hi = sh().consts[3] + 1e-9;
        sh().c = c;
        sh().a1ln2 = c.alpha1 * kLn2;
        sh().a1logj = c.alpha1 * c.logJ;
        sh().ku = -(c.alpha1 * c.inv_eps + c.inv_l1e);
        sh().a2ln2 = c.alpha2 * kLn2;
        sh().bconst = c.alpha2 * (c.logq + c.logI);
        sh().kv = -(c.alpha2 * c.inv_eps + c.inv_l2e);
        sh().iel2 = c.inv_eps * kLog2e;
        sh().a1h = (float)c.alpha1;
        sh().a1l = (float)(c.alpha1 - (double)sh().a1h);
        sh().a2h = (float)c.alpha2;
        sh().a2l = (float)(c.alpha2 - (double)sh().a2h);
      }
    }
    __syncthreads();
  }

  __device__ static __forceinline__ bool over_tau(double l) {
    if (l < sh().c.ltau_lo) return false;
    if (l > sh().c.ltau_hi) return INFINITY > A().tau;
    return exp(l) > A().tau;
  }

  // Cross-CTA sums of the NQ values that every CTA has written to its place in
  // V.red: one barrier, then every CTA adds them in the same order into sh().tot.
  template <int NQ>
  __device__ static bool reduce_ctas() {
    if (!sync()) return false;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w < NQ) {
      double t = 0.0;
      for (int b = lane; b < (int)gridDim.x; b += 32) t += A().V.red[b * kNq + w];
      t = warp_sum(t);
      if (lane == 0) sh().tot[w] = t;
    }
    __syncthreads();
    return true;
  }

  // Sum over all threads of the pairs h + l, over I J.
  __device__ static bool total_pairs(float h, float l, double* out) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float h2 = __shfl_xor_sync(0xffffffffu, h, o), l2 = __shfl_xor_sync(0xffffffffu, l, o);
      df_add(h, l, h2, l2);
    }
    __syncthreads();
    if (lane == 0) sh().pairs[w] = make_float2(h, l);
    __syncthreads();
    if (w == 0) {
      const float2 r = lane < (int)(blockDim.x >> 5) ? sh().pairs[lane] : make_float2(0.f, 0.f);
      const double t = warp_sum((double)r.x + (double)r.y);
      if (lane == 0) A().V.red[blockIdx.x * kNq] = t;
    }
    if (!reduce_ctas<1>()) return false;
    *out = sh().tot[0] / ((double)A().g.I * (double)A().g.J);
    return true;
  }

  // Stage-exit decision from |a~ - old|^2, |a~|^2 and the same of b in sh().tot.
  __device__ static bool stage_decision(bool* go_on) {
    if (threadIdx.x < 32) {
      // ga = sqrt(h0) / (1 + sqrt(h1)), gb likewise; Python's max (the first unless
      // the second is larger) and the comparison with 1e-6 as products
      const double r = sqrt(sh().tot[threadIdx.x & 3]);
      const double na = __shfl_sync(0xffffffffu, r, 0), nb = __shfl_sync(0xffffffffu, r, 2);
      const double da = 1.0 + __shfl_sync(0xffffffffu, r, 1), db = 1.0 + __shfl_sync(0xffffffffu, r, 3);
      const bool b = nb * da > na * db;
      const double num = b ? nb : na, den = b ? db : da;
      if (threadIdx.x == 0) {
        sh().decision = num > 1e-6 * den;
        if (blockIdx.x == 0) {
          A().ctl->gap_num = num;
          A().ctl->gap_den = den;
        }
      }
    }
    __syncthreads();
    *go_on = sh().decision != 0;
    return true;
  }

  // Duality-gap decision from the sums of gap_test in sh().tot.
  __device__ static bool gap_decision(double sumk, bool* go_on, bool* nan) {
    if (threadIdx.x == 0) {
      const double* h = sh().tot;
      const Coef& c = sh().c;
      const double dx = sh().dx, dy = sh().dy;
      const double num = dx * h[0] + dy * h[1];
      const double pri = c.lambda1 * dx * h[2] + c.lambda2 * dy * h[3] + dx * h[4] + dy * h[5] +
                         c.eps * (sumk - dx * h[6]);
      const double den = fabs(pri);
      // gap = num / den, as a comparison (the quotient is formed once, on the host)
      const bool isnan_ = num != num || den != den || (num == 0.0 && den == 0.0) || (isinf(num) && isinf(den));
      sh().decision = isnan_ ? 2 : num > A().tolerance * den ? 1 : 0;
      if (blockIdx.x == 0) {
        A().ctl->gap_num = num;
        A().ctl->gap_den = den;
      }
    }
    __syncthreads();
    *go_on = sh().decision == 1;
    *nan = sh().decision == 2;
    return true;
  }

  // q = mean(p) from its sum, and the constants of the coefficients.
  __device__ static bool publish_mean() {
    if (threadIdx.x == 0 && blockIdx.x == 0) A().ctl->q = sh().tot[0] / (double)A().g.I;
    return sync();
  }
  __device__ static void constants() {
    if (threadIdx.x < 32) {
      const double x = threadIdx.x == 0 ? (double)A().g.I : threadIdx.x == 1 ? (double)A().g.J
                       : threadIdx.x == 2 ? *(volatile double*)&A().ctl->q : A().tau;
      const double y = log(x), z = 1.0 / x;
      if (threadIdx.x < 4) sh().consts[threadIdx.x] = y;
      if (threadIdx.x == 0) sh().dx = z;
      if (threadIdx.x == 1) sh().dy = z;
    }
  }
  __device__ static void reset_gap() {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      A().ctl->gap_num = INFINITY;
      A().ctl->gap_den = 1.0;
    }
  }
};

// A CTA's share of the O(I + J) work, state in global memory: rows [r0, r1),
// columns [j0, j1).
struct Owned : PersistBase {
  __device__ static __forceinline__ int r0() { return sh().r0; }
  __device__ static __forceinline__ int r1() { return sh().r1; }
  __device__ static __forceinline__ int j0() { return sh().j0; }
  __device__ static __forceinline__ int j1() { return sh().j1; }

  // Sums over all CTAs of per-thread values (threads 0..127 hold row terms,
  // 128..255 column terms, the others none): every thread ends with the totals
  // in sh().tot. One barrier.
  template <int NQ>
  __device__ static bool total(double (&acc)[NQ], bool any) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (w < 8) {
      if (__any_sync(0xffffffffu, any)) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) acc[q] = warp_sum(acc[q]);
      }
      if (lane == 0)
#pragma unroll
        for (int q = 0; q < NQ; ++q) sh().sums[w][q] = acc[q];
    }
    __syncthreads();
    if (threadIdx.x < NQ) {
      double t = 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k) t += sh().sums[k][threadIdx.x];
      A().V.red[blockIdx.x * kNq + threadIdx.x] = t;
    }
    return reduce_ctas<NQ>();
  }

  // Stage-exit test (optimal_transport.py:158-160) in the reference's expressions.
  __device__ static bool stage_test(bool* go_on) {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    bool any = false;
    const bool rows = threadIdx.x < 128;
    const double* u = rows ? A().V.u : A().V.v;
    const double* la = rows ? A().V.la : A().V.lb;
    const double* lo = rows ? A().V.la_old : A().V.lb_old;
    const int n0 = rows ? r0() : j0(), n1 = rows ? r1() : j1();
    if (threadIdx.x < 256) {
      double d2 = 0.0, a2 = 0.0;
      for (int k = n0 + (threadIdx.x & 127); k < n1; k += 128) {
        const double e = exp(u[k] * sh().c.inv_eps);
        const double ta = exp(la[k]) * e;
        const double d = ta - exp(lo[k]) * e;
        d2 += d * d;
        a2 += ta * ta;
        any = true;
      }
      acc[rows ? 0 : 2] = d2;
      acc[rows ? 1 : 3] = a2;
    }
    if (!total<4>(acc, any)) return false;
    return stage_decision(go_on);
  }

  // Duality-gap test in O(I + J) (see wotg_sinkhorn.cu) after a fresh row phase.
  // lcol(j): the column's log-sum-exp (natural).
  template <class Lcol>
  __device__ static bool gap_test_with(const Lcol& lcol, double sumk, bool* go_on, bool* nan) {
    double acc[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const Coef& c = sh().c;
    bool any = false;
    if (threadIdx.x < 128) {
      for (int i = r0() + threadIdx.x; i < r1(); i += 128) {
        const double ui = A().V.u[i], la = A().V.la[i];
        const double ue = ui * c.inv_eps, ub = ui + c.eps * la;
        double x, f, conj;
        gap_terms(la + ue + A().V.Lrow[i] - c.logJ, la, ue, A().V.p[i], A().V.logp[i], c.lambda1, c.eps, &x, &f, &conj);
        acc[0] += c.lambda1 * f + conj + ub * x;
        acc[2] += f;
        acc[4] += ub * x;
        acc[6] += x;
        any = true;
      }
    } else if (threadIdx.x < 256) {
      for (int j = j0() + threadIdx.x - 128; j < j1(); j += 128) {
        const double vj = A().V.v[j], lb = A().V.lb[j];
        const double ve = vj * c.inv_eps, vb = vj + c.eps * lb;
        double y, f, conj;
        gap_terms(lb + ve + lcol(j) - c.logI, lb, ve, c.q, c.logq, c.lambda2, c.eps, &y, &f, &conj);
        acc[1] += c.lambda2 * f + conj + vb * y;
        acc[3] += f;
        acc[5] += vb * y;
        any = true;
      }
    }
    if (!total<7>(acc, any)) return false;
    return gap_decision(sumk, go_on, nan);
  }

  // sum_ij exp(-kappa C_ij) / (I J) (the reference's sum of its _K).
  __device__ static bool sum_exp(double* out) {
    const int lane = threadIdx.x & 31;
    const float k2 = sh().c.kappa2;
    const int64_t nv = A().g.ldc >> 2;
    float h = 0.f, l = 0.f;
    for (int i = r0() + (threadIdx.x >> 5); i < r1(); i += (int)(blockDim.x >> 5)) {
      const float4* row = reinterpret_cast<const float4*>(A().C + (int64_t)i * A().g.ldc);
      for (int64_t k = lane; k < nv; k += 32) {
        const float4 cc = ld_stream(row + k);   // padding is +inf: exp2(-inf) = 0
        df_add(h, l, (ex2(-k2 * cc.x) + ex2(-k2 * cc.y)) + (ex2(-k2 * cc.z) + ex2(-k2 * cc.w)), 0.f);
      }
    }
    return total_pairs(h, l, out);
  }

  __device__ static bool mean_growth() {
    double acc[1] = {0.0};
    bool any = false;
    if (threadIdx.x < 128)
      for (int i = r0() + threadIdx.x; i < r1(); i += 128) {
        acc[0] += A().V.p[i];
        any = true;
      }
    if (!total<1>(acc, any)) return false;
    return publish_mean();
  }
};

// Costs of more bytes than stay in L2 are loaded evict-first, and each warp's lines are
// asked for kAhead chunks before their loads: 100 iterations at 20000 x 25000 82 -> 72 ms,
// 40000 x 9000 66 -> 54, 6000 x 8000 (192 MB) 9.7 -> 7.8; at 4001 x 5003 (80 MB) it would
// take 21.3 ms for a solve instead of 18.3.
constexpr int64_t kKeptBytes = 100000000;
constexpr int kAhead = 4;
__device__ __forceinline__ void prefetch_line(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void async16(void* to, const void* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from)
               : "memory");
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The streamed variant: C read from L2 or HBM in both passes, the FP64 state in
// global memory (own rows and columns only), any size.
//
// What bounds it: the instructions per element. A pass over 4001 x 5003 took 44000
// cycles of each SM for its rows and 34000 for its columns, of which the exponentials
// are 5400, whether its costs came ahead of use through a ring in shared memory or
// not; 23000 and 24000 with the arithmetic on packed FP32 pairs (wotg_state.cuh) and
// the weights and their low parts, twice the bytes of the costs, in shared memory
// (22.3 -> 18.4 ms a solve). Two rows per warp, or 24 or 32 warps, were no faster.
template <bool KEPT>
struct Streamed : Owned {
  __device__ static __forceinline__ float* wstage() { return reinterpret_cast<float*>(persist_smem + kMergeHeaderBytes); }
  // Copies a pass's weights and their low parts (n floats each) to shared memory.
  __device__ static __forceinline__ void stage(const float* w, const float* wl, int n) {
    if (!A().wfloats) return;
    float* to = wstage();
    for (int k = threadIdx.x * 4; k < n; k += kPersistThreads * 4) {
      if (k + 4 <= n) {
        async16(to + k, w + k);
        async16(to + A().wfloats + k, wl + k);
      } else {
        for (int q = k; q < n; ++q) {
          to[q] = w[q];
          to[A().wfloats + q] = wl[q];
        }
      }
    }
    async_commit();
    async_wait<0>();
  }
  __device__ static __forceinline__ int c0() { return sh().c0; }
  __device__ static __forceinline__ int c1() { return sh().c1; }
  // Offsets on the weight grid: the rows' in rowc's memory, free during the solve, the
  // columns' in Lcol's. The columns' base-2 log-sum-exps stay FP64 for the gap test: in
  // the final stage they take the place of the old scalings, which its tests don't read.
  __device__ static __forceinline__ float* orow() { return reinterpret_cast<float*>(A().V.rowc); }
  __device__ static __forceinline__ float* ocol() { return reinterpret_cast<float*>(A().V.Lcol); }

  __device__ Streamed() {
    fill_table();
    if (threadIdx.x == 0) {
      PersistShared& s = sh();
      const Geom& g = A().g;
      const int64_t nv = g.ldc >> 2;
      s.c0 = (int)(nv * blockIdx.x / gridDim.x);
      s.c1 = (int)(nv * (blockIdx.x + 1) / gridDim.x);
      s.j0 = (int)min((int64_t)s.c0 * 4, g.J);
      s.j1 = (int)min((int64_t)s.c1 * 4, g.J);
    }
    __syncthreads();
  }

  // The reference's a-update (optimal_transport.py:133) of row i from its base-2
  // log-sum-exp; true when a_i > tau.
  __device__ static __forceinline__ bool update_row(int64_t i, double L2) {
    const double ui = A().V.u[i];
    const double la = fma(-sh().a1ln2, L2, fma(sh().c.alpha1, A().V.logp[i], fma(ui, sh().ku, sh().a1logj)));
    A().V.la_old[i] = A().V.la[i];
    A().V.la[i] = la;
    const float2 w = split_pair(fma(la, kLog2e, ui * sh().iel2));
    A().V.wrow[i] = w.x;
    A().V.wrow_lo[i] = w.y;
    return over_tau(la);
  }
  __device__ static __forceinline__ bool update_col(int64_t j, double L2) {
    const double vj = A().V.v[j];
    const double lb = fma(-sh().a2ln2, L2, fma(vj, sh().kv, sh().bconst));
    A().V.lb_old[j] = sh().rs.stage == kScalings ? L2 : A().V.lb[j];
    A().V.lb[j] = lb;
    const float2 w = split_pair(fma(lb, kLog2e, vj * sh().iel2));
    A().V.wcol[j] = w.x;
    A().V.wcol_lo[j] = w.y;
    return over_tau(lb);
  }

  // Row sums of rows [b, e) into res, a warp per row.
  template <bool STAGED>
  __device__ static __noinline__ void row_sums(int b, int e) {
    const int lane = threadIdx.x & 31, nv = (int)(A().g.ldc >> 2);
    const float4* const w4 = reinterpret_cast<const float4*>(STAGED ? wstage() : A().V.wcol);
    const float4* const wl4 = reinterpret_cast<const float4*>(STAGED ? wstage() + A().wfloats : A().V.wcol_lo);
    for (int i = b + (threadIdx.x >> 5); i < e; i += kPersistWarps) {
      float m, s, cmp, h, l;
      const float4* row = reinterpret_cast<const float4*>(A().C + (int64_t)i * A().g.ldc);
      // a 128-byte line per lane of the chunk kAhead chunks on, or of the warp's next row
      const bool more = i + kPersistWarps < e;
      auto ahead = [row, nv, lane, more](int k) {
        int q = k + 128 * kAhead + lane * 8;
        const float4* p = row + q;
        if (q >= nv) {
          q -= nv;
          p = row + (int64_t)kPersistWarps * nv + q;
          if (!more || q >= nv) return;
        }
        if (lane < 16) prefetch_line(p);
      };
      auto ask = [&ahead](int k) {
        if constexpr (!KEPT) ahead(k);
      };
      row_lse<true>([row](int k) { return KEPT ? ld_stream(row + k) : ld_once(row + k); }, [w4](int k) { return w4[k]; },
                    [wl4](int k) { return wl4[k]; }, nv, lane, orow()[i], sh().c.kappa2, sh().c.kappa2_lo, m, s, cmp, ask);
      two_sum(s, -cmp, h, l);
      df_merge_lanes<16, 1>(m, h, l);
      if (lane == 0) mg().res[i - b] = make_float4(m, h, l, 0.f);
    }
  }

  // Row phase. FRESH: the row sums with the current b only (a gap check), kept
  // for the a-update of the next iteration.
  template <bool FRESH>
  __device__ static bool row_phase() {
    bool over = false;
    for (int b = r0(); b < r1(); b += kPersistBlk) {
      const int e = min(r1(), b + kPersistBlk);
      stage(A().V.wcol, A().V.wcol_lo, (int)A().g.ldc);
      __syncthreads();
      if (A().wfloats)
        row_sums<true>(b, e);
      else
        row_sums<false>(b, e);
      __syncthreads();
      for (int i = b + threadIdx.x; i < e; i += kPersistThreads) {
        const float4 r = mg().res[i - b];
        const double L2 = lse2_pair(orow()[i], r.x, r.y, r.z, mg().tab);
        orow()[i] = fabs(L2) < 1e30 ? grid_near(L2) : 0.f;
        if (FRESH)
          A().V.Lrow[i] = L2 * kLn2;
        else
          over |= update_row(i, L2);
      }
    }
    return over;
  }

  // The a-update from the row sums of the preceding check.
  __device__ static bool row_update_cached() {
    bool over = false;
    for (int i = r0() + threadIdx.x; i < r1(); i += kPersistThreads) over |= update_row(i, A().V.Lrow[i] * kLog2e);
    return over;
  }

  // Column phase: partials of (float4 column, row block) at part[(c4 nrb + r) 4 + q], a
  // warp per unit (row block, 128 columns).
  template <bool STAGED>
  __device__ static __noinline__ void col_sums() {
    const int lane = threadIdx.x & 31;
    const int64_t ld4 = A().g.ldc >> 2;
    const int nv = (int)ld4, ncg = (nv + 31) >> 5, rows_per = (int)A().g.rows_per, I = (int)A().g.I;
    // the CTA's units: about the rows it has in the row phase, so that it reads them
    // through the same die's L2 (any other order has each die keep its own copy)
    const int64_t all = (int64_t)ncg * A().g.nrb;
    const int units = (int)(all * (blockIdx.x + 1) / gridDim.x), first = (int)(all * blockIdx.x / gridDim.x) + (threadIdx.x >> 5);
    const float* const w = STAGED ? wstage() : A().V.wrow;
    const float* const wl = STAGED ? wstage() + A().wfloats : A().V.wrow_lo;
    for (int u = first; u < units; u += kPersistWarps) {
      const int r = u / ncg, c4 = (u - r * ncg) * 32 + lane;
      if (c4 >= nv) continue;
      float o[4], m[4], s[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) o[q] = c4 * 4 + q < A().g.J ? ocol()[c4 * 4 + q] : 0.f;
      const int a = r * rows_per;
      const float4* col = reinterpret_cast<const float4*>(A().C) + c4;
      // as for the rows: four lines of each of the four rows kAhead chunks on, or of the
      // warp's next unit
      const int last = min(I, a + rows_per), u2 = u + kPersistWarps, r2 = u2 / ncg;
      const int line = (lane & 3) * 8, skew = lane >> 2;
      auto ahead = [=](int i) {
        int q = i + kColRowChunk * kAhead + skew, c = (u - r * ncg) * 32 + line;
        if (q >= last) {
          if (u2 >= units) return;
          q = r2 * rows_per + (q - last);
          c = (u2 - r2 * ncg) * 32 + line;
        }
        if (lane < 16 && q < I && c < nv) prefetch_line(reinterpret_cast<const float4*>(A().C) + q * ld4 + c);
      };
      auto ask = [&ahead](int i) {
        if constexpr (!KEPT) ahead(i);
      };
      col_lse<true>([=](int i) { return KEPT ? ld_stream(col + i * ld4) : ld_once(col + i * ld4); }, [w](int i) { return w[i]; },
                    [wl](int i) { return wl[i]; }, a, last, o, sh().c.kappa2, sh().c.kappa2_lo, m, s, ask);
      float4* out = reinterpret_cast<float4*>(A().V.part + ((int64_t)c4 * A().g.nrb + r) * 4);
      out[0] = make_float4(m[0], s[0], m[1], s[1]);
      out[1] = make_float4(m[2], s[2], m[3], s[3]);
    }
  }
  __device__ static void col_phase() {
    stage(A().V.wrow, A().V.wrow_lo, (int)A().g.I);
    __syncthreads();
    if (A().wfloats)
      col_sums<true>();
    else
      col_sums<false>();
  }

  // Merge phase: eight lanes per column over its row blocks, then the b-update.
  __device__ static bool merge_phase() {
    const int lane = threadIdx.x & 31, q = lane & 3, rl = lane >> 2;
    constexpr int kCols4 = kPersistBlk / 4;
    bool over = false;
    for (int b = c0(); b < c1(); b += kCols4) {
      const int e = min(c1(), b + kCols4);
      for (int c4 = b + (threadIdx.x >> 5); c4 < e; c4 += kPersistWarps) {
        const float2* p = A().V.part + (int64_t)c4 * A().g.nrb * 4 + q;
        float m = kNegBig, h = 0.f, l = 0.f;
#pragma unroll 4
        for (int r = rl; r < A().g.nrb; r += 8) m = fmaxf(m, p[(int64_t)r * 4].x);
#pragma unroll
        for (int o = 16; o >= 4; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
#pragma unroll 4
        for (int r = rl; r < A().g.nrb; r += 8) {
          const float2 ps = p[(int64_t)r * 4];
          const float f = ex2(ps.x - m);
          const float x = __fmul_rn(ps.y, f);
          df_add(h, l, x, __fmaf_rn(ps.y, f, -x));
        }
#pragma unroll
        for (int o = 16; o >= 4; o >>= 1) {
          const float h2 = __shfl_xor_sync(0xffffffffu, h, o), l2 = __shfl_xor_sync(0xffffffffu, l, o);
          df_add(h, l, h2, l2);
        }
        if (rl == 0) mg().res[(c4 - b) * 4 + q] = make_float4(m, h, l, 0.f);
      }
      __syncthreads();
      for (int t = threadIdx.x; t < (e - b) * 4; t += kPersistThreads) {
        const int j = b * 4 + t;
        if (j >= A().g.J) break;
        const float4 r = mg().res[t];
        const double L2 = lse2_pair(ocol()[j], r.x, r.y, r.z, mg().tab);
        ocol()[j] = fabs(L2) < 1e30 ? grid_near(L2) : 0.f;
        over |= update_col(j, L2);
      }
      __syncthreads();
    }
    return over;
  }

  // u += eps log a, a = 1 (and for v, b): tau-absorption (optimal_transport.py:
  // 137-141), or with RESCALE the start of a stage (:118-125), whose weights
  // are for the new epsilon. The caller separates it from the next pass.
  template <bool RESCALE>
  __device__ static void absorb(double eps_old) {
    for (int i = r0() + threadIdx.x; i < r1(); i += kPersistThreads) {
      const double un = A().V.u[i] + eps_old * A().V.la[i];
      A().V.u[i] = un;
      A().V.la[i] = 0.0;
      if (RESCALE) A().V.la_old[i] = 0.0;
      split_weight(un * sh().c.inv_eps * kLog2e, A().V.wrow, A().V.wrow_lo, i);
    }
    for (int j = j0() + threadIdx.x; j < j1(); j += kPersistThreads) {
      const double vn = A().V.v[j] + eps_old * A().V.lb[j];
      A().V.v[j] = vn;
      A().V.lb[j] = 0.0;
      if (RESCALE) A().V.lb_old[j] = 0.0;
      split_weight(vn * sh().c.inv_eps * kLog2e, A().V.wcol, A().V.wcol_lo, j);
    }
  }

  // One iteration; *absorb_now when max(a, b) > tau.
  __device__ static bool iterate(bool lrow_valid, bool* absorb_now) {
    bool over = lrow_valid ? row_update_cached() : row_phase<false>();
    if (!sync()) return false;
    col_phase();
    if (!sync()) return false;
    over |= merge_phase();
    over = __syncthreads_or(over);
    return sync(over, absorb_now);
  }

  __device__ static bool gap_test(double sumk, bool* go_on, bool* nan) {
    const double* l2 = A().V.lb_old;
    return gap_test_with([l2](int j) { return l2[j] * kLn2; }, sumk, go_on, nan);
  }

  // Absorbs with the old epsilon and starts a stage at `eps`.
  __device__ static bool start_stage(double eps_old, double eps) {
    set_coef(eps);
    reset_gap();
    absorb<true>(eps_old);
    return sync();
  }
  __device__ static bool absorb_now(double eps) {
    absorb<false>(eps);
    return sync();
  }
  __device__ static bool fresh() {
    row_phase<true>();
    __syncthreads();
    return true;
  }
  // Refinement starts from loaded potentials and weights.
  __device__ static bool start_refine(double eps) {
    set_coef(eps);
    return true;
  }
  __device__ static bool resume(double eps) {
    set_coef(eps);
    return true;
  }
  __device__ static bool save(bool done) { return true; }
};

// The reference's control (stages, batches, tests) over a variant's phases.
// Every CTA runs it on its own copy of the state (sh().rs).
template <bool GAP, class P>
__device__ void persist_run(P& p) {
  const PersistArgs& A = P::A();
  PersistCtl* ctl = A.ctl;
  RunState& rs = P::sh().rs;
  // one thread changes the state, between two barriers of the CTA
  auto change = [&](auto f) {
    __syncthreads();
    if (threadIdx.x == 0) f();
    __syncthreads();
  };
  // the state this launch starts from (CTA 0 writes it back at the end, after
  // barriers that every CTA has passed)
  const int started = ctl->started;
  change([&] {
    rs.eps = ctl->eps;
    rs.sumk = ctl->sumk;
    rs.it = ctl->it;
    rs.checks = ctl->checks;
    rs.absorptions = ctl->absorptions;
    rs.used = 0;
    rs.stage = ctl->stage;
    rs.status = ctl->status;
    rs.lrow_valid = ctl->lrow_valid;
    rs.since = ctl->since;
    rs.index = ctl->index;
    rs.stage_done = 0;
    rs.batch = ctl->batch;
  });
  if (rs.status != kRunning) return;
  if (!started && !p.mean_growth()) return;
  p.constants();
  if (started && !p.resume(rs.eps)) return;
  if constexpr (GAP) {
    if (!started) {
      // epsilon0 * factor / factor, as the reference's arithmetic
      const double old = A.epsilon0 * A.scale_factor;
      change([&] { rs.eps = old / A.scale_factor; });
      if (!p.start_stage(old, rs.eps)) return;
    }
    while (rs.status == kRunning && rs.used < A.budget) {
      if (rs.stage_done) {
        const double old = rs.eps;
        change([&] {
          rs.eps = old / A.scale_factor;
          ++rs.stage;
          rs.lrow_valid = 0;
          rs.stage_done = 0;
        });
        if (!p.start_stage(old, rs.eps)) return;
        if (rs.stage == kScalings) {
          if (!(INFINITY > A.tolerance)) {   // `while gap > tolerance` from gap = inf: no iteration
            if (!p.fresh()) return;
            change([&] { rs.status = kConverged; });
            break;
          }
          double sumk;
          if (!p.sum_exp(&sumk)) return;
          change([&] { rs.sumk = sumk; });
        }
      }
      const int nb = rs.stage == kScalings ? A.batch_size : 5;
      // a batch may be longer than the launch, which then ends inside it (the next one
      // runs at least one of its iterations before the test)
      const int t0 = rs.batch;
      bool cached = rs.lrow_valid != 0, last = false;
      int t = t0;
      while (t < nb && !last && rs.used + (t - t0) < A.budget) {
        bool over = false;
        if (!p.iterate(cached, &over)) return;
        cached = false;
        ++t;
        if (over) {
          change([&] { ++rs.absorptions; });
          if (!p.absorb_now(rs.eps)) return;
        }
        last = (double)(rs.it + (t - t0)) >= A.max_iter;
      }
      const bool part = !last && t < nb;
      change([&] {
        rs.it += t - t0;
        rs.used += t - t0;
        rs.lrow_valid = 0;
        rs.batch = part ? t : 0;
        if (last)
          rs.status = kMaxIter;
        else if (!part)
          ++rs.checks;
      });
      if (part) break;
      if (last) {
        if (!p.fresh()) return;
        break;
      }
      bool go_on = true, nan = false;
      if (rs.stage == kScalings) {
        if (!p.fresh()) return;
        if (!p.gap_test(rs.sumk, &go_on, &nan)) return;
        change([&] {
          rs.lrow_valid = 1;
          if (!go_on) rs.status = nan ? kNonfinite : kConverged;
        });
      } else {
        if (!p.stage_test(&go_on)) return;
        change([&] {
          rs.stage_done = !go_on;
          if (!go_on && rs.used >= A.budget) rs.used = A.budget - 1;   // the next launch starts inside a stage
        });
      }
    }
  } else {
    const bool fixed = A.mode == kModeFixed;
    if (!started) {
      change([&] { rs.eps = fixed ? A.epsilon0 : A.epsilon; });
      if (!(fixed ? p.start_stage(0.0, rs.eps) : p.start_refine(rs.eps))) return;
    }
    const long long with_absorb = fixed ? A.scaling_iter : A.n_iter;
    const long long total_it = with_absorb + (fixed ? A.extra_iter : 0);
    while (rs.it < total_it && rs.used < A.budget) {
      bool over = false;
      if (!p.iterate(false, &over)) return;
      if (over && rs.it < with_absorb) {
        change([&] { ++rs.absorptions; });
        if (!p.absorb_now(rs.eps)) return;
      }
      const double old = rs.eps;
      bool new_eps = false;
      if (fixed && rs.it < with_absorb) new_eps = rs.since + 1 == A.inner_iter_max;
      change([&] {
        ++rs.it;
        ++rs.used;
        if (fixed) ++rs.since;
        if (new_eps) {
          ++rs.index;
          rs.since = 0;
          rs.eps = (A.epsilon0 - A.epsilon) * exp(-(double)rs.index) + A.epsilon;
        }
      });
      if (new_eps && !p.start_stage(old, rs.eps)) return;
    }
    if (rs.it >= total_it) {
      if (fixed && !p.fresh()) return;
      change([&] { rs.status = kConverged; });
    }
  }
  if (!p.save(rs.status != kRunning)) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    ctl->eps = rs.eps;
    ctl->sumk = rs.sumk;
    ctl->it = rs.it;
    ctl->checks = rs.checks;
    ctl->absorptions = rs.absorptions;
    ctl->stage = rs.stage;
    ctl->status = rs.status;
    ctl->lrow_valid = rs.lrow_valid;
    ctl->started = 1;
    ctl->since = rs.since;
    ctl->index = rs.index;
    ctl->batch = rs.batch;
  }
}

// GAP: the duality-gap solver (kModeGap); else kModeFixed or kModeRefine.
// KEPT: the cost stays in L2 (kKeptBytes).
template <bool GAP, bool KEPT>
__global__ void __launch_bounds__(kPersistThreads, 1) persist_kernel(const __grid_constant__ PersistArgs A) {
  PersistBase::begin(A);
  Streamed<KEPT> p;
  persist_run<GAP>(p);
}

}  // namespace wotg
