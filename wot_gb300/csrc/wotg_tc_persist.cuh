// wotg_tc_persist.cuh — a whole on-the-fly solve in one persistent kernel: the
// tensor-core half-step (see wotg_tc_kernel.cuh for its roles, partition and
// epilogue, which are the same here) looped over both sides, with the grid
// barriers, tests and control of wotg_persist.cuh in place of launches.
//
// What bounds it. A launch per half-step cost 14 us at 2000 x 2500, where each
// CTA has one 128 x 128 tile (about 1 us of tensor and exponential work), plus
// 2.5 to 3 us each for the launches that recompute out-of-range rows and test
// for absorption, both almost always empty. Most of the 14 us was the row-tile
// finish: its partials were read one CTA after another (an L2 round trip each)
// and its FP64 update took some 50 instructions of 64 cycles. Here a half-step is
// followed by a grid barrier, then every CTA finishes its own points: the
// partials loaded eight CTAs at a time and merged in the same order, the update
// folded to 19 FP64 instructions, recompute and absorption as flags in the second
// barrier. (Finishing a tile in the warp that wrote its last partial stalled that
// epilogue for 5 us at every row-tile boundary: a fence, an atomic, the loads and the
// FP64 chain, one after another.) At the largest sizes the half-step itself (the
// exponentials) is the bound, as before.
//
// A CTA is two of the half-step kernel's CTAs side by side (20 warps, one CTA per
// SM: a grid barrier needs all CTAs resident, and the runtime grants kernels that
// allocate tensor memory one CTA per SM only). Each half is a virtual CTA with its
// own roles, buffers and 256 TMEM columns; the partition is over the virtual CTAs.
//
// The accumulator and stage counters of the roles run on from one half-step to
// the next (jbase, segbase), so barriers, TMEM and the copy ring are set up once
// per launch. Column-form biases are written with ordinary stores and read by
// bulk copies in other CTAs: both sides of the grid barrier fence the proxies.
#pragma once

#include "wotg_persist.cuh"
#include "wotg_tc_kernel.cuh"

namespace wotg {

// One side of the problem as the kernel sees it.
struct TcSide {
  __half* row;            // packed row form [gamma x, 1, 1]
  __half* col;            // packed column form [x, bias columns]
  const float* pts;       // FP32 points
  int64_t ld, n;
  const double* norm;     // |x_i|^2
  float* off;             // offsets of the speculative sums
  int* redo;              // [count, rows...] to recompute exactly
  int tiles;
};

constexpr int kTcHalves = 2;
constexpr int kTcPersistThreads = kTcHalves * kTcThreads;

struct TcPersistArgs {
  PersistArgs p;
  int vctas;              // virtual CTAs (of the partition); CTA b holds b and b + gridDim.x
  TcSide x, y;
  int d;
  float2* part;
  unsigned long long* redo_total;
  double logs[4];         // log I, log J, log of the growth's mean, log tau
};

template <int KP>
struct TcPersist : Owned {
  using L = TcSmem<KP>;
  static constexpr int S = L::kStages, NA = L::kABuf;
  static constexpr uint32_t kHalfSmem = (L::kBytes + 1023u) & ~1023u;
  static constexpr uint32_t kAlloc = (uint32_t)kPlainHeaderBytes + kTcHalves * kHalfSmem;

  __device__ static __forceinline__ const TcPersistArgs& T() {
    return *reinterpret_cast<const TcPersistArgs*>(persist_hdr().args);
  }
  // this thread's half, its warp's role within it, the half's buffers and virtual CTA
  __device__ static __forceinline__ int half() { return threadIdx.x >= kTcThreads ? 1 : 0; }
  __device__ static __forceinline__ int role() { return ((int)threadIdx.x >> 5) - half() * (kTcThreads / 32); }
  __device__ static __forceinline__ unsigned char* buf() {
    return persist_smem + kPlainHeaderBytes + (uint32_t)half() * kHalfSmem;
  }
  __device__ static __forceinline__ int vb() { return blockIdx.x + half() * gridDim.x; }

  __device__ static __forceinline__ uint64_t* full() { return reinterpret_cast<uint64_t*>(buf() + L::kBar); }
  __device__ static __forceinline__ uint64_t* empty() { return full() + S; }
  __device__ static __forceinline__ uint64_t* a_full() { return full() + 2 * S; }
  __device__ static __forceinline__ uint64_t* a_empty() { return full() + 2 * S + NA; }
  __device__ static __forceinline__ uint64_t* acc_full() { return full() + 2 * S + 2 * NA; }
  __device__ static __forceinline__ uint64_t* acc_empty() { return full() + 2 * S + 2 * NA + kTcAcc; }
  __device__ static __forceinline__ uint64_t* drain() { return full() + 2 * S + 2 * NA + 2 * kTcAcc; }
  __device__ static __forceinline__ volatile int* abort_flag() { return reinterpret_cast<volatile int*>(drain() + 1); }
  // the TMEM allocation's address (one for both halves, beside half 0's abort flag)
  __device__ static __forceinline__ uint32_t* tmem_slot() {
    return reinterpret_cast<uint32_t*>(persist_smem + kPlainHeaderBytes + L::kBar +
                                       8 * (2 * S + 2 * NA + 2 * kTcAcc + 1) + 4);
  }
  __device__ static __forceinline__ uint32_t tmem() { return *tmem_slot() + (uint32_t)half() * L::kTmemCols; }

  __device__ TcPersist() {
    if (threadIdx.x >> 5 == 1) {
      tc::tmem_alloc(tmem_slot(), kTcHalves * L::kTmemCols);
      tc::tmem_relinquish();
    }
    if (threadIdx.x == 0) {
      const int flags = A().ctl->epoch;
      sh().row_ok = flags & 1;
      sh().col_ok = flags >> 1 & 1;
    }
    if (role() == 0 && (threadIdx.x & 31) == 0) {
      for (int b = 0; b < S; ++b) {
        tc::mbar_init(full() + b, 1);
        tc::mbar_init(empty() + b, 1);
      }
      for (int b = 0; b < NA; ++b) {
        tc::mbar_init(a_full() + b, 1);
        tc::mbar_init(a_empty() + b, 1);
      }
      for (int b = 0; b < kTcAcc; ++b) {
        tc::mbar_init(acc_full() + b, 1);
        tc::mbar_init(acc_empty() + b, kTcEpiWarps);
      }
      tc::mbar_init(drain(), 1);
      *abort_flag() = 0;
      tc::mbar_fence_init();
      find_stretch<true>();
      find_stretch<false>();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
  }

  // Everything asynchronous that this CTA issued has finished; TMEM is freed.
  __device__ static void finish() {
    __syncthreads();
    const bool lane0 = (threadIdx.x & 31) == 0;
    const int n = sh().copied[half()], seg = sh().copied_seg[half()];
    if (role() == 0 && lane0) {
      // the last copy into each buffer has landed (n tiles, seg segments issued)
      for (int b = 0; b < S && b < n; ++b) {
        const int jb = n - 1 - (n - 1 - b) % S;
        if (!tc::mbar_wait(full() + b, (uint32_t)((jb / S) & 1), kTcWaitTries)) atomicExch(&A().ctl->err, 2);
      }
      for (int b = 0; b < NA && b < seg; ++b) {
        const int sb = seg - 1 - (seg - 1 - b) % NA;
        if (!tc::mbar_wait(a_full() + b, (uint32_t)((sb / NA) & 1), kTcWaitTries)) atomicExch(&A().ctl->err, 2);
      }
    }
    if (role() == 1 && lane0) {
      // a last commit arrives once every MMA issued by this thread has completed
      tc::mma_commit(drain());
      if (!tc::mbar_wait(drain(), 0, kTcWaitTries)) atomicExch(&A().ctl->err, 2);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (threadIdx.x >> 5 == 1) tc::tmem_dealloc(*tmem_slot(), kTcHalves * L::kTmemCols);
  }
  // A bounded wait of this half ran out.
  __device__ static void give_up() {
    *abort_flag() = 1;
    atomicExch(&A().ctl->err, 1);
    sh().ok = 0;
  }

  // State of a point that its update reads.
  struct Point {
    double pot, ls, logp, norm;
  };
  template <bool ROW>
  __device__ static __forceinline__ Point load(int64_t i) {
    const Vecs& V = A().V;
    return Point{ROW ? V.u[i] : V.v[i], ROW ? V.la[i] : V.lb[i], ROW ? V.logp[i] : 0.0,
                 (ROW ? T().x : T().y).norm[i]};
  }
  // The FP64 update of point i from its natural log-sum-exp L (optimal_transport.py:
  // 133-134), its column-form bias for the other side's next half-step; true when the
  // scaling is above tau. In the reference's expressions, unfolded: the biases
  // keep 44 bits, so the last bit of the FP64 state reaches the FP32 exponents, and
  // another order of these operations moves results by FP32 roundings.
  template <bool ROW>
  __device__ static __forceinline__ bool update(int64_t i, const Point& p, double L) {
    const Coef& c = sh().c;
    double x;
    if (ROW) {
      const double logs = p.pot * c.inv_eps + L - c.logJ;
      x = c.alpha1 * (p.logp - logs) - p.pot * c.inv_l1e;
    } else {
      const double logt = p.pot * c.inv_eps + L - c.logI;
      x = c.alpha2 * (c.logq - logt) - p.pot * c.inv_l2e;
    }
    (ROW ? A().V.la_old : A().V.lb_old)[i] = p.ls;
    (ROW ? A().V.la : A().V.lb)[i] = x;
    bias<ROW>(i, p.pot, x, p.norm);
    return over_tau(x);
  }
  template <bool ROW>
  __device__ static __forceinline__ void bias(int64_t i, double pot, double ls, double norm) {
    const Coef& c = sh().c;
    tc_write_bias(i, (pot * c.inv_eps + ls) * kLog2e - (c.kappa * kLog2e) * norm, T().d, KP,
                  (ROW ? T().x : T().y).col);
  }

  // Grid barrier after a half-step, then the finish of the owned points: a thread per
  // point merges the partials of its row tile in the order of the virtual CTAs (FP32,
  // eight in flight), then updates the point or lists it for the exact recompute (a
  // speculative sum outside [2^-80, 2^100]). UPDATE: apply the update; else keep the row
  // sums (a gap check). What the barrier does not guard is read ahead of it.
  template <bool ROW, bool UPDATE>
  __device__ static __noinline__ bool finish_points(bool spec) {
    const TcSide& s = ROW ? T().x : T().y;
    const int end = ROW ? r1() : j1();
    int i = (ROW ? r0() : j0()) + threadIdx.x;
    Span w{0, 0};
    Point p{};
    if (i < end) {
      w = span<ROW>(i);
      p = load<ROW>(i);
    }
    if (!sync()) return false;
    while (i < end) {
      float m = kNegBig, sum = 0.f;
      for (int c = 0; c < w.n; c += 8) {
        float4 v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (c + k < w.n) v[k] = __ldcg(w.p + (int64_t)(c + k) * 128);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (c + k < w.n) {
            if (spec) {   // every partial is relative to the row's offset: the merge is a sum
              m = v[k].x;
              sum = (sum + v[k].y) + v[k].w;
            } else {
              lse_merge(m, sum, v[k].x, v[k].y);
              lse_merge(m, sum, v[k].z, v[k].w);
            }
          }
      }
      if (spec && !(sum >= 0x1p-80f && sum <= 0x1p100f)) {
        const int k = atomicAdd(s.redo, 1);
        s.redo[1 + k] = i;
        sh().row_flag = 1;
      } else {
        const double D = lse2(m, sum);
        finish_row<ROW, UPDATE>(i, p, D, D * kLn2 - sh().c.kappa * p.norm);
      }
      i += kTcPersistThreads;
      if (i < end) {
        w = span<ROW>(i);
        p = load<ROW>(i);
      }
    }
    async_fence();
    return true;
  }
  // The partials of point i's row: n virtual CTAs' from p on, 128 apart.
  struct Span {
    const float4* p;
    int n;
  };
  template <bool ROW>
  __device__ static __forceinline__ Span span(int i) {
    static_assert(kTcParts == 2, "a row's two column halves are one float4");
    const int nq = ROW ? T().y.tiles : T().x.tiles, t = i >> 7;
    const int64_t total = (int64_t)T().x.tiles * T().y.tiles;
    const int lo = (int)tc_cta_of((int64_t)t * nq, total, T().vctas);
    const int hi = (int)tc_cta_of(((int64_t)t + 1) * nq - 1, total, T().vctas);
    return Span{reinterpret_cast<const float4*>(T().part) + ((int64_t)lo + t) * 128 + (i & 127), hi - lo + 1};
  }
  // Biases written with ordinary stores are read by other CTAs' bulk copies after the
  // grid barrier that follows.
  __device__ static __forceinline__ void async_fence() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
  // D: base-2 log-sum-exp of the MMA exponents (without the row's -kappa |x|^2); L: the
  // row's natural log-sum-exp.
  template <bool ROW, bool UPDATE>
  __device__ static __forceinline__ void finish_row(int64_t i, const Point& p, double D, double L) {
    const TcSide& s = ROW ? T().x : T().y;
    s.off[i] = (float)D;
    if (!ROW) A().V.Lcol[i] = L;
    if (!UPDATE) {
      A().V.Lrow[i] = L;
    } else if (update<ROW>(i, p, L)) {
      sh().over_flag = 1;
    }
  }

  // This half's stretch of a half-step: n tiles from (row tile t, column tile q) on,
  // in nseg row tiles. Kept in the header: its 64-bit divisions took as long as a tile.
  template <bool ROW>
  __device__ static __forceinline__ TcStretch stretch() {
    return sh().stretch[ROW ? 0 : 1][half()];
  }
  template <bool ROW>
  __device__ static void find_stretch() {
    TcStretch r{0, 0, 0, 0, ROW ? T().y.tiles : T().x.tiles};
    const int64_t total = (int64_t)T().x.tiles * T().y.tiles;
    const int v = vb();
    if (v < T().vctas) {
      const int64_t f0 = tc_stretch_begin(v, total, T().vctas), f1 = tc_stretch_begin(v + 1, total, T().vctas);
      r.n = (int)(f1 - f0);
      r.t = (int)(f0 / r.nq);
      r.q = (int)(f0 % r.nq);
      r.nseg = r.n > 0 ? (int)((f1 - 1) / r.nq) - r.t + 1 : 0;
    }
    sh().stretch[ROW ? 0 : 1][half()] = r;
  }

  // Producer (one thread): bulk copies of row tiles (one per segment) and column
  // tiles; counts what it issued in jbase and segbase.
  template <bool ROW>
  __device__ static __noinline__ void produce(const TcStretch r) {
    const unsigned char* P = reinterpret_cast<const unsigned char*>(ROW ? T().x.row : T().y.row);
    const unsigned char* Q = reinterpret_cast<const unsigned char*>(ROW ? T().y.col : T().x.col);
    const uint32_t sA = tc::smem_u32(buf() + L::kA), sB = tc::smem_u32(buf() + L::kB);
    uint64_t* const b_full = full();
    uint64_t* const b_empty = empty();
    uint64_t* const b_afull = a_full();
    uint64_t* const b_aempty = a_empty();
    const volatile int* const abort = abort_flag();
    async_fence();
    int t = r.t, q = r.q, J = sh().jbase[half()], seg = sh().segbase[half()];
    const int end = J + r.n, nq = r.nq;
    bool fresh = true, good = true;
    while (J < end) {
      const int stage = J % S, a = seg % NA;
      good = J < S || tc::mbar_wait_or_abort(b_empty + stage, (uint32_t)((J / S - 1) & 1), kTcWaitTries, abort);
      if (good && fresh) {
        good = seg < NA || tc::mbar_wait_or_abort(b_aempty + a, (uint32_t)((seg / NA - 1) & 1), kTcWaitTries, abort);
        if (good) {
          tc::mbar_expect_tx(b_afull + a, L::kTileBytes);
          tc::bulk_g2s(sA + (uint32_t)a * L::kTileBytes, P + (int64_t)t * L::kTileBytes, L::kTileBytes, b_afull + a);
          ++seg;
        }
      }
      if (!good) break;
      tc::mbar_expect_tx(b_full + stage, L::kTileBytes);
      tc::bulk_g2s(sB + (uint32_t)stage * L::kTileBytes, Q + (int64_t)q * L::kTileBytes, L::kTileBytes,
                   b_full + stage);
      ++J;
      fresh = ++q == nq;
      if (fresh) {
        q = 0;
        ++t;
      }
    }
    sh().copied[half()] = J;
    sh().copied_seg[half()] = seg;
    if (!good) give_up();
  }

  // MMA issuer (one thread).
  __device__ static __noinline__ void multiply(const TcStretch r) {
    const uint32_t sA = tc::smem_u32(buf() + L::kA), sB = tc::smem_u32(buf() + L::kB);
    uint64_t* const b_full = full();
    uint64_t* const b_empty = empty();
    uint64_t* const b_afull = a_full();
    uint64_t* const b_aempty = a_empty();
    uint64_t* const b_accfull = acc_full();
    uint64_t* const b_accempty = acc_empty();
    const uint32_t td = tmem();
    int q = r.q, J = sh().jbase[half()], seg = sh().segbase[half()];
    const int end = J + r.n, nq = r.nq;
    bool fresh = true, good = true;
    int a = 0;
    while (J < end) {
      const int stage = J % S, b = J % kTcAcc;
      if (fresh) {
        a = seg % NA;
        good = tc::mbar_wait(b_afull + a, (uint32_t)((seg / NA) & 1), kTcWaitTries);
        ++seg;
      }
      good = good && tc::mbar_wait(b_full + stage, (uint32_t)((J / S) & 1), kTcWaitTries);
      if (J >= kTcAcc)
        good = good && tc::mbar_wait(b_accempty + b, (uint32_t)((J / kTcAcc - 1) & 1), kTcWaitTries);
      if (!good) break;
      tc::fence_after_sync();
      tc_issue_mma<KP>(td + (uint32_t)(128 * b), sA + (uint32_t)a * L::kTileBytes,
                       sB + (uint32_t)stage * L::kTileBytes);
      tc::mma_commit(b_empty + stage);
      tc::mma_commit(b_accfull + b);
      ++J;
      fresh = ++q == nq;
      if (fresh) q = 0;
      if (J == end || fresh) tc::mma_commit(b_aempty + a);
    }
    if (!good) give_up();
  }

  // One warp's share of tiles [J, end) of a row tile: its 64 columns of each
  // accumulator into the row's partial (m, s).
  template <bool SPEC>
  __device__ static __forceinline__ float2 segment(uint32_t tbase, int J, int end, float mm) {
    uint64_t* const accfull = acc_full();
    uint64_t* const accempty = acc_empty();
    float s = 0.f;
    float2 acc[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    for (; J < end; ++J) {
      const int b = J % kTcAcc;
      if (!__all_sync(0xffffffffu, tc::mbar_wait(accfull + b, (uint32_t)((J / kTcAcc) & 1), kTcWaitTries))) {
        if ((threadIdx.x & 31) == 0) give_up();
        break;
      }
      tc::fence_after_sync();
      const uint32_t taddr = tbase + (uint32_t)(128 * b);
      float d0[32], d1[32];
      tc::tmem_read64(taddr, d0, d1);
      tc::fence_before_sync();
      __syncwarp();
      if ((threadIdx.x & 31) == 0) tc::mbar_arrive(accempty + b);
      if (SPEC) {
        sum32_off(d0, mm, acc);
        sum32_off(d1, mm, acc);
      } else {
        lse32(d0, mm, s);
        lse32(d1, mm, s);
      }
    }
    if (SPEC) {
      const float2 a = __fadd2_rn(__fadd2_rn(acc[0], acc[1]), __fadd2_rn(acc[2], acc[3]));
      s = a.x + a.y;
    }
    return make_float2(mm, s);
  }

  // Epilogue: warp w reads TMEM lanes 32 (w % 4) .. + 31, columns of group (w - 2) / 4,
  // and writes one partial per row and segment. A function of its own with the tile loop
  // in it: the 64 accumulator values leave no room for a caller's registers (as a call
  // per segment the loop spilled and took 12 % longer).
  template <bool ROW>
  __device__ static __noinline__ void epilogue(const TcStretch& r, bool spec) {
    const int lane = threadIdx.x & 31;
    const int wq = ((int)threadIdx.x >> 5) & 3, cq = (role() - 2) >> 2;   // the hardware's lane quarter of the warp
    const int row = 32 * wq + lane;
    const float* off = (ROW ? T().x.off : T().y.off) + row;
    const uint32_t tbase = tmem() + ((uint32_t)(32 * wq) << 16) + (uint32_t)(kTcColsPerWarp * cq);
    float2* const part = T().part + ((int64_t)vb() * 128 + row) * kTcParts + cq;
    int t = r.t, q = r.q, J = sh().jbase[half()];
    const int end = J + r.n;
    while (J < end) {
      const int stop = min(end, J + r.nq - q);
      part[(int64_t)t * 128 * kTcParts] =
          spec ? segment<true>(tbase, J, stop, off[(int64_t)t * 128]) : segment<false>(tbase, J, stop, kNegBig);
      __syncwarp();
      if (!*(volatile int*)&sh().ok) break;
      J = stop;
      q = 0;
      ++t;
    }
  }

  // One half-step of a side over the other side's column form: the partials.
  template <bool ROW>
  __device__ static __noinline__ bool half_step(bool spec) {
    const TcStretch r = stretch<ROW>();
    const int w = role();
    const bool lane0 = (threadIdx.x & 31) == 0;
    if (w == 0) {
      if (lane0) produce<ROW>(r);
    } else if (w == 1) {
      if (lane0) multiply(r);
    } else {
      epilogue<ROW>(r, spec);
    }
    if (threadIdx.x == 0) sh().row_flag = sh().over_flag = 0;
    __syncthreads();
    if (w == 0 && lane0) {   // read again only after the grid barrier
      sh().jbase[half()] += r.n;
      sh().segbase[half()] += r.nseg;
    }
    return sh().ok != 0;
  }

  // Rows whose speculative sum left the safe range, exactly: a warp per row from the
  // FP32 points with a running maximum, over the whole grid.
  template <bool ROW, bool UPDATE>
  __device__ static __noinline__ void exact_rows() {
    const TcSide& P = ROW ? T().x : T().y;
    const TcSide& Q = ROW ? T().y : T().x;
    const int lane = threadIdx.x & 31;
    const int cnt = *(volatile int*)P.redo;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(T().redo_total, (unsigned long long)cnt);
    const double* pot = ROW ? A().V.v : A().V.u;
    const double* lsc = ROW ? A().V.lb : A().V.la;
    const float k2 = (float)(sh().c.kappa * kLog2e);
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < cnt; w += nw) {
      const int64_t i = *(volatile int*)(P.redo + 1 + w);
      const float* x = P.pts + i * P.ld;
      float m = kNegBig, s = 0.f;
      for (int64_t j = lane; j < Q.n; j += 32) {
        const float* y = Q.pts + j * Q.ld;
        float cc = 0.f;
        for (int t = 0; t < T().d; ++t) {
          const float df = x[t] - y[t];
          cc = fmaf(df, df, cc);
        }
        const float tt = (float)((pot[j] * sh().c.inv_eps + lsc[j]) * kLog2e) - k2 * cc;
        const float mn = fmaxf(m, tt);
        s = s * ex2(m - mn) + ex2(tt - mn);
        m = mn;
      }
      warp_lse(m, s);
      if (lane == 0) {
        const double L2 = lse2(m, s);
        finish_row<ROW, UPDATE>(i, load<ROW>(i), L2 + (double)k2 * P.norm[i], L2 * kLn2);
      }
    }
    async_fence();
  }

  // A half-step with its barrier, and the exact recompute where rows ask for it;
  // `over` or-ed over the grid.
  template <bool ROW, bool UPDATE>
  __device__ static __noinline__ bool side(bool* over) {
    const TcSide& P = ROW ? T().x : T().y;
    const bool spec = (ROW ? sh().row_ok : sh().col_ok) != 0;
    if (!half_step<ROW>(spec) || !finish_points<ROW, UPDATE>(spec)) return false;
    __syncthreads();
    if (threadIdx.x == 0) (ROW ? sh().row_ok : sh().col_ok) = 1;
    bool redo = false, ov = false, ov2 = false;
    if (!sync(sh().over_flag != 0, &ov, sh().row_flag != 0, &redo)) return false;
    if (redo) {
      __syncthreads();
      if (threadIdx.x == 0) sh().over_flag = 0;
      __syncthreads();
      exact_rows<ROW, UPDATE>();
      __syncthreads();
      if (!sync(sh().over_flag != 0, &ov2)) return false;
      // nobody reads the list any more; the next half-step of this side is two barriers away
      if (blockIdx.x == 0 && threadIdx.x == 0) P.redo[0] = 0;
    }
    *over = ov || ov2;
    return true;
  }

  // The growth's mean and the logarithms come from the host (as far as the last bit).
  __device__ static bool mean_growth() { return true; }
  __device__ static void constants() {
    PersistBase::constants();
    if (threadIdx.x < 4) sh().consts[threadIdx.x] = T().logs[threadIdx.x];
  }

  __device__ static bool iterate(bool cached, bool* over) {
    bool o1 = false, o2 = false;
    if (cached) {
      bool o = false;
      for (int i = r0() + threadIdx.x; i < r1(); i += kTcPersistThreads) o |= update<true>(i, load<true>(i), A().V.Lrow[i]);
      async_fence();
      o = __syncthreads_or(o);
      if (!sync(o, &o1)) return false;
    } else {
      if (!side<true, true>(&o1)) return false;
    }
    if (!side<false, true>(&o2)) return false;
    *over = o1 || o2;
    return true;
  }
  __device__ static bool fresh() {
    bool o;
    return side<true, false>(&o);
  }

  // u += eps log a, a = 1 (and for v, b); RESCALE: the start of a stage, whose row
  // forms carry the new gamma and whose offsets are stale. Biases of both sides.
  template <bool RESCALE>
  __device__ static __noinline__ bool absorb(double eps_old) {
    for (int i = r0() + threadIdx.x; i < r1(); i += kTcPersistThreads) {
      const double un = A().V.u[i] + eps_old * A().V.la[i];
      A().V.u[i] = un;
      A().V.la[i] = 0.0;
      if (RESCALE) A().V.la_old[i] = 0.0;
      bias<true>(i, un, 0.0, T().x.norm[i]);
    }
    for (int j = j0() + threadIdx.x; j < j1(); j += kTcPersistThreads) {
      const double vn = A().V.v[j] + eps_old * A().V.lb[j];
      A().V.v[j] = vn;
      A().V.lb[j] = 0.0;
      if (RESCALE) A().V.lb_old[j] = 0.0;
      bias<false>(j, vn, 0.0, T().y.norm[j]);
    }
    if (RESCALE) {
      pack_rows();
      __syncthreads();
      if (threadIdx.x == 0) sh().row_ok = sh().col_ok = 0;
    }
    async_fence();
    return sync();
  }
  // Row forms of both sides for the current epsilon: gamma = 2 kappa log2 e /
  // sqrt(cost_scale) times the points (the column forms hold sqrt(cost_scale) y).
  __device__ static void pack_rows() {
    const float gamma = (float)(2.0 * sh().c.kappa * kLog2e / sqrt(A().cost_scale));
    pack_side(T().x, gamma);
    pack_side(T().y, gamma);
  }
  __device__ static void pack_side(const TcSide& s, float gamma) {
    const int64_t total = (int64_t)s.tiles * 128 * KP;
    for (int64_t k = (int64_t)blockIdx.x * kTcPersistThreads + threadIdx.x; k < total;
         k += (int64_t)gridDim.x * kTcPersistThreads)
      tc_pack_entry(s.pts, s.n, s.ld, T().d, KP, gamma, 1, s.row, k);
  }
  __device__ static bool start_stage(double eps_old, double eps) {
    set_coef(eps);
    reset_gap();
    return absorb<true>(eps_old);
  }
  __device__ static bool absorb_now(double eps) { return absorb<false>(eps); }
  __device__ static bool start_refine(double eps) {
    set_coef(eps);
    return absorb<true>(0.0);   // a = b = 1: packs only
  }
  __device__ static bool resume(double eps) {
    set_coef(eps);
    return true;
  }
  __device__ static bool gap_test(double sumk, bool* go_on, bool* nan) {
    const double* l = A().V.Lcol;
    return gap_test_with([l](int j) { return l[j]; }, sumk, go_on, nan);
  }
  // The column weights of the dense coupling; which offsets exist, for the next launch.
  __device__ static bool save(bool done) {
    if (done)
      for (int j = j0() + threadIdx.x; j < j1(); j += kTcPersistThreads)
        split_weight((A().V.v[j] * sh().c.inv_eps + A().V.lb[j]) * kLog2e, A().V.wcol, A().V.wcol_lo, j);
    if (blockIdx.x == 0 && threadIdx.x == 0) A().ctl->epoch = sh().row_ok | sh().col_ok << 1;
    return true;
  }
};

template <int KP, bool GAP>
__global__ void __launch_bounds__(kTcPersistThreads, 1) tc_persist_kernel(const __grid_constant__ TcPersistArgs T) {
  PersistBase::begin(T);
  TcPersist<KP> p;
  persist_run<GAP>(p);
  p.finish();
}

}  // namespace wotg
