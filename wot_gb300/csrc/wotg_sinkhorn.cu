// wotg_sinkhorn.cu — stabilised unbalanced Sinkhorn on a materialised FP32 cost (sm_103a).
//
// Reference: wot/ot/optimal_transport.py (wot 1.0.8)
//   compute_transport_matrix        :10-33   -> wotg_compute_transport_matrix (growth loop)
//   optimal_transport_duality_gap   :67-164  -> solve_persistent, kModeGap
//   transport_stablev2              :167-236 -> solve_persistent, kModeFixed
//   primal / dual                   :45-62   -> gap_test (O(I+J), see below)
//
// State. The reference keeps FP64 absorbed potentials u, v, scalings a, b and
// the stabilised kernel K = exp((u_i - C_ij + v_j)/eps) as a dense matrix that
// it rebuilds at every absorption and epsilon change. Here the dense object is
// the FP32 cost C (written once per day pair) and the scalings are kept in the
// log domain (la = log a, lb = log b, FP64), so one half-step is
//   log(K (b dy))_i = u_i/eps + log sum_j exp(v_j/eps + lb_j - cost_scale C_ij/eps) - log J
// evaluated as a streaming base-2 log-sum-exp over the row of C, followed by the
// reference's update a = (p / K(b dy))^alpha1 exp(-u/(lambda1+eps)) in FP64.
// Absorption (u += eps log a, a = 1) then only touches O(I+J) vectors and no
// matrix is ever rebuilt; the sequence of (u, v, a, b) is the reference's.
//
// Duality gap. With R = diag(a) K diag(b) the identity
//   eps R_ij log R_ij + R_ij C_ij = R_ij (ubar_i + vbar_j),  ubar = u + eps log a,
// turns the reference's primal - dual (two I x J passes with log) into sums over
// the row sums x = R dy and column sums y = R^T dx only:
//   primal - dual = F1(x) + F2(y) + F1*(-eps log a~) + F2*(-eps log b~) + dx<ubar,x> + dy<vbar,y>
// (a~ = a exp(u/eps) evaluated as the reference does, overflow included), and
//   primal = F1(x) + F2(y) + dx<ubar,x> + dy<vbar,y> + eps (sum(exp(-C/eps))/(IJ) - dx sum x).
// The row sums with the current b are exactly the next iteration's first
// half-step, so a gap check costs one row pass that the next iteration reuses.
//
// A solve is one cooperative kernel, launched anew every 20 ms of iterations:
// wotg_resident.cuh (costs that fit in shared memory), wotg_persist.cuh (any cost, and
// the control of all three) or wotg_tc_persist.cuh (costs formed on the fly). Here are
// the entry points, the choice and the outputs.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "wotg_coef.cuh"
#include "wotg_common.cuh"
#include "wotg_onthefly.cuh"
#include "wotg_persist.cuh"
#include "wotg_resident.cuh"
#include "wotg_state.cuh"
#include "wotg_tc_kernel.cuh"
#include "wotg_tc_persist.cuh"

namespace wotg {

// Buffers of the on-the-fly (tensor-core) form.
struct TcState {
  bool on;
  int kp;                   // packed dimension (32 or 64)
  int n_xt, n_yt;           // 128-point tiles of X and Y
  int64_t I_pad, J_pad;
  int ctas_row, ctas_col;   // persistent grid of each pass
  __half* Xa;               // row form of X: [gamma x, 1, 1]   (repacked per epsilon)
  __half* Xb;               // column form of X: [x, bias columns] (bias per half-step)
  __half* Ya;
  __half* Yb;
  const float* X;
  const float* Y;
  int64_t ldx, ldy;
  int d;
  double* normX;            // |x_i|^2 (FP64)
  double* normY;
  float2* part;
  // Speculative half-steps: each row's base-2 log-sum-exp of the MMA exponents
  // from the previous half-step (row side offX, column side offY), valid while
  // epsilon is unchanged; rows whose sum left the safe range are listed in
  // redoX / redoY = [count, rows...] (row and column passes) and recomputed exactly.
  float* offX;
  float* offY;
  int* redoX;
  int* redoY;
  unsigned long long* redo_total;  // rows recomputed exactly, over the solve (diagnostic)
};

// Standalone row pass: one warp per row, 128-bit streaming loads of C, online
// base-2 LSE of one FP32 weight vector.
__global__ void __launch_bounds__(256) row_pass_kernel(const float* __restrict__ C, Geom g, const float* w, float k2,
                                                       double* __restrict__ L) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const float4* w4 = reinterpret_cast<const float4*>(w);
  for (int64_t i = warp; i < g.I; i += nwarps) {
    float m, s, cmp;
    const float4* row = reinterpret_cast<const float4*>(C + i * g.ldc);
    auto wk = [w4](int k) { return __ldg(w4 + k); };
    row_lse<false>([row](int k) { return ld_once(row + k); }, wk, wk, (int)(g.ldc >> 2), lane, 0.f, k2, 0.f, m, s, cmp);
    warp_lse(m, s);
    if (lane == 0) L[i] = ((double)m + log2((double)s)) * kLn2;
  }
}

// Standalone column pass, phase 1: CTA = 1024 columns (float4 per thread) x
// rows_per rows; writes one (m, s) base-2 LSE partial per column and row block.
__global__ void __launch_bounds__(256) col_partial_kernel(const float* __restrict__ C, Geom g, const float* w, float k2,
                                                          float2* __restrict__ part) {
  const int64_t c4 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.y * g.rows_per;
  if (c4 >= g.ldc >> 2) return;
  const float o[4] = {0.f, 0.f, 0.f, 0.f};
  float m[4], s[4];
  const float4* col = reinterpret_cast<const float4*>(C) + c4;
  const int64_t ld4 = g.ldc >> 2;
  auto wi = [w](int64_t i) { return __ldg(w + i); };
  col_lse<false>([=](int64_t i) { return ld_once(col + i * ld4); }, wi, wi, r0, min(g.I, r0 + g.rows_per), o, k2, 0.f,
                 m, s);
  float4* out = reinterpret_cast<float4*>(part + (int64_t)blockIdx.y * g.ldc + c4 * 4);
  out[0] = make_float4(m[0], s[0], m[1], s[1]);
  out[1] = make_float4(m[2], s[2], m[3], s[3]);
}

// Phase 2: the row-block partials of each column.
__global__ void col_combine_kernel(Geom g, const float2* __restrict__ part, double* __restrict__ L) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= g.J) return;
  float m = kNegBig, s = 0.f;
  for (int r = 0; r < g.nrb; ++r) {
    const float2 ps = part[(int64_t)r * g.ldc + j];
    lse_merge(m, s, ps.x, ps.y);
  }
  L[j] = lse2(m, s) * kLn2;
}

// Zero state for a new solve; p = G; padding of wcol = 0.
__global__ void init_kernel(Geom g, Vecs V, const double* __restrict__ G) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < g.I) {
    V.u[idx] = 0.0;
    V.la[idx] = 0.0;
    V.la_old[idx] = 0.0;
    const double pi = G[idx];
    V.p[idx] = pi;
    V.logp[idx] = log(pi);
    V.wrow[idx] = 0.f;
    V.wrow_lo[idx] = 0.f;
    V.Lrow[idx] = 0.0;
    reinterpret_cast<float*>(V.rowc)[idx] = 0.f;   // row offsets of the persistent solver
  }
  if (idx < g.ldc) {
    V.wcol[idx] = 0.f;
    V.wcol_lo[idx] = 0.f;
    if (idx < g.J) {
      V.v[idx] = 0.0;
      V.lb[idx] = 0.0;
      V.lb_old[idx] = 0.0;
      V.Lcol[idx] = 0.0;
    }
  }
}

// Warm start from absorbed potentials: u = u_bar, v = v_bar, a = b = 1.
__global__ void load_potentials_kernel(Geom g, Vecs V, const double* __restrict__ ubar,
                                       const double* __restrict__ vbar, double inv_eps) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < g.I) {
    V.u[idx] = ubar[idx];
    V.la[idx] = 0.0;
    V.la_old[idx] = 0.0;
    V.Lrow[idx] = 0.0;
    split_weight(ubar[idx] * inv_eps * kLog2e, V.wrow, V.wrow_lo, idx);
  } else if (idx < g.I + g.J) {
    const int64_t j = idx - g.I;
    V.v[j] = vbar[j];
    V.lb[j] = 0.0;
    V.lb_old[j] = 0.0;
    V.Lcol[j] = 0.0;
    split_weight(vbar[j] * inv_eps * kLog2e, V.wcol, V.wcol_lo, j);
  }
}

// Outputs. `log_scale` is the log of the factor applied to R = diag(a) K diag(b):
// -log J for the reference's normal return R / J, 0 for its max_iter return R.
// Row sums of the returned coupling (tmap.sum(axis=1)); needs Lrow with the final b.
__global__ void row_sums_kernel(Geom g, Vecs V, Coef c, double log_scale, double* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < g.I;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = exp(V.la[i] + V.u[i] * c.inv_eps + V.Lrow[i] + log_scale);
}

__global__ void potentials_kernel(Geom g, Vecs V, Coef c, double* __restrict__ ubar,
                                  double* __restrict__ vbar) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < g.I) {
    if (ubar) ubar[idx] = V.u[idx] + c.eps * V.la[idx];
  } else if (idx < g.I + g.J) {
    const int64_t j = idx - g.I;
    if (vbar) vbar[j] = V.v[j] + c.eps * V.lb[j];
  }
}

// Per-row constants of the dense coupling: the row's base-2 exponent
//   t_ij = wr_i + wc_j - k2 C_ij,   wr_i = (u_i / eps + la_i + log_scale) log2 e,
// is evaluated as t_ij = x_ij + E_i with x_ij = (wc_j - o_i) - k2 C_ij in FP32
// (the streamed passes' split arithmetic, o_i the row's grid offset from its
// log-sum-exp L_i, so x <= ~0 for the entries that carry mass) and
// E_i = o_i + wr_i = n_i + f_i in FP64: rowc = (o_i, 2^f_i, n_i, 1); w = 0 marks
// a row whose constants are not finite (its entries take the FP64 path).
__global__ void coupling_rows_kernel(Geom g, Vecs V, Coef c, double log_scale) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.I) return;
  const double wr = (V.u[i] * c.inv_eps + V.la[i] + log_scale) * kLog2e;
  const double L = V.Lrow[i];
  const float o = grid_offset(L);
  const double E = (double)o + wr;
  float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
  if (fabs(L) < 1e30 && fabs(E) < 900.0) {
    const double n = floor(E);
    r = make_float4(o, (float)exp2(E - n), (float)n, 1.f);
  }
  V.rowc[i] = r;
}

// 2^t for an FP64 exponent t: the integer part exactly (as the FP64 exponent
// field), the fraction by FP32 ex2 (relative error ~2^-22); 0 below 2^-1020,
// NaN for NaN.
__device__ __forceinline__ double exp2_split(double t) {
  if (!(t > -1020.0)) return t != t ? t : 0.0;
  if (t >= 1024.0) return INFINITY;
  const double ti = floor(t);
  const double scale = __longlong_as_double((long long)(ti + 1023.0) << 52);
  return (double)ex2((float)(t - ti)) * scale;
}

// Dense coupling tmap_ij = a_i exp((u_i - C_ij + v_j)/eps) b_j * exp(log_scale), written
// FP64 row-major (stride J) like the reference's ndarray. 2^t_ij = (2^x_ij 2^f_i) 2^n_i
// (coupling_rows_kernel): x_ij = fma(-k2hi, C, wc_hi - o_i) + fma(-k2lo, C, wc_lo) as in
// the streamed passes (one FP32 rounding of a value that is small for the entries that
// carry mass, below the FP32 storage of C), 2^x 2^f in FP32, and the power 2^n_i put into
// the FP64 exponent field by integer arithmetic, so that no element needs FP64
// arithmetic (slow on this part) and the kernel streams C in and the map out. Entries
// whose 2^x or result leaves the normal ranges (far below a row's mass, or non-finite
// inputs) take the FP64 exponent (exp2_split), which is exact in the same way.
__global__ void __launch_bounds__(256) coupling_kernel(const float* __restrict__ C, Geom g, Vecs V,
                                                       Coef c, double log_scale, double* __restrict__ out) {
  for (int64_t j0 = (int64_t)blockIdx.x * blockDim.x; j0 < g.J; j0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = j0 + threadIdx.x;
    if (j >= g.J) continue;
    const float hi = V.wcol[j], lo = V.wcol_lo[j];   // once per column
    for (int64_t i = blockIdx.y; i < g.I; i += gridDim.y) {
      const float4 rc = V.rowc[i];
      const float cc = C[i * g.ldc + j];
      const float x = fmaf(-c.kappa2, cc, hi - rc.x) + fmaf(-c.kappa2_lo, cc, lo);
      double val;
      bool done = false;
      if (rc.w != 0.f && x > -125.f && x < 125.f) {
        const float y = ex2(x) * rc.y;                              // normal, positive
        const uint32_t yb = __float_as_uint(y);
        const int e = (int)(yb >> 23) - 127 + (int)rc.z;           // exponent of the result
        if (e > -1022 && e < 1023) {
          val = __longlong_as_double((long long)((uint64_t)(e + 1023) << 52 | (uint64_t)(yb & 0x7FFFFFu) << 29));
          done = true;
        }
      }
      if (!done) {
        const double wr = (V.u[i] * c.inv_eps + V.la[i] + log_scale) * kLog2e;
        const double wc = (V.v[j] * c.inv_eps + V.lb[j]) * kLog2e;
        val = exp2_split(wr + wc - c.kappa * kLog2e * (double)cc);
      }
      out[i * g.J + j] = val;
    }
  }
}

// Sum of n values on kRedBlocks + 1 blocks of 256 threads, in a fixed order (the
// growth's mean of the on-the-fly solver; its last bit reaches the results).
__device__ __forceinline__ void block_sum_store(double acc, double* out) {
  __shared__ double sh[8];
  const int lane = threadIdx.x & 31;
  acc = warp_sum(acc);
  if (lane == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    const double t = warp_sum(lane < 8 ? sh[lane] : 0.0);
    if (lane == 0) *out = t;
  }
}
__global__ void __launch_bounds__(256) sum_vec_kernel(const double* __restrict__ x, int64_t n, double* red) {
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) acc += x[i];
  block_sum_store(acc, red + blockIdx.x);
}
__global__ void __launch_bounds__(256) finalize_sum_kernel(const double* __restrict__ red, int n, double* out) {
  double acc = 0.0;
  for (int b = threadIdx.x; b < n; b += 256) acc += red[b];
  block_sum_store(acc, out);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
struct Solver {
  const float* C;
  Geom g;
  Vecs V;
  cudaStream_t st;
  double cost_scale;
  TcState tc;

  Coef coef(double eps, const wotg_params& P, double q) const {
    return make_coef(eps, P.lambda1, P.lambda2, cost_scale, g.I, g.J, q);
  }

  int vec_blocks(int64_t n) const { return (int)std::max<int64_t>(1, (n + 255) / 256); }

  // Rows that the speculative on-the-fly half-steps recomputed exactly; synchronises.
  int exact_rows(int32_t* out) const {
    if (!tc.on) return WOTG_OK;
    unsigned long long redo = 0;
    WOTG_CUDA(cudaMemcpyAsync(&redo, tc.redo_total, sizeof(redo), cudaMemcpyDeviceToHost, st));
    WOTG_CUDA(cudaStreamSynchronize(st));
    *out = (int32_t)std::min<unsigned long long>(redo, 0x7fffffffull);
    return WOTG_OK;
  }

  int mean_of(const double* x, int64_t n, double* out) const {
    sum_vec_kernel<<<kRedBlocks, 256, 0, st>>>(x, n, V.red);
    finalize_sum_kernel<<<1, 256, 0, st>>>(V.red, kRedBlocks, V.scal);
    WOTG_LAUNCHED();
    double h;
    WOTG_CUDA(cudaMemcpyAsync(&h, V.scal, sizeof(h), cudaMemcpyDeviceToHost, st));
    WOTG_CUDA(cudaStreamSynchronize(st));
    *out = h / (double)n;
    return WOTG_OK;
  }

  // Solver outputs for one solve: learned row sums (device), optionally the
  // dense coupling and potentials.
  int outputs(const Coef& c, bool no_div_j, double* tmap, double* row_sums, double* ubar,
              double* vbar) {
    const double log_scale = no_div_j ? 0.0 : -c.logJ;
    if (row_sums) {
      row_sums_kernel<<<vec_blocks(g.I), 256, 0, st>>>(g, V, c, log_scale, row_sums);
      WOTG_LAUNCHED();
    }
    if (ubar || vbar) {
      potentials_kernel<<<vec_blocks(g.I + g.J), 256, 0, st>>>(g, V, c, ubar, vbar);
      WOTG_LAUNCHED();
    }
    if (tmap) {
      coupling_rows_kernel<<<vec_blocks(g.I), 256, 0, st>>>(g, V, c, log_scale);
      WOTG_LAUNCHED();
      // every column in one wave of x blocks (its weight read once per thread), rows over y
      dim3 grid((unsigned)std::min<int64_t>((g.J + 255) / 256, 65535), (unsigned)std::min<int64_t>(g.I, 128));
      coupling_kernel<<<grid, 256, 0, st>>>(C, g, V, c, log_scale, tmap);
      WOTG_LAUNCHED();
    }
    return WOTG_OK;
  }
};

struct SolveResult {
  int status = WOTG_OK;
  bool max_iter = false;
  int64_t iterations = 0;
  int64_t checks = 0;
  int64_t absorptions = 0;
  double gap = NAN;
  double eps = 0.0;
  Coef final_coef{};
};

static const void* streamed_kernel(bool gap, bool kept) {
  if (gap) return kept ? reinterpret_cast<const void*>(persist_kernel<true, true>) : reinterpret_cast<const void*>(persist_kernel<true, false>);
  return kept ? reinterpret_cast<const void*>(persist_kernel<false, true>) : reinterpret_cast<const void*>(persist_kernel<false, false>);
}

// Shared memory the solvers on a cost may use beside their static part; their limit
// is raised to it once per device.
static int resident_room(int* room) {
  static std::atomic<int> known[64] = {};
  int dev = 0;
  WOTG_CUDA(cudaGetDevice(&dev));
  if (dev < 64 && (*room = known[dev].load(std::memory_order_acquire)) > 0) return WOTG_OK;
  int limit = 0;
  WOTG_CUDA(cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const void* const kernels[] = {reinterpret_cast<const void*>(resident_kernel<true>),
                                 reinterpret_cast<const void*>(resident_kernel<false>),
                                 streamed_kernel(true, true), streamed_kernel(true, false),
                                 streamed_kernel(false, true), streamed_kernel(false, false)};
  *room = limit;
  for (const void* k : kernels) {
    cudaFuncAttributes a{};
    WOTG_CUDA(cudaFuncGetAttributes(&a, k));
    *room = std::min(*room, limit - (int)a.sharedSizeBytes);
  }
  for (const void* k : kernels) WOTG_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, *room));
  if (dev < 64) known[dev].store(*room, std::memory_order_release);
  return WOTG_OK;
}

// A solve (mode kModeGap / kModeFixed) or n_iter refinement iterations at epsilon
// `eps` (kModeRefine): launches of the form's persistent kernel until it reports an
// end. A launch is kept to some 20 ms (an iteration costs about 8 us and 2.5 ps per
// entry streamed, 0.4 ps per entry on the tensor cores), so that a long solve
// stays a sequence of short kernels.
static int solve_persistent(Solver& S, const wotg_params& P, int mode, double eps, int n_iter, SolveResult& res) {
  static_assert(sizeof(PersistCtl) <= 16 * sizeof(double), "PersistCtl lives in Vecs::scal");
  PersistArgs A{};
  A.C = S.C;
  A.g = S.g;
  A.V = S.V;
  A.ctl = reinterpret_cast<PersistCtl*>(S.V.scal);
  A.epsilon = eps;
  A.lambda1 = P.lambda1;
  A.lambda2 = P.lambda2;
  A.epsilon0 = P.epsilon0;
  A.tau = P.tau;
  A.tolerance = P.tolerance;
  A.max_iter = P.max_iter;
  A.cost_scale = S.cost_scale;
  A.scale_factor = std::exp(-std::log(P.epsilon) / kScalings);
  A.batch_size = P.batch_size;
  A.scaling_iter = P.scaling_iter;
  A.inner_iter_max = P.inner_iter_max;
  A.extra_iter = P.extra_iter;
  A.n_iter = n_iter;
  A.mode = mode;
  const double per_iter = 8e-6 + (S.tc.on ? 4e-13 : 2.5e-12) * (double)S.g.I * (double)S.g.J;
  // at most 2000, or as many as the barrier's flag counts last
  const int flagged = S.tc.on ? 4 : 1;
  A.budget = std::min<long long>(2000, ((1 << kBarrierFlagBits) - 1) / (flagged * std::min(sm_count(), kRedBlocks)));
  A.budget = std::max<long long>(8, std::min<long long>(A.budget, (long long)(0.02 / per_iter)));
  PersistCtl h{};
  if (S.tc.on) {
    int s = S.mean_of(S.V.p, S.g.I, &h.q);
    if (s) return s;
  }
  WOTG_CUDA(cudaMemcpyAsync(A.ctl, &h, sizeof(h), cudaMemcpyHostToDevice, S.st));
  // one CTA per SM; fewer only where the device grants the process fewer SMs
  int grid = std::min(sm_count(), kRedBlocks);
  int rows_cap = 0, cols_cap = 0;
  size_t streamed_smem = kMergeHeaderBytes, smem = streamed_smem;
  const bool gap = mode == kModeGap;
  const void* streamed = streamed_kernel(gap, 4 * S.g.I * S.g.ldc <= kKeptBytes);
  const void* kernel = streamed;
  TcPersistArgs T{};
  int threads = kPersistThreads;
  if (S.tc.on) {
    const TcState& t = S.tc;
    T.p = A;
    T.x = TcSide{t.Xa, t.Xb, t.X, t.ldx, S.g.I, t.normX, t.offX, t.redoX, t.n_xt};
    T.y = TcSide{t.Ya, t.Yb, t.Y, t.ldy, S.g.J, t.normY, t.offY, t.redoY, t.n_yt};
    T.d = t.d;
    T.part = t.part;
    T.redo_total = t.redo_total;
    const Coef c = S.coef(eps, P, h.q);
    T.logs[0] = c.logI;
    T.logs[1] = c.logJ;
    T.logs[2] = c.logq;
    T.logs[3] = std::log(P.tau);
    WOTG_CUDA(cudaMemsetAsync(t.redoX, 0, sizeof(int), S.st));
    WOTG_CUDA(cudaMemsetAsync(t.redoY, 0, sizeof(int), S.st));
    kernel = t.kp == 32 ? (gap ? reinterpret_cast<const void*>(tc_persist_kernel<32, true>)
                               : reinterpret_cast<const void*>(tc_persist_kernel<32, false>))
                        : (gap ? reinterpret_cast<const void*>(tc_persist_kernel<64, true>)
                               : reinterpret_cast<const void*>(tc_persist_kernel<64, false>));
    smem = t.kp == 32 ? TcPersist<32>::kAlloc : TcPersist<64>::kAlloc;
    WOTG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    T.vctas = t.ctas_row;
    grid = std::min(grid, t.ctas_row);
    threads = kTcPersistThreads;
  } else {
    const ResidentPlan plan = resident_plan(S.g, grid);
    int room = 0;
    int s = resident_room(&room);
    if (s) return s;
    if (resident_fits(plan, S.g, (size_t)room)) {
      grid = plan.grid;
      rows_cap = plan.rows;
      cols_cap = plan.cols4 * 4;
      smem = plan.bytes;
      threads = kResidentThreads;
      kernel = gap ? reinterpret_cast<const void*>(resident_kernel<true>)
                   : reinterpret_cast<const void*>(resident_kernel<false>);
    }
    const int64_t longest = (std::max(S.g.ldc, S.g.I) + 3) & ~int64_t(3);
    if (streamed_smem + 8 * longest <= room) {
      A.wfloats = (int)longest;
      streamed_smem += 8 * longest;
    }
    if (kernel == streamed) smem = streamed_smem;
  }
  for (;;) {
    WOTG_CUDA(cudaMemsetAsync(&A.ctl->bar, 0, 2 * sizeof(unsigned long long), S.st));
    void* args[] = {S.tc.on ? (void*)&T : (void*)&A, &rows_cap, &cols_cap};
    cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(threads), args, smem, S.st);
    while (e == cudaErrorCooperativeLaunchTooLarge && (threads == kResidentThreads || grid > 1)) {
      // fewer SMs than the device has: a smaller grid, which the streamed and the
      // on-the-fly kernels run on as well
      cudaGetLastError();
      if (threads == kResidentThreads) {
        kernel = streamed;
        threads = kPersistThreads;
        smem = streamed_smem;
      } else {
        grid /= 2;
        T.vctas = std::min(T.vctas, kTcHalves * grid);
      }
      e = cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(threads), args, smem, S.st);
    }
    WOTG_CUDA(e);
    WOTG_LAUNCHED();
    WOTG_CUDA(cudaMemcpyAsync(&h, A.ctl, sizeof(h), cudaMemcpyDeviceToHost, S.st));
    WOTG_CUDA(cudaStreamSynchronize(S.st));
    if (h.err) {
      set_last_message(S.tc.on ? "tensor-core solver: a bounded wait timed out"
                               : "persistent solver: a bounded grid barrier ran out");
      return WOTG_CUDA_ERROR;
    }
    if (h.status != kRunning) break;
  }
  res.iterations = h.it;
  res.checks = h.checks;
  res.absorptions = h.absorptions;
  res.gap = mode == kModeGap ? h.gap_num / h.gap_den : NAN;
  res.eps = h.eps;
  res.max_iter = h.status == kMaxIter;
  res.final_coef = S.coef(h.eps, P, h.q);
  return h.status == kNonfinite ? WOTG_NONFINITE : WOTG_OK;
}

// Row blocks of the column pass: about kColCtasPerSm CTAs of 1024 columns per
// SM. The partition fixes the order of a column's sum, so it stays the same for
// every kernel that walks it. kRowCtasPerSm sizes the standalone row pass.
constexpr int kRowCtasPerSm = 3, kColCtasPerSm = 4;

static Geom make_geom(int64_t I, int64_t J, int64_t ldc) {
  Geom g;
  g.I = I;
  g.J = J;
  g.ldc = ldc;
  const int sms = sm_count();
  const int64_t max_warps = (int64_t)sms * kRowCtasPerSm * 8;
  const int64_t rows_per_warp = (I + max_warps - 1) / max_warps;
  const int64_t warps = (I + rows_per_warp - 1) / rows_per_warp;
  g.row_grid = (int)std::max<int64_t>(1, (warps + 7) / 8);
  const int64_t nv = ldc >> 2;
  g.ncb = (int)std::max<int64_t>(1, (nv + 255) / 256);
  int64_t nrb = std::max<int64_t>(1, ((int64_t)sms * kColCtasPerSm) / g.ncb);
  nrb = std::min<int64_t>(nrb, std::max<int64_t>(1, I / 8));
  int64_t rows_per = (I + nrb - 1) / nrb;
  rows_per = (rows_per + kColRowChunk - 1) / kColRowChunk * kColRowChunk;
  g.rows_per = rows_per;
  g.nrb = (int)((I + rows_per - 1) / rows_per);
  return g;
}

static size_t layout(Bump& b, const Geom& g, Vecs& V) {
  V.u = b.take<double>(g.I);
  V.la = b.take<double>(g.I);
  V.la_old = b.take<double>(g.I);
  V.logp = b.take<double>(g.I);
  V.p = b.take<double>(g.I);
  V.Lrow = b.take<double>(g.I);
  V.v = b.take<double>(g.J);
  V.lb = b.take<double>(g.J);
  V.lb_old = b.take<double>(g.J);
  V.Lcol = b.take<double>(g.J);
  V.rowc = b.take<float4>(g.I);
  V.wrow = b.take<float>(g.I);
  V.wcol = b.take<float>(g.ldc);
  V.wrow_lo = b.take<float>(g.I);
  V.wcol_lo = b.take<float>(g.ldc);
  V.part = b.take<float2>((size_t)g.nrb * g.ldc);
  b.take<unsigned long long>(2);   // unused, like the ints below: the scratch need stays what callers sized for
  V.red = b.take<double>((size_t)kRedBlocks * kNq);
  V.scal = b.take<double>(16);
  b.take<int>(8);
  return b.off + 256;
}

}  // namespace wotg

using namespace wotg;

extern "C" size_t wotg_lse_matvec_workspace_bytes(int64_t I, int64_t J, int64_t ldc) {
  if (I <= 0 || J <= 0 || ldc < J) return 0;
  Geom g = make_geom(I, J, ldc);
  return (size_t)g.nrb * (size_t)ldc * sizeof(float2) + 256;
}

extern "C" int wotg_lse_matvec(const float* C, int64_t I, int64_t J, int64_t ldc, const float* w, float kappa2,
                               int32_t axis, double* L, void* workspace, size_t workspace_bytes, void* stream) {
  if (!C || !w || !L || I <= 0 || J <= 0 || ldc < J || (ldc & 3) || (axis != 0 && axis != 1)) return WOTG_BADARG;
  if ((reinterpret_cast<uintptr_t>(C) & 15) || (axis == 0 && (reinterpret_cast<uintptr_t>(w) & 15)))
    return WOTG_BADARG;
  Geom g = make_geom(I, J, ldc);
  cudaStream_t st = (cudaStream_t)stream;
  if (axis == 0) {
    row_pass_kernel<<<g.row_grid, 256, 0, st>>>(C, g, w, kappa2, L);
    WOTG_LAUNCHED();
    return WOTG_OK;
  }
  if (!workspace || workspace_bytes < wotg_lse_matvec_workspace_bytes(I, J, ldc)) return WOTG_WORKSPACE;
  float2* part = reinterpret_cast<float2*>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~uintptr_t(255));
  col_partial_kernel<<<dim3(g.ncb, g.nrb), 256, 0, st>>>(C, g, w, kappa2, part);
  WOTG_LAUNCHED();
  col_combine_kernel<<<(unsigned)((J + 255) / 256), 256, 0, st>>>(g, part, L);
  WOTG_LAUNCHED();
  return WOTG_OK;
}

static bool tc_requested(const wotg_problem* prob) { return prob->form == WOTG_FORM_ONTHEFLY; }

static int tc_valid(const wotg_problem* prob) {
  if (!tc_requested(prob)) return prob->form == WOTG_FORM_MATERIALIZED ? WOTG_OK : WOTG_BADARG;
  if (!(prob->cost_scale > 0)) return WOTG_BADARG;
  if (!prob->X || !prob->Y || prob->d < 1 || prob->d > tc_max_dim() || prob->ldx < prob->d || prob->ldy < prob->d)
    return WOTG_BADARG;
  return WOTG_OK;
}

static void tc_layout(Bump& b, const wotg_problem* prob, TcState& tc) {
  tc.on = true;
  tc.kp = tc_kp(prob->d);
  tc.n_xt = (int)((prob->I + 127) / 128);
  tc.n_yt = (int)((prob->J + 127) / 128);
  tc.I_pad = (int64_t)tc.n_xt * 128;
  tc.J_pad = (int64_t)tc.n_yt * 128;
  const int slots = sm_count() * std::max(1, tc_ctas_per_sm(tc.kp));
  tc.ctas_row = (int)std::min<int64_t>(slots, (int64_t)tc.n_xt * tc.n_yt);
  tc.ctas_col = (int)std::min<int64_t>(slots, (int64_t)tc.n_yt * tc.n_xt);
  const size_t tb = tc_tile_bytes(tc.kp);
  tc.Xa = reinterpret_cast<__half*>(b.take<unsigned char>(tb * tc.n_xt));
  tc.Xb = reinterpret_cast<__half*>(b.take<unsigned char>(tb * tc.n_xt));
  tc.Ya = reinterpret_cast<__half*>(b.take<unsigned char>(tb * tc.n_yt));
  tc.Yb = reinterpret_cast<__half*>(b.take<unsigned char>(tb * tc.n_yt));
  tc.X = prob->X;
  tc.Y = prob->Y;
  tc.ldx = prob->ldx;
  tc.ldy = prob->ldy;
  tc.d = prob->d;
  tc.normX = b.take<double>(prob->I);
  tc.normY = b.take<double>(prob->J);
  tc.part = b.take<float2>((size_t)(std::max(tc.ctas_row, tc.ctas_col) + std::max(tc.n_xt, tc.n_yt)) * 128 *
                           tc_parts());
  b.take<int>(4);   // unused, as below
  tc.offX = b.take<float>(tc.I_pad);
  tc.offY = b.take<float>(tc.J_pad);
  tc.redoX = b.take<int>(2 + prob->I);
  tc.redoY = b.take<int>(2 + prob->J);
  b.take<int>((size_t)4 * std::max(tc.n_xt, tc.n_yt));   // unused: the scratch need stays what callers sized for
  tc.redo_total = b.take<unsigned long long>(1);
}

// The on-the-fly form's buffers; column forms (coordinates; the bias columns are
// written by the solver) and norms.
static int tc_setup(Bump& b, const wotg_problem* prob, Solver& S) {
  tc_layout(b, prob, S.tc);
  WOTG_CUDA(cudaMemsetAsync(S.tc.redo_total, 0, sizeof(unsigned long long), S.st));
  const float sigma = (float)std::sqrt(prob->cost_scale);
  int s = tc_pack_points(prob->X, prob->I, prob->ldx, prob->d, S.tc.kp, sigma, 0, S.tc.Xb, S.tc.normX, S.st);
  if (s) return s;
  return tc_pack_points(prob->Y, prob->J, prob->ldy, prob->d, S.tc.kp, sigma, 0, S.tc.Yb, S.tc.normY, S.st);
}

extern "C" size_t wotg_problem_workspace_bytes(const wotg_problem* prob) {
  if (!prob || prob->I <= 0 || prob->J <= 0 || prob->ldc < prob->J || tc_valid(prob) != WOTG_OK) return 0;
  Geom g = make_geom(prob->I, prob->J, prob->ldc);
  Bump b{nullptr, 0};
  Vecs V{};
  b.take<double>(prob->I);
  size_t n = layout(b, g, V);
  if (tc_requested(prob)) {
    TcState tc{};
    tc_layout(b, prob, tc);
    n = b.off + 256;
  }
  return n;
}

extern "C" size_t wotg_solve_workspace_bytes(int64_t I, int64_t J, int64_t ldc) {
  if (I <= 0 || J <= 0 || ldc < J) return 0;
  Geom g = make_geom(I, J, ldc);
  Bump b{nullptr, 0};
  Vecs V{};
  // extra I doubles: learned-growth carry between growth iterations
  b.take<double>(I);
  return layout(b, g, V);
}

extern "C" int wotg_compute_transport_matrix(const wotg_problem* prob, const wotg_params* params,
                                             double* tmap, double* learned_growth, double* row_sums,
                                             double* u_bar, double* v_bar, wotg_stats* stats,
                                             void* workspace, size_t workspace_bytes, void* stream) {
  if (!prob || !params) return WOTG_BADARG;
  const wotg_params P = *params;
  const int64_t I = prob->I, J = prob->J, ldc = prob->ldc;
  if (I <= 0 || J <= 0 || ldc < J || (ldc & 3) || !prob->C || !prob->G) return WOTG_BADARG;
  if ((reinterpret_cast<uintptr_t>(prob->C) & 15) != 0) return WOTG_BADARG;
  if (!(P.epsilon > 0) || !(P.epsilon0 > 0) || P.growth_iters < 1) return WOTG_BADARG;
  if (P.solver == WOTG_SOLVER_DUALITY_GAP) {
    if (P.batch_size < 1) return WOTG_BADARG;
  } else if (P.solver == WOTG_SOLVER_FIXED_ITERS) {
    if (P.scaling_iter < 1 || P.extra_iter < 0) return WOTG_BADARG;
  } else {
    return WOTG_BADARG;
  }
  if (tc_valid(prob) != WOTG_OK) return WOTG_BADARG;
  if (!workspace || workspace_bytes < wotg_problem_workspace_bytes(prob)) return WOTG_WORKSPACE;

  Geom g = make_geom(I, J, ldc);
  // layout() leaves 256 bytes of slack for aligning the caller's base pointer
  Bump b{reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~uintptr_t(255)), 0};
  double* carry = b.take<double>(I);
  Vecs V{};
  layout(b, g, V);
  cudaStream_t st = (cudaStream_t)stream;
  Solver S{prob->C, g, V, st, prob->cost_scale, TcState{}};
  if (tc_requested(prob)) {
    int s = tc_setup(b, prob, S);
    if (s) return s;
  }

  wotg_stats total{};
  int status = WOTG_OK;
  const double* G = prob->G;
  for (int gi = 0; gi < P.growth_iters; ++gi) {
    if (learned_growth) {
      WOTG_CUDA(cudaMemcpyAsync(learned_growth + (int64_t)gi * I, G, I * sizeof(double),
                                cudaMemcpyDeviceToDevice, st));
    }
    init_kernel<<<S.vec_blocks(std::max(I, ldc)), 256, 0, st>>>(g, V, G);
    WOTG_LAUNCHED();
    SolveResult res;
    int s = solve_persistent(S, P, P.solver == WOTG_SOLVER_DUALITY_GAP ? kModeGap : kModeFixed, P.epsilon, 0, res);
    total.iterations += res.iterations;
    total.absorptions += res.absorptions;
    total.checks += res.checks;
    total.gap = res.gap;
    total.final_epsilon = res.eps;
    if (s == WOTG_NONFINITE) {
      status = WOTG_NONFINITE;
      break;
    }
    if (s) return s;
    if (res.max_iter) {
      total.hit_max_iter = 1;
      status = WOTG_MAX_ITER;
    }
    const bool last = gi == P.growth_iters - 1;
    if (!last) {
      s = S.outputs(res.final_coef, res.max_iter, nullptr, carry, nullptr, nullptr);
      if (s) return s;
      G = carry;
    } else {
      s = S.outputs(res.final_coef, res.max_iter, tmap, row_sums, u_bar, v_bar);
      if (s) return s;
    }
  }
  WOTG_CUDA(cudaStreamSynchronize(st));
  int s = S.exact_rows(&total.exact_rows);
  if (s) return s;
  if (stats) *stats = total;
  return status;
}

// Warm-started fixed-epsilon iterations (no counterpart in the reference; its
// iterations at the final epsilon are optimal_transport.py:131-141): from
// absorbed potentials (u_bar, v_bar), n_iter iterations of the reference's a/b
// updates with tau-absorption at `epsilon`, potentials written back in place.
// Polishes a solve stopped on the duality gap towards the exact optimum (used
// before differentiating the objective).
extern "C" int wotg_refine_potentials(const wotg_problem* prob, const wotg_params* params, double epsilon,
                                      int32_t n_iter, double* u_bar, double* v_bar, wotg_stats* stats,
                                      void* workspace, size_t workspace_bytes, void* stream) {
  if (!prob || !params || !u_bar || !v_bar || n_iter < 0 || !(epsilon > 0)) return WOTG_BADARG;
  const wotg_params P = *params;
  const int64_t I = prob->I, J = prob->J, ldc = prob->ldc;
  if (I <= 0 || J <= 0 || ldc < J || (ldc & 3) || !prob->C || !prob->G) return WOTG_BADARG;
  if ((reinterpret_cast<uintptr_t>(prob->C) & 15) != 0) return WOTG_BADARG;
  if (tc_valid(prob) != WOTG_OK) return WOTG_BADARG;
  if (!workspace || workspace_bytes < wotg_problem_workspace_bytes(prob)) return WOTG_WORKSPACE;
  Geom g = make_geom(I, J, ldc);
  Bump b{reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~uintptr_t(255)), 0};
  b.take<double>(I);
  Vecs V{};
  layout(b, g, V);
  cudaStream_t st = (cudaStream_t)stream;
  Solver S{prob->C, g, V, st, prob->cost_scale, TcState{}};
  if (tc_requested(prob)) {
    int s = tc_setup(b, prob, S);
    if (s) return s;
  }
  init_kernel<<<S.vec_blocks(std::max(I, ldc)), 256, 0, st>>>(g, V, prob->G);
  WOTG_LAUNCHED();
  load_potentials_kernel<<<S.vec_blocks(I + J), 256, 0, st>>>(g, V, u_bar, v_bar, 1.0 / epsilon);
  WOTG_LAUNCHED();
  SolveResult res;
  int s = solve_persistent(S, P, kModeRefine, epsilon, n_iter, res);
  if (s) return s;
  const Coef c = res.final_coef;
  s = S.outputs(c, false, nullptr, nullptr, u_bar, v_bar);
  if (s) return s;
  WOTG_CUDA(cudaStreamSynchronize(st));
  wotg_stats out{};
  out.iterations = n_iter;
  out.final_epsilon = epsilon;
  out.gap = NAN;
  out.absorptions = res.absorptions;
  s = S.exact_rows(&out.exact_rows);
  if (s) return s;
  if (stats) *stats = out;
  return WOTG_OK;
}

// ---------------------------------------------------------------------------
// No-allocation variant of wotg_compute_transport_matrix.
//
// Some callers cannot call cudaMalloc: hosts whose device memory is owned by
// another allocator or pool (a JVM or Go service handing out pre-sized
// buffers, a framework that forbids raw device allocations) and code paths
// where cudaMalloc's implicit device synchronisation is not acceptable. They
// still pass every input and output buffer, but get the solver's scratch from
// the file-scope array below instead of a caller workspace.
//
// The array is wotg_noalloc_scratch_bytes() = 32 MiB on every device that
// loads this module and stays allocated until the process exits. Its device
// address is looked up once per device, on that device's first call, with
// cudaGetSymbolAddress (host code cannot use the symbol itself: on the host it
// names a stand-in, not device memory); make that first call before any stream
// capture. The looked-up address is cached per device for the life of the
// process; it does not survive cudaDeviceReset (or any other teardown of the
// device's primary context), after which this entry point must not be called
// again in the process. All calls share the array: calls whose work overlaps
// on the GPU (other streams, other host threads) race on it, so serialise
// them. The solver re-initialises everything it reads from the scratch at the
// start of each solve (state vectors, control words, the tensor-core
// form's packed points), so no clearing between calls is needed.
// ---------------------------------------------------------------------------
namespace {
constexpr size_t kNoAllocScratchBytes = size_t(32) << 20;
__device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];
constexpr int kNoAllocMaxDevices = 64;
std::atomic<void*> g_noalloc_ptr[kNoAllocMaxDevices] = {};
}  // namespace

extern "C" size_t wotg_noalloc_scratch_bytes(void) { return kNoAllocScratchBytes; }

extern "C" int wotg_compute_transport_matrix_noalloc(const wotg_problem* prob, const wotg_params* params,
                                                     double* tmap, double* learned_growth, double* row_sums,
                                                     double* u_bar, double* v_bar, wotg_stats* stats,
                                                     void* stream) {
  if (!prob || !params) return WOTG_BADARG;
  const int64_t I = prob->I, J = prob->J, ldc = prob->ldc;
  if (I <= 0 || J <= 0 || ldc < J || (ldc & 3) || !prob->C || !prob->G || tc_valid(prob) != WOTG_OK)
    return WOTG_BADARG;
  const size_t need = wotg_problem_workspace_bytes(prob);
  if (need == 0) return WOTG_BADARG;
  if (need > kNoAllocScratchBytes) {
    char msg[256];
    snprintf(msg, sizeof(msg),
             "wotg_compute_transport_matrix_noalloc: a %lld x %lld problem needs %zu bytes of scratch, "
             "more than the %zu-byte static array",
             (long long)I, (long long)J, need, kNoAllocScratchBytes);
    wotg::set_last_message(msg);
    return WOTG_TOO_LARGE;
  }
  int dev = 0;
  WOTG_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoAllocMaxDevices) return WOTG_BADARG;
  void* scratch = g_noalloc_ptr[dev].load(std::memory_order_acquire);
  if (!scratch) {
    // set-up, once per device with that device current (two threads racing here
    // look up and store the same address)
    WOTG_CUDA(cudaGetSymbolAddress(&scratch, g_noalloc_scratch));
    g_noalloc_ptr[dev].store(scratch, std::memory_order_release);
  }
  return wotg_compute_transport_matrix(prob, params, tmap, learned_growth, row_sums, u_bar, v_bar, stats,
                                       scratch, kNoAllocScratchBytes, stream);
}
