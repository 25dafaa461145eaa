// wotg_tmap.cu — population transport through dense FP64 couplings (sm_103a).
//
// Replaces the NumPy products of the reference's TransportMapModel:
//   push_forward: p = p @ tmap.X                 wot/tmap/transport_map_model.py:290
//   pull_back:    p = (tmap.X @ p.T).T           wot/tmap/transport_map_model.py:356
// plus the optional row normalisation p = (p.T / p.sum(axis=1)).T (:291-292, :357-358).
// Accumulation is FP64 like the reference (k populations at a time, k <= 16 per
// pass); X is read once per pass with coalesced loads.
#include <algorithm>
#include <type_traits>

#include "wotg_common.cuh"

namespace wotg {

constexpr int kMaxK = 16;

// Both kernels take exactly KC populations (P and out at the first of them). What
// bounds them is FP64 FMAs, 64 cycles each on an SM's quarter: with KC = 16 and the
// populations past k predicated off, eight of them cost as much as sixteen (5003 x
// 7001: 1.5 ms pull, 1.1 ms push; the FMAs of eight take 0.5 ms).

// out[r][i] = sum_j X[i][j] P[r][j]; one warp per row i of X, the loads of two steps
// ahead of their FMAs.
template <int KC>
__global__ void __launch_bounds__(256) pull_kernel(const double* __restrict__ X, int64_t I, int64_t J,
                                                   const double* __restrict__ P, double* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = warp; i < I; i += nwarps) {
    double acc[KC];
#pragma unroll
    for (int r = 0; r < KC; ++r) acc[r] = 0.0;
    const double* row = X + i * J;
    int64_t j = lane;
    for (; j - lane + 64 <= J; j += 64) {   // whole steps of the warp: a split one would take its FMAs twice
      const double x0 = row[j], x1 = row[j + 32];
      double p0[KC], p1[KC];
#pragma unroll
      for (int r = 0; r < KC; ++r) {
        p0[r] = __ldg(P + r * J + j);
        p1[r] = __ldg(P + r * J + j + 32);
      }
#pragma unroll
      for (int r = 0; r < KC; ++r) acc[r] = fma(x0, p0[r], acc[r]);
#pragma unroll
      for (int r = 0; r < KC; ++r) acc[r] = fma(x1, p1[r], acc[r]);
    }
    for (; j < J; j += 32) {
      const double x = row[j];
#pragma unroll
      for (int r = 0; r < KC; ++r) acc[r] = fma(x, __ldg(P + r * J + j), acc[r]);
    }
#pragma unroll
    for (int r = 0; r < KC; ++r) {
      const double t = warp_sum(acc[r]);
      if (lane == 0) out[r * I + i] = t;
    }
  }
}

// out[r][j] += sum_{i in block rows} P[r][i] X[i][j]; thread per column, grid.y
// splits the rows, FP64 atomics merge the row blocks.
template <int KC>
__global__ void __launch_bounds__(256) push_kernel(const double* __restrict__ X, int64_t I, int64_t J,
                                                   const double* __restrict__ P, int64_t rows_per,
                                                   double* __restrict__ out) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.y * rows_per;
  const int64_t r1 = min(I, r0 + rows_per);
  if (j >= J) return;
  double acc[KC];
#pragma unroll
  for (int r = 0; r < KC; ++r) acc[r] = 0.0;
  const double* x = X + r0 * J + j;
#pragma unroll 2
  for (int64_t i = r0; i < r1; ++i, x += J) {
    const double xi = *x;
#pragma unroll
    for (int r = 0; r < KC; ++r) acc[r] = fma(__ldg(P + r * I + i), xi, acc[r]);
  }
#pragma unroll
  for (int r = 0; r < KC; ++r) atomicAdd(out + r * J + j, acc[r]);
}

// Calls f with the number of populations as a compile-time constant.
template <int KC = kMaxK, class F>
static void with_count(int k, const F& f) {
  if constexpr (KC > 1) {
    if (k < KC) return with_count<KC - 1>(k, f);
  }
  f(std::integral_constant<int, KC>{});
}

// Divide each of the k rows (length n) by its sum; one CTA per row.
__global__ void normalize_rows_kernel(double* __restrict__ out, int64_t n) {
  __shared__ double sh[32];
  double* row = out + (int64_t)blockIdx.x * n;
  double s = 0.0;
  for (int64_t t = threadIdx.x; t < n; t += blockDim.x) s += row[t];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0.0;
    t = warp_sum(t);
    if (threadIdx.x == 0) sh[0] = t;
  }
  __syncthreads();
  const double total = sh[0];
  for (int64_t t = threadIdx.x; t < n; t += blockDim.x) row[t] = row[t] / total;
}

}  // namespace wotg

using namespace wotg;

extern "C" int wotg_apply_coupling_f64(const double* X, int64_t I, int64_t J, const double* P, int32_t k,
                                       int32_t transpose, int32_t normalize, double* out, void* stream) {
  if (!X || !P || !out || I <= 0 || J <= 0 || k <= 0) return WOTG_BADARG;
  cudaStream_t st = (cudaStream_t)stream;
  const int sms = sm_count();
  if (transpose) {
    const int grid = (int)std::min<int64_t>((I + 7) / 8, (int64_t)sms * 8);
    for (int k0 = 0; k0 < k; k0 += kMaxK) {
      with_count(std::min(k - k0, kMaxK), [&](auto kc) {
        pull_kernel<kc><<<grid, 256, 0, st>>>(X, I, J, P + k0 * J, out + k0 * I);
      });
      WOTG_LAUNCHED();
    }
    if (normalize) {
      normalize_rows_kernel<<<k, 256, 0, st>>>(out, I);
      WOTG_LAUNCHED();
    }
  } else {
    WOTG_CUDA(cudaMemsetAsync(out, 0, (size_t)k * J * sizeof(double), st));
    const int64_t ncb = (J + 255) / 256;
    int64_t nrb = std::max<int64_t>(1, ((int64_t)sms * 8) / ncb);
    nrb = std::min<int64_t>(nrb, std::max<int64_t>(1, I / 16));
    nrb = std::min<int64_t>(nrb, 65535);
    const int64_t rows_per = (I + nrb - 1) / nrb;
    nrb = (I + rows_per - 1) / rows_per;
    for (int k0 = 0; k0 < k; k0 += kMaxK) {
      with_count(std::min(k - k0, kMaxK), [&](auto kc) {
        push_kernel<kc><<<dim3((unsigned)ncb, (unsigned)nrb), 256, 0, st>>>(X, I, J, P + k0 * I, rows_per, out + k0 * J);
      });
      WOTG_LAUNCHED();
    }
    if (normalize) {
      normalize_rows_kernel<<<k, 256, 0, st>>>(out, J);
      WOTG_LAUNCHED();
    }
  }
  return WOTG_OK;
}
