// wotg_gemm.cu — dense FP64 product for chaining transport maps (sm_103a).
//
// The long-range coupling of the reference is the matrix product of
// consecutive dense maps (wot/tmap/util.py:74-94, np.dot of tmap_0.X with the
// rows of tmap_1.X that tmap_0's columns name; chained by
// wot/tmap/chaining.py:4-40). Here: C (M x N) = A (M x K) . B[rows] (K x N),
// row-major FP64, the rows of B gathered by an optional index.
//
// FP64 runs at 1/64 of the FP32 rate on this part, so the product is bound by
// the FP64 FMA pipe, not by memory: each CTA computes a 64 x 64 tile of C from
// 64 x 16 and 16 x 64 tiles of A and B staged in shared memory (double
// buffered), every thread a 4 x 4 block of C in registers, i.e. 16 FMAs per 8
// shared-memory loads.
#include <algorithm>

#include "wotg_common.cuh"

namespace wotg {

constexpr int kGemmTile = 64;
constexpr int kGemmK = 16;
constexpr int kGemmThreads = 256;

__global__ void __launch_bounds__(kGemmThreads) gemm_f64_kernel(const double* __restrict__ A, int64_t lda,
                                                                const double* __restrict__ B, int64_t ldb,
                                                                const int64_t* __restrict__ b_rows,
                                                                double* __restrict__ C, int64_t ldc, int64_t M,
                                                                int64_t N, int64_t K) {
  __shared__ double sA[2][kGemmK][kGemmTile + 1];   // A tile transposed: [k][m], padded against bank conflicts
  __shared__ double sB[2][kGemmK][kGemmTile];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;           // thread (ty, tx) owns rows 4 ty.., columns 4 tx..
  const int64_t m0 = (int64_t)blockIdx.y * kGemmTile, n0 = (int64_t)blockIdx.x * kGemmTile;
  double acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;

  // loads of one K-chunk: A is 64 x 16 (4 per thread), B is 16 x 64 (4 per thread)
  auto load = [&](int buf, int64_t k0) {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int idx = tid + t * kGemmThreads;       // 0 .. 1023
      const int am = idx >> 4, ak = idx & 15;       // A: row am, column ak
      const int64_t gm = m0 + am, gk = k0 + ak;
      sA[buf][ak][am] = (gm < M && gk < K) ? A[gm * lda + gk] : 0.0;
      const int bk = idx >> 6, bn = idx & 63;       // B: row bk, column bn
      const int64_t gk2 = k0 + bk, gn = n0 + bn;
      double v = 0.0;
      if (gk2 < K && gn < N) {
        const int64_t r = b_rows ? b_rows[gk2] : gk2;
        v = B[r * ldb + gn];
      }
      sB[buf][bk][bn] = v;
    }
  };

  const int64_t nk = (K + kGemmK - 1) / kGemmK;
  load(0, 0);
  __syncthreads();
  for (int64_t c = 0; c < nk; ++c) {
    const int buf = (int)(c & 1);
    if (c + 1 < nk) load(buf ^ 1, (c + 1) * kGemmK);
#pragma unroll
    for (int k = 0; k < kGemmK; ++k) {
      double a[4], b[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) a[t] = sA[buf][k][ty * 4 + t];
#pragma unroll
      for (int t = 0; t < 4; ++t) b[t] = sB[buf][k][tx * 4 + t];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t gn = n0 + tx * 4 + j;
      if (gn < N) C[gm * ldc + gn] = acc[i][j];
    }
  }
}

// Narrow products (N, K <= 64; the orthonormalisations of a PCA, n x 40 by 40 x 40): a
// thread per element of C, B in shared memory, the sum over k in the same order. What
// bounds it: the FP64 FMAs, of which a 64 x 64 tile does 1.9 times as many for N = K =
// 40 and gives them to 71 SMs (53 us at n = 4500); warps full of elements on every
// SM's four FP64 units leave 12 us.
constexpr int kNarrow = 64, kNarrowThreads = 128;
__global__ void __launch_bounds__(kNarrowThreads) gemm_narrow_kernel(const double* __restrict__ A, int64_t lda,
                                                                     const double* __restrict__ B, int64_t ldb,
                                                                     const int64_t* __restrict__ b_rows,
                                                                     double* __restrict__ C, int64_t ldc, int64_t M,
                                                                     int N, int K) {
  __shared__ double sB[kNarrow * kNarrow];
  for (int e = threadIdx.x; e < K * N; e += kNarrowThreads) {
    const int k = e / N;
    sB[e] = B[(b_rows ? b_rows[k] : k) * ldb + (e - k * N)];
  }
  __syncthreads();
  const int64_t total = M * N;
  for (int64_t e = (int64_t)blockIdx.x * kNarrowThreads + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * kNarrowThreads) {
    const int64_t i = e / N;
    const int j = (int)(e - i * N);
    const double* a = A + i * lda;
    double s = 0.0;
    int k = 0;
    for (; k + 8 <= K; k += 8) {
      double v[8];
#pragma unroll
      for (int t = 0; t < 8; ++t) v[t] = a[k + t];
#pragma unroll
      for (int t = 0; t < 8; ++t) s = fma(v[t], sB[(k + t) * N + j], s);
    }
    for (; k < K; ++k) s = fma(a[k], sB[k * N + j], s);
    C[i * ldc + j] = s;
  }
}

}  // namespace wotg

using namespace wotg;

// Whether the rows x cols block at x (leading dimension ld) shares memory with the one at c.
static bool overlaps(const double* x, int64_t ld, int64_t rows, int64_t cols, const double* c, int64_t ldc,
                     int64_t c_rows, int64_t c_cols) {
  const uintptr_t x0 = reinterpret_cast<uintptr_t>(x), c0 = reinterpret_cast<uintptr_t>(c);
  const uintptr_t x1 = x0 + 8 * (uint64_t)((rows - 1) * ld + cols), c1 = c0 + 8 * (uint64_t)((c_rows - 1) * ldc + c_cols);
  return x0 < c1 && c0 < x1;
}

extern "C" int wotg_gemm_f64(const double* A, int64_t lda, const double* B, int64_t ldb, const int64_t* b_rows,
                             double* C, int64_t ldc, int64_t M, int64_t N, int64_t K, void* stream) {
  if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0 || lda < K || ldb < N || ldc < N) return WOTG_BADARG;
  const int64_t gx = (N + kGemmTile - 1) / kGemmTile, gy = (M + kGemmTile - 1) / kGemmTile;
  if (gx > 2147483647LL || gy > 65535) return WOTG_BADARG;
  // a product in place stays with the tiles: with N <= 64 a CTA has read its rows of A when
  // it writes them, while the narrow kernel's threads share them with others'
  if (N <= kNarrow && K <= kNarrow && !overlaps(A, lda, M, K, C, ldc, M, N) &&
      (b_rows || !overlaps(B, ldb, K, N, C, ldc, M, N))) {
    const int64_t blocks = std::min<int64_t>((M * N + kNarrowThreads - 1) / kNarrowThreads, (int64_t)sm_count() * 12);
    gemm_narrow_kernel<<<(unsigned)blocks, kNarrowThreads, 0, (cudaStream_t)stream>>>(A, lda, B, ldb, b_rows, C, ldc, M,
                                                                                     (int)N, (int)K);
    WOTG_LAUNCHED();
    return WOTG_OK;
  }
  gemm_f64_kernel<<<dim3((unsigned)gx, (unsigned)gy), kGemmThreads, 0, (cudaStream_t)stream>>>(
      A, lda, B, ldb, b_rows, C, ldc, M, N, K);
  WOTG_LAUNCHED();
  return WOTG_OK;
}
