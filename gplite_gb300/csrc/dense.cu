// Dense FP64 linear algebra for the GP hot path (column-major, lower factors).
//
// Replaces the LAPACK/BLAS calls the reference makes from R: chol (dpotrf,
// R/laplace.R:28, R/ep.R:38, R/linear_algebra.R:28), forwardsolve/backsolve
// (dtrsv/dtrsm, R/laplace.R:29, R/gp_pred.R:218) and %*% (dgemm/dgemv,
// R/laplace.R:30, R/gp_pred.R:209).
//
// The factorisation is blocked right-looking with NB = 64: the diagonal block
// is factored and inverted by one cluster of CTAs (diag.cu; the inverses serve the
// solves); the panel below is solved by row-parallel substitution,
// which stays backward stable when a diagonal block is ill-conditioned (FITC's
// K_z); the trailing update is a lower-only GEMM on the FP64 pipe. (FP64 fits of
// SLICED_MIN points and more factor on the tensor cores, mixed_la.cu.) The triangular solves
// are single launches ordered by the solution's entries, which are their own flags.
#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "dfloat.cuh"
#include "fp64math.cuh"

namespace gpgp {

// ---------------------------------------------------------------------------
// FP64 GEMM: C = alpha op(A) op(B) + beta C, 64x64 tiles, 4x4 per thread
// ---------------------------------------------------------------------------
constexpr int GBM = 64, GBN = 64, GBK = 16;

template <bool TA, bool TB>
__global__ void __launch_bounds__(256) gemm64_kernel(int64_t M, int64_t N, int64_t K, double alpha,
                                                     const double *__restrict__ A, int64_t lda,
                                                     const double *__restrict__ B, int64_t ldb,
                                                     double beta, double *__restrict__ C,
                                                     int64_t ldc, int lower_only, int tri_mode,
                                                     int64_t sA, int64_t sB, int64_t sC, int64_t kchunk) {
  const int64_t bm = blockIdx.x, bn = blockIdx.y;
  // blockIdx.z: the problem of a batch (strides sA, sB, sC), or with kchunk > 0 the
  // K range [z kchunk, (z + 1) kchunk) of one product whose partial goes to C + z sC
  A += blockIdx.z * sA;
  B += blockIdx.z * sB;
  C += blockIdx.z * sC;
  int64_t kend = K;
  const int64_t row0 = bm * GBM, col0 = bn * GBN;
  if (lower_only && col0 > row0 + GBM - 1) return;
  __shared__ double As[GBK][GBM + 1];
  __shared__ double Bs[GBK][GBN + 1];
  const int tid = threadIdx.x;
  const int tx = tid % 16, ty = tid / 16;
  double acc[4][4];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
  int64_t kstart = 0;
  if (tri_mode == 1) kstart = (row0 / GBK) * GBK;  // W^T W with W lower: k >= row
  if (kchunk > 0) {
    const int64_t kb = (int64_t)blockIdx.z * kchunk;
    kstart = kstart > kb ? kstart : kb;
    kend = kb + kchunk < K ? kb + kchunk : K;
  }
  for (int64_t k0 = kstart; k0 < kend; k0 += GBK) {
    // load A tile: op(A) is M x K
#pragma unroll
    for (int e = 0; e < (GBM * GBK) / 256; ++e) {
      int idx = tid + e * 256;
      int r, kk;
      if (!TA) {
        r = idx % GBM;
        kk = idx / GBM;
      } else {
        kk = idx % GBK;
        r = idx / GBK;
      }
      int64_t gr = row0 + r, gk = k0 + kk;
      double v = 0.0;
      if (gr < M && gk < kend) v = TA ? A[gk + gr * lda] : A[gr + gk * lda];
      As[kk][r] = v;
    }
    // load B tile: op(B) is K x N
#pragma unroll
    for (int e = 0; e < (GBN * GBK) / 256; ++e) {
      int idx = tid + e * 256;
      int c, kk;
      if (!TB) {
        kk = idx % GBK;
        c = idx / GBK;
      } else {
        c = idx % GBN;
        kk = idx / GBN;
      }
      int64_t gc = col0 + c, gk = k0 + kk;
      double v = 0.0;
      if (gc < N && gk < kend) v = TB ? B[gc + gk * ldb] : B[gk + gc * ldb];
      Bs[kk][c] = v;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GBK; ++kk) {
      double a[4], b[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        a[q] = As[kk][tx + 16 * q];
        b[q] = Bs[kk][ty + 16 * q];
      }
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[p][q] = fma(a[p], b[q], acc[p][q]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int p = 0; p < 4; ++p) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      int64_t r = row0 + tx + 16 * p, c = col0 + ty + 16 * q;
      if (r < M && c < N && (!lower_only || r >= c)) {
        double *dst = C + r + c * ldc;
        *dst = (beta == 0.0) ? alpha * acc[p][q] : alpha * acc[p][q] + beta * *dst;
      }
    }
  }
}

// C = alpha sum_z P_z + beta C over the split-K partials (fixed order); go_on: the sum goes
// on from the one in C (alpha 1, beta 0), as if the partials had followed each other
__global__ void splitk_reduce_kernel(int64_t M, int64_t N, int nz, const double *__restrict__ P,
                                     double alpha, double beta, double *__restrict__ C, int64_t ldc,
                                     int lower_only, int go_on) {
  const int64_t MN = M * N;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < MN;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = idx % M, c = idx / M;
    if (lower_only && r < c) continue;
    double *dst = C + r + c * ldc;
    double s = go_on ? *dst : 0.0;
    for (int z = 0; z < nz; ++z) s += P[idx + z * MN];
    *dst = (beta == 0.0) ? alpha * s : alpha * s + beta * *dst;
  }
}

void splitk_reduce(cudaStream_t s, int64_t M, int64_t N, int nz, const double *P, double alpha, double beta,
                   double *C, int64_t ldc, bool lower_only, bool go_on) {
  splitk_reduce_kernel<<<(unsigned)std::min<int64_t>((M * N + 255) / 256, 4096), 256, 0, s>>>(
      M, N, nz, P, alpha, beta, C, ldc, lower_only ? 1 : 0, go_on ? 1 : 0);
  GPGP_CHECK_LAUNCH();
}

template <bool TA, bool TB>
static void launch_gemm64(cudaStream_t s, dim3 grid, int64_t M, int64_t N, int64_t K, double alpha,
                          const double *A, int64_t lda, const double *B, int64_t ldb, double beta, double *C,
                          int64_t ldc, int lo, int tri_mode, int64_t sA, int64_t sB, int64_t sC, int64_t kchunk) {
  double fl = 0.0;
  if (tl_kt) {  // executed FP64 arithmetic of the tiles this launch runs
    for (int64_t bm = 0; bm < (int64_t)grid.x; ++bm)
      for (int64_t bn = 0; bn < (int64_t)grid.y; ++bn) {
        const int64_t row0 = bm * GBM, col0 = bn * GBN;
        if (lo && col0 > row0 + GBM - 1) continue;
        const int64_t ks = tri_mode == 1 ? (row0 / GBK) * GBK : 0;
        fl += 2.0 * GBM * GBN * (double)std::max<int64_t>(0, K - ks);
      }
    if (kchunk == 0) fl *= (double)grid.z;
  }
  KTScope kts(GPGP_KPROF_GEMM64, s, fl);
  gemm64_kernel<TA, TB><<<grid, 256, 0, s>>>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, lo, tri_mode, sA,
                                             sB, sC, kchunk);
  GPGP_CHECK_LAUNCH();
}

static void gemm64_dispatch(cudaStream_t s, bool ta, bool tb, dim3 grid, int64_t M, int64_t N, int64_t K,
                            double alpha, const double *A, int64_t lda, const double *B, int64_t ldb,
                            double beta, double *C, int64_t ldc, int lo, int tri_mode, int64_t sA, int64_t sB,
                            int64_t sC, int64_t kchunk) {
  if (!ta && !tb)
    launch_gemm64<false, false>(s, grid, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, lo, tri_mode, sA, sB, sC, kchunk);
  else if (!ta && tb)
    launch_gemm64<false, true>(s, grid, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, lo, tri_mode, sA, sB, sC, kchunk);
  else if (ta && !tb)
    launch_gemm64<true, false>(s, grid, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, lo, tri_mode, sA, sB, sC, kchunk);
  else
    launch_gemm64<true, true>(s, grid, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, lo, tri_mode, sA, sB, sC, kchunk);
}

// Small products (few 64 x 64 tiles, short K): one thread per element of C, so
// that the FP64 work spreads over many SMs instead of a few tile CTAs (an FP64
// warp instruction holds its sub-partition for 64 cycles on this part). A CTA is a warp
// per sub-partition, 32 x 4 elements, whose operands come 64 K at a time through shared
// memory: all of a chunk's loads are in flight at once (a load for each term from the L2
// took 24 us for 256 x 64 x 64, this 7).
constexpr int SG_N = 4, SG_K = 64;

__global__ void __launch_bounds__(128) gemm64_small_kernel(int64_t M, int64_t N, int64_t K, double alpha,
                                                           const double *__restrict__ A, int64_t lda, int ta,
                                                           const double *__restrict__ B, int64_t ldb, int tb,
                                                           double beta, double *__restrict__ C, int64_t ldc,
                                                           int lower) {
  __shared__ double As[SG_K][33], Bs[SG_K][SG_N + 1];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int64_t i0 = (int64_t)blockIdx.x * 32, j0 = (int64_t)blockIdx.y * SG_N;
  if (lower && j0 > i0 + 31) return;
  const int64_t i = i0 + lane, j = j0 + w;
  const bool mine = i < M && j < N && !(lower && j > i);
  const double c = mine && beta != 0.0 ? C[i + j * ldc] : 0.0;
  double s0 = 0.0, s1 = 0.0;
  for (int64_t k0 = 0; k0 < K; k0 += SG_K) {
    const int kn = (int)(K - k0 < SG_K ? K - k0 : SG_K);
    double ra[32 * SG_K / 128], rb[SG_N * SG_K / 128];
#pragma unroll
    for (int t = 0; t < 32 * SG_K / 128; ++t) {
      const int idx = tid + 128 * t, r = ta ? idx / SG_K : idx & 31, k = ta ? idx % SG_K : idx >> 5;
      ra[t] = k < kn && i0 + r < M ? A[ta ? k0 + k + (i0 + r) * lda : i0 + r + (k0 + k) * lda] : 0.0;
    }
#pragma unroll
    for (int t = 0; t < SG_N * SG_K / 128; ++t) {
      const int idx = tid + 128 * t, r = tb ? idx & (SG_N - 1) : idx / SG_K, k = tb ? idx / SG_N : idx % SG_K;
      rb[t] = k < kn && j0 + r < N ? B[tb ? j0 + r + (k0 + k) * ldb : k0 + k + (j0 + r) * ldb] : 0.0;
    }
    if (k0 > 0) __syncthreads();
#pragma unroll
    for (int t = 0; t < 32 * SG_K / 128; ++t) {
      const int idx = tid + 128 * t;
      As[ta ? idx % SG_K : idx >> 5][ta ? idx / SG_K : idx & 31] = ra[t];
    }
#pragma unroll
    for (int t = 0; t < SG_N * SG_K / 128; ++t) {
      const int idx = tid + 128 * t;
      Bs[tb ? idx / SG_N : idx % SG_K][tb ? idx & (SG_N - 1) : idx / SG_K] = rb[t];
    }
    __syncthreads();
    if (mine) {
      int k = 0;
#pragma unroll 4
      for (; k + 1 < kn; k += 2) {
        s0 = fma(As[k][lane], Bs[k][w], s0);
        s1 = fma(As[k + 1][lane], Bs[k + 1][w], s1);
      }
      if (k < kn) s0 = fma(As[k][lane], Bs[k][w], s0);
    }
  }
  if (!mine) return;
  const double v = alpha * (s0 + s1);
  C[i + j * ldc] = (beta == 0.0) ? v : v + beta * c;
}

void gemm64_batched(cudaStream_t s, bool ta, bool tb, int64_t M, int64_t N, int64_t K, double alpha,
                    const double *A, int64_t lda, int64_t sA, const double *B, int64_t ldb, int64_t sB,
                    double beta, double *C, int64_t ldc, int64_t sC, int64_t batch, bool lower_only,
                    int tri_mode) {
  if (M <= 0 || N <= 0 || batch <= 0) return;
  dim3 grid((unsigned)((M + GBM - 1) / GBM), (unsigned)((N + GBN - 1) / GBN), (unsigned)batch);
  int lo = lower_only ? 1 : 0;
  const int64_t tiles = (int64_t)grid.x * grid.y;
  // few output tiles and a long K (Gram matrices of tall n x M factors): split K
  // over the third grid axis so that every SM gets work, then reduce the
  // partials in a fixed order
  if (batch == 1 && tiles < 152 && K >= 4096) {
    int64_t nz = std::min<int64_t>((2 * 152 + tiles - 1) / tiles, K / 1024);
    const int64_t kchunk = ((K + nz - 1) / nz + GBK - 1) / GBK * GBK;
    nz = (K + kchunk - 1) / kchunk;
    double *P = nullptr;
    GPGP_CUDA(cudaMallocAsync((void **)&P, (size_t)nz * M * N * sizeof(double), s));
    dim3 g2(grid.x, grid.y, (unsigned)nz);
    gemm64_dispatch(s, ta, tb, g2, M, N, K, 1.0, A, lda, B, ldb, 0.0, P, M, 0, tri_mode, 0, 0, M * N, kchunk);
    splitk_reduce(s, M, N, (int)nz, P, alpha, beta, C, ldc, lower_only);
    GPGP_CUDA(cudaFreeAsync(P, s));
    return;
  }
  gemm64_dispatch(s, ta, tb, grid, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, lo, tri_mode, sA, sB, sC, 0);
}

void gemm64(cudaStream_t s, bool ta, bool tb, int64_t M, int64_t N, int64_t K, double alpha,
            const double *A, int64_t lda, const double *B, int64_t ldb, double beta, double *C,
            int64_t ldc, bool lower_only, int tri_mode) {
  // (the batched entry keeps the tile kernel for every batch size, so that a
  // problem's result does not depend on how many others share its launch)
  if (M > 0 && N > 0 && tri_mode == 0 && K <= 256 && ((M + GBM - 1) / GBM) * ((N + GBN - 1) / GBN) < 152) {
    dim3 g((unsigned)((M + 31) / 32), (unsigned)((N + SG_N - 1) / SG_N));
    gemm64_small_kernel<<<g, 128, 0, s>>>(M, N, K, alpha, A, lda, ta ? 1 : 0, B, ldb, tb ? 1 : 0, beta, C, ldc,
                                          lower_only ? 1 : 0);
    GPGP_CHECK_LAUNCH();
    return;
  }
  gemm64_batched(s, ta, tb, M, N, K, alpha, A, lda, 0, B, ldb, 0, beta, C, ldc, 0, 1, lower_only,
                 tri_mode);
}

// ---------------------------------------------------------------------------
// substitution solves for small factors (M x M lower L), as R's forwardsolve /
// backsolve do, on the rows of a column-major n x M matrix
// ---------------------------------------------------------------------------
// mode 0: X = B L^-T (x L^T = b, forward); mode 1: X = B L^-1 (x L = b, backward).
// Blocked in TB columns: a block's columns are solved by substitution, then the columns
// still to come take one product with them, so that most of the n M^2 / 2 multiply-adds
// are a GEMM's. (One thread per row over all M columns, as before, is one chain of M^2 / 2
// FP64 instructions: 1.6 ms for 256 rows of M = 256, and 65536 rows took 8.1 ms.)
constexpr int TB = 64;

// One block: rows of B (n x kb) against the kb x kb lower block L, into X (which may be B).
// The lanes
// of a warp share few rows: lane q of a group of eight owns columns q, q + 8, .. of its
// row, so that an FP64 instruction (64 cycles of its sub-partition, whatever the number
// of active lanes) works on four rows and eight columns. CG: groups of eight columns, as
// many as kb needs (a chain step to each: all 64 took a FITC prediction through one inducing
// input from 124 to 159 us).
template <int MODE, int CG>
__global__ void __launch_bounds__(128) tri_block_kernel(const double *__restrict__ L, int64_t ldl, int kb,
                                                        const double *B, int64_t ldb, double *X, int64_t ldx,
                                                        int64_t n, const int *__restrict__ status) {
  if (status && *(volatile const int *)status != 0) return;
  constexpr int W = 8 * CG;
  __shared__ double Ls[W][W + 1];  // [c][r] = L(r, c): a step reads one column (mode 0) or row (mode 1)
  __shared__ double rd[W];
  for (int idx = threadIdx.x; idx < W * W; idx += 128) {
    const int r = idx % W, c = idx / W;
    Ls[c][r] = (r < kb && c < kb && r >= c) ? L[r + c * ldl] : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < W) rd[threadIdx.x] = threadIdx.x < kb ? 1.0 / Ls[threadIdx.x][threadIdx.x] : 0.0;
  __syncthreads();
  const int lane = threadIdx.x & 31, q = lane & 7;
  const int64_t i = ((int64_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * 4 + (lane >> 3);
  double x[CG];
#pragma unroll
  for (int t = 0; t < CG; ++t) {
    const int c = 8 * t + q;
    x[t] = (i < n && c < kb) ? B[i + c * ldb] : 0.0;
  }
#pragma unroll
  for (int s0 = 0; s0 < CG; ++s0) {
    const int t0 = MODE == 0 ? s0 : CG - 1 - s0;  // the eight columns 8 t0 ..
#pragma unroll
    for (int s1 = 0; s1 < 8; ++s1) {
      const int cq = MODE == 0 ? s1 : 7 - s1, c = 8 * t0 + cq;
      // the owner's value scaled by 1 / L(c, c); a column past kb holds zeros and has rd = 0
      const double xc = __shfl_sync(0xffffffffu, x[t0] * rd[c], cq, 8);
      if (q == cq) x[t0] = xc;
      else if (MODE == 0 ? q > cq : q < cq) x[t0] = fma(-xc, MODE == 0 ? Ls[c][8 * t0 + q] : Ls[8 * t0 + q][c], x[t0]);
#pragma unroll
      for (int t = MODE == 0 ? t0 + 1 : 0; t < (MODE == 0 ? CG : t0); ++t)
        x[t] = fma(-xc, MODE == 0 ? Ls[c][8 * t + q] : Ls[8 * t + q][c], x[t]);
    }
  }
  if (i < n)
#pragma unroll
    for (int t = 0; t < CG; ++t) {
      const int c = 8 * t + q;
      if (c < kb) X[i + c * ldx] = x[t];
    }
}

template <int MODE>
static void tri_block(cudaStream_t s, const double *L, int64_t ldl, int kb, const double *B, int64_t ldb, double *X,
                      int64_t ldx, int64_t n, const int *status) {
  const unsigned grid = (unsigned)((n + 15) / 16);
  auto kern = kb > 32 ? tri_block_kernel<MODE, 8> : kb > 16 ? tri_block_kernel<MODE, 4>
              : kb > 8 ? tri_block_kernel<MODE, 2> : tri_block_kernel<MODE, 1>;
  kern<<<grid, 128, 0, s>>>(L, ldl, kb, B, ldb, X, ldx, n, status);
  GPGP_CHECK_LAUNCH();
}

// C = alpha A B^T + beta C (n x N, alpha 1 or -1, beta 0 or 1) for many rows n: on the
// tensor cores at FP64 accuracy where rows_take_slices.
void rows_times_bt(cudaStream_t s, int64_t n, int64_t N, int64_t K, double alpha, const double *A, int64_t lda,
                   const double *B, int64_t ldb, double beta, double *C, int64_t ldc, int *err) {
  SplitBuf a(s), b(s);
  if (!rows_take_slices(n, N, K) || !with_scratch([&] {
        a.bind(n, K, OZ_FP64);
        b.bind(N, K, OZ_FP64);
      })) {
    gemm64(s, false, true, n, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
    return;
  }
  oz_split(s, A, lda, 0, n, K, &a.sp);
  oz_split(s, B, ldb, 0, N, K, &b.sp);
  oz_gemm(s, a.sp, 0, b.sp, 0, n, N, 0, a.sp.nkb, 0, alpha, beta, C, ldc, false, err);
}

// X may alias B. err (optional): the products of many rows then go through the sliced
// tensor-core GEMM, whose bounded waits report there.
void tri_rows(cudaStream_t s, const double *L, int64_t M, int64_t ldl, const double *B, int64_t ldb,
              double *X, int64_t ldx, int64_t n, int mode, int *err) {
  if (n <= 0 || M <= 0) return;
  if (M <= TB) {
    if (mode == 0) tri_block<0>(s, L, ldl, (int)M, B, ldb, X, ldx, n, nullptr);
    else tri_block<1>(s, L, ldl, (int)M, B, ldb, X, ldx, n, nullptr);
    return;
  }
  if (X != B)
    GPGP_CUDA(cudaMemcpy2DAsync(X, ldx * sizeof(double), B, ldb * sizeof(double), n * sizeof(double), M,
                                cudaMemcpyDeviceToDevice, s));
  SplitBuf xs(s), ls(s);
  // (the first block has the most columns after it)
  const bool sliced = err && rows_take_slices(n, M - TB, TB) && with_scratch([&] {
                        xs.bind(n, TB, OZ_FP64);
                        ls.bind(M, TB, OZ_FP64);
                      });
  const int64_t nblk = (M + TB - 1) / TB;
  for (int64_t b = 0; b < nblk; ++b) {
    const int64_t k0 = (mode == 0 ? b : nblk - 1 - b) * TB;
    const int kb = (int)std::min<int64_t>(TB, M - k0);
    double *Xk = X + k0 * ldx;
    if (mode == 0) tri_block<0>(s, L + k0 * (ldl + 1), ldl, kb, Xk, ldx, Xk, ldx, n, nullptr);
    else tri_block<1>(s, L + k0 * (ldl + 1), ldl, kb, Xk, ldx, Xk, ldx, n, nullptr);
    // the columns after the block (mode 0: X_rest -= X_k L_rest,k^T) or before it
    // (mode 1: X_rest -= X_k L_k,rest)
    const int64_t rest = mode == 0 ? M - k0 - kb : k0;
    if (rest <= 0) continue;
    double *Xr = mode == 0 ? X + (k0 + kb) * ldx : X;
    const double *Lr = mode == 0 ? L + (k0 + kb) + k0 * ldl : L + k0;
    if (sliced && rows_take_slices(n, rest, TB)) {
      oz_split(s, Xk, ldx, 0, n, kb, &xs.sp);
      oz_split(s, Lr, ldl, mode == 0 ? 0 : 1, rest, kb, &ls.sp);
      oz_gemm(s, xs.sp, 0, ls.sp, 0, n, rest, 0, 1, 0, -1.0, 1.0, Xr, ldx, false, err);
    } else {
      gemm64(s, false, mode == 0, n, rest, kb, -1.0, Xk, ldx, Lr, ldl, 1.0, Xr, ldx);
    }
  }
}

// x = L^-1 b (trans = 0) or x = L^-T b (trans = 1), x may alias b: one CTA, 32 rows at a
// time. Warp 0 solves the diagonal block in registers (one row per lane) while the other
// rows' entries of the block's columns are already in flight; then every row still to
// come takes its 32 multiply-adds at once. (A row's dot product by one warp, row after
// row, was a chain of shuffles and FP64 latencies: 500 us at M = 256.)
constexpr int TV = 32, TV_THREADS = 256;

__global__ void __launch_bounds__(TV_THREADS) tri_vec_kernel(const double *__restrict__ L, int64_t M, int64_t ldl,
                                                             const double *b, double *x, int trans) {
  __shared__ double D[TV][TV + 1];  // the diagonal block, D[c][r] = L(r, c)
  __shared__ double xs[TV];
  const int tid = threadIdx.x, lane = tid & 31;
  if (x != b)
    for (int64_t r = tid; r < M; r += TV_THREADS) x[r] = b[r];
  const int64_t nblk = (M + TV - 1) / TV;
  for (int64_t st = 0; st < nblk; ++st) {
    const int64_t k0 = (trans ? nblk - 1 - st : st) * TV;
    const int kb = (int)(M - k0 < TV ? M - k0 : TV);
    for (int idx = tid; idx < TV * TV; idx += TV_THREADS) {
      const int r = idx % TV, c = idx / TV;
      D[c][r] = (r < kb && c < kb && r >= c) ? L[(k0 + r) + (k0 + c) * ldl] : 0.0;
    }
    // rows after the block (trans: before it); this thread's first row is loaded now
    const int64_t r0 = trans ? 0 : k0 + kb, r1 = trans ? k0 : M;
    const int64_t r = r0 + tid;
    double l[TV];
#pragma unroll
    for (int c = 0; c < TV; ++c)
      l[c] = (r < r1 && c < kb) ? (trans ? L[(k0 + c) + r * ldl] : L[r + (k0 + c) * ldl]) : 0.0;
    __syncthreads();
    if (tid < 32) {
      double v = lane < kb ? x[k0 + lane] : 0.0;
      const double rd = lane < kb ? 1.0 / D[lane][lane] : 0.0;
      for (int t = 0; t < kb; ++t) {
        const int c = trans ? kb - 1 - t : t;
        const double xc = __shfl_sync(0xffffffffu, v * rd, c);
        if (lane == c) v = xc;
        else if (trans ? lane < c : lane > c) v = fma(-xc, trans ? D[lane][c] : D[c][lane], v);
      }
      xs[lane] = v;
      if (lane < kb) x[k0 + lane] = v;
    }
    __syncthreads();
    if (r < r1) {
      double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int c = 0; c < TV; ++c) a[c & 3] = fma(l[c], xs[c], a[c & 3]);
      x[r] -= (a[0] + a[1]) + (a[2] + a[3]);
    }
    for (int64_t rr = r + TV_THREADS; rr < r1; rr += TV_THREADS) {
      double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int c = 0; c < TV; ++c)
        if (c < kb) a[c & 3] = fma(trans ? L[(k0 + c) + rr * ldl] : L[rr + (k0 + c) * ldl], xs[c], a[c & 3]);
      x[rr] -= (a[0] + a[1]) + (a[2] + a[3]);
    }
    __syncthreads();
  }
}

void tri_vec(cudaStream_t s, const double *L, int64_t M, int64_t ldl, const double *b, double *x,
             bool trans) {
  if (M <= 0) return;
  tri_vec_kernel<<<1, TV_THREADS, 0, s>>>(L, M, ldl, b, x, trans ? 1 : 0);
  GPGP_CHECK_LAUNCH();
}

// panel: L21 = A21 L11^-T by forward substitution, one row per thread (in place), for
// the many rows of a batch (a single matrix's panel takes tri_block_kernel, whose rows
// are 12 us instead of this one's 62 to 116 while they are few). Substitution keeps the
// factorisation backward stable when a diagonal block is ill-conditioned (FITC's K_z);
// the inverse W is used by the solves instead.
__global__ void __launch_bounds__(128) potrf_panel_kernel(double *__restrict__ A21, int64_t m, int kb,
                                                          int64_t lda, const double *__restrict__ L11,
                                                          const int *__restrict__ status, int64_t sA) {
  // batched: problem blockIdx.y (A21 and L11 offset by sA, one status word per problem)
  A21 += blockIdx.y * sA;
  L11 += blockIdx.y * sA;
  status += blockIdx.y;
  __shared__ double Ls[NB][NB + 1];
  __shared__ double rd[NB];
  if (*(volatile const int *)status != 0) return;
  for (int idx = threadIdx.x; idx < NB * NB; idx += blockDim.x) {
    int r = idx % NB, c = idx / NB;
    Ls[r][c] = (r < kb && c < kb && r >= c) ? L11[r + c * lda] : 0.0;
  }
  __syncthreads();
  if (threadIdx.x < kb) rd[threadIdx.x] = 1.0 / Ls[threadIdx.x][threadIdx.x];
  __syncthreads();
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= m) return;
  double x[NB];
#pragma unroll
  for (int c = 0; c < NB; ++c) {
    if (c < kb) {
      double s = A21[r + c * lda];
      for (int k = 0; k < c; ++k) s = fma(-x[k], Ls[c][k], s);
      x[c] = s * rd[c];
    }
  }
#pragma unroll
  for (int c = 0; c < NB; ++c)
    if (c < kb) A21[r + c * lda] = x[c];
}

// panel by the diagonal block's inverse: L21 = A21 W11^T, L21(r, c) = sum_{k <= c}
// A21(r, k) W11(c, k). A CTA takes 4 rows (one element per thread), staged in
// shared memory with W11, so the FP64 work spreads over m / 4 CTAs; the four warps of a
// sub-partition pair hold columns c and 63 - c, whose sums add up to the same length. For
// the well-conditioned diagonal blocks of B = I + S K S the error is that of the
// substitution to within the block's condition number.
__global__ void __launch_bounds__(256) potrf_panel_inv_kernel(double *__restrict__ A21, int64_t m, int kb,
                                                              int64_t lda, const double *__restrict__ W,
                                                              const int *__restrict__ status) {
  __shared__ double Ws[NB][NB + 1];
  __shared__ double As[4][NB + 1];
  if (status && *(volatile const int *)status != 0) return;
  const int64_t r0 = (int64_t)blockIdx.x * 4;
#pragma unroll
  for (int t = 0; t < NB * NB / 256; ++t) {
    const int idx = threadIdx.x + 256 * t;
    Ws[idx % NB][idx / NB] = W[idx];
  }
  {
    const int rr = threadIdx.x & 3, c = threadIdx.x >> 2;
    As[rr][c] = (r0 + rr < m && c < kb) ? A21[r0 + rr + c * lda] : 0.0;
  }
  __syncthreads();
  // warps w and w + 4 share a sub-partition: columns 8w.. and 56 - 8w..
  const int w = threadIdx.x >> 5, cg = w < 4 ? w : 11 - w;
  const int rr = threadIdx.x & 3, c = 8 * cg + ((threadIdx.x & 31) >> 2);
  if (r0 + rr >= m || c >= kb) return;
  double s0 = 0.0, s1 = 0.0;
  int k = 0;
  for (; k + 1 <= c; k += 2) {
    s0 = fma(As[rr][k], Ws[c][k], s0);
    s1 = fma(As[rr][k + 1], Ws[c][k + 1], s1);
  }
  if (k <= c) s0 = fma(As[rr][k], Ws[c][k], s0);
  A21[r0 + rr + c * lda] = s0 + s1;
}

// The next diagonal block's update, D -= L L^T (lower triangle) for its m <= 64 rows L
// (m x 64): 32 CTAs share the 2080 entries, two threads to an entry (even and odd
// terms, as the small GEMM sums them), so that each sub-partition runs one warp of 32 FP64
// multiply-adds (the chain of the Cholesky waits for this: 5 us, against 12 as a small
// GEMM whose every operand came from L2).
constexpr int SU_CTAS = 32, SU_ENT = (NB * (NB + 1) / 2 + SU_CTAS - 1) / SU_CTAS;  // 65 entries

__global__ void __launch_bounds__(160) syrk_block_kernel(const double *__restrict__ Ln, int64_t lda, int m,
                                                         double *__restrict__ D) {
  __shared__ double Ls[NB][NB + 1];  // [k][r]
  const int tid = threadIdx.x;
  const int e = blockIdx.x * SU_ENT + (tid >> 1), half = tid & 1;
  int r = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
  if (r * (r + 1) / 2 > e) --r;
  if ((r + 1) * (r + 2) / 2 <= e) ++r;
  const int c = e - r * (r + 1) / 2;
  const bool mine = (tid >> 1) < SU_ENT && r < m;
  const double d = mine && half == 0 ? D[r + c * lda] : 0.0;
#pragma unroll
  for (int t = 0; t < (NB * NB + 159) / 160; ++t) {
    const int idx = tid + 160 * t, lr = idx % NB, lk = idx / NB;
    if (idx < NB * NB) Ls[lk][lr] = lr < m ? Ln[lr + lk * lda] : 0.0;
  }
  __syncthreads();
  double s = 0.0;
  if (mine)
#pragma unroll 8
    for (int k = half; k < NB; k += 2) s = fma(Ls[k][r], Ls[k][c], s);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  if (mine && half == 0) D[r + c * lda] = d - s;
}

void syrk_block(cudaStream_t s, const double *Ln, int64_t lda, int m, double *D) {
  if (m <= 0) return;
  syrk_block_kernel<<<SU_CTAS, 160, 0, s>>>(Ln, lda, m, D);
  GPGP_CHECK_LAUNCH();
}

void potrf(cudaStream_t s, double *A, int64_t n, int64_t lda, double *Winv, double *logdet_part,
           int *status, int panel_mode) {
  for (int64_t k0 = 0, blk = 0; k0 < n; k0 += NB, ++blk) {
    const int kb = (int)std::min<int64_t>(NB, n - k0);
    double *Akk = A + k0 + k0 * lda;
    double *W = Winv + blk * NB * NB;
    potrf_diag(s, Akk, kb, lda, W, logdet_part + blk, status, k0, 0, 0, 0, 1);
    const int64_t m = n - k0 - kb;
    if (m > 0) {
      double *A21 = A + (k0 + kb) + k0 * lda;
      if (panel_mode == 1) {
        potrf_panel_inv_kernel<<<(unsigned)((m + 3) / 4), 256, 0, s>>>(A21, m, kb, lda, W, status);
        GPGP_CHECK_LAUNCH();
      } else {
        tri_block<0>(s, Akk, lda, kb, A21, lda, A21, lda, m, status);
      }
      double *A22 = A + (k0 + kb) + (k0 + kb) * lda;
      gemm64(s, false, true, m, m, kb, -1.0, A21, lda, A21, lda, 1.0, A22, lda, true, 0);
    }
  }
}

// Batched: `batch` problems of the same size n, matrices sA apart, inverses sW
// apart, logdet partials sL apart, one status word each.
void potrf_batched(cudaStream_t s, double *A, int64_t n, int64_t lda, int64_t sA, double *Winv,
                   int64_t sW, double *logdet_part, int64_t sL, int *status, int64_t batch) {
  for (int64_t k0 = 0, blk = 0; k0 < n; k0 += NB, ++blk) {
    const int kb = (int)std::min<int64_t>(NB, n - k0);
    double *Akk = A + k0 + k0 * lda;
    potrf_diag(s, Akk, kb, lda, Winv + blk * NB * NB, logdet_part + blk, status, k0, sA, sW, sL, batch);
    const int64_t m = n - k0 - kb;
    if (m > 0) {
      double *A21 = A + (k0 + kb) + k0 * lda;
      dim3 pg((unsigned)((m + 127) / 128), (unsigned)batch);
      potrf_panel_kernel<<<pg, 128, 0, s>>>(A21, m, kb, lda, Akk, status, sA);
      GPGP_CHECK_LAUNCH();
      double *A22 = A + (k0 + kb) + (k0 + kb) * lda;
      gemm64_batched(s, false, true, m, m, kb, -1.0, A21, lda, sA, A21, lda, sA, 1.0, A22, lda, sA, batch,
                     true, 0);
    }
  }
}

// ---------------------------------------------------------------------------
// triangular solves with one right-hand side
// ---------------------------------------------------------------------------
// Step k of the forward solve: every CTA recomputes xk = W_kk b_k (64x64), CTA 0
// stores it into xo, and each CTA updates its 256-row slice of b below the block.
__global__ void __launch_bounds__(256) trsv_fwd_step(const double *__restrict__ L, int64_t n, int64_t lda,
                                                     const double *__restrict__ W, int64_t k0, int kb,
                                                     double *__restrict__ b, double *__restrict__ xo,
                                                     const int *__restrict__ status) {
  __shared__ double bk[NB];
  __shared__ double xk[NB];
  if (*(volatile const int *)status != 0) return;
  const int tid = threadIdx.x;
  if (tid < NB) bk[tid] = tid < kb ? b[k0 + tid] : 0.0;
  __syncthreads();
  if (tid < NB) {
    double s = 0.0;
    for (int c = 0; c <= tid && c < kb; ++c) s = fma(W[tid + c * NB], bk[c], s);
    xk[tid] = tid < kb ? s : 0.0;
  }
  __syncthreads();
  if (blockIdx.x == 0 && tid < kb) xo[k0 + tid] = xk[tid];
  const int64_t r = k0 + kb + (int64_t)blockIdx.x * 256 + tid;
  if (r < n) {
    double s = 0.0;
    for (int c = 0; c < kb; ++c) s = fma(L[r + (k0 + c) * lda], xk[c], s);
    b[r] -= s;
  }
}

void trsv_lower(cudaStream_t s, const double *L, int64_t n, int64_t lda, const double *Winv,
                double *b, double *x, const int *status) {
  // b is consumed (rows below the current block are updated in place); x receives L^-1 b
  for (int64_t k0 = 0, blk = 0; k0 < n; k0 += NB, ++blk) {
    const int kb = (int)std::min<int64_t>(NB, n - k0);
    const int64_t rest = n - k0 - kb;
    unsigned g = (unsigned)std::max<int64_t>(1, (rest + 255) / 256);
    trsv_fwd_step<<<g, 256, 0, s>>>(L, n, lda, Winv + blk * NB * NB, k0, kb, b, x, status);
    GPGP_CHECK_LAUNCH();
  }
}

// Backward step: x_k = W_kk^T b_k, then b[0:k0] -= L[k-block rows, 0:k0]^T x_k.
__global__ void __launch_bounds__(256) trsv_bwd_step(const double *__restrict__ L, int64_t lda,
                                                     const double *__restrict__ W, int64_t k0, int kb,
                                                     double *__restrict__ b, double *__restrict__ xo,
                                                     const int *__restrict__ status) {
  __shared__ double bk[NB];
  __shared__ double xk[NB];
  if (*(volatile const int *)status != 0) return;
  const int tid = threadIdx.x;
  if (tid < NB) bk[tid] = tid < kb ? b[k0 + tid] : 0.0;
  __syncthreads();
  if (tid < NB) {
    double s = 0.0;
    for (int r = tid; r < kb; ++r) s = fma(W[r + tid * NB], bk[r], s);
    xk[tid] = tid < kb ? s : 0.0;
  }
  __syncthreads();
  if (blockIdx.x == 0 && tid < kb) xo[k0 + tid] = xk[tid];
  // one warp per column c < k0
  const int lane = tid & 31, warp = tid >> 5;
  const int64_t c = (int64_t)blockIdx.x * 8 + warp;
  if (c < k0) {
    double s = 0.0;
    for (int r = lane; r < kb; r += 32) s = fma(L[(k0 + r) + c * lda], xk[r], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) b[c] -= s;
  }
}

void trsv_lower_t(cudaStream_t s, const double *L, int64_t n, int64_t lda, const double *Winv,
                  double *b, double *x, const int *status) {
  // b is consumed; x receives L^-T b
  const int64_t nblk = (n + NB - 1) / NB;
  for (int64_t blk = nblk - 1; blk >= 0; --blk) {
    const int64_t k0 = blk * NB;
    const int kb = (int)std::min<int64_t>(NB, n - k0);
    unsigned g = (unsigned)std::max<int64_t>(1, (k0 + 7) / 8);
    trsv_bwd_step<<<g, 256, 0, s>>>(L, lda, Winv + blk * NB * NB, k0, kb, b, x, status);
    GPGP_CHECK_LAUNCH();
  }
}

// ---------------------------------------------------------------------------
// single-launch triangular solves, ordered by the solution's blocks
// ---------------------------------------------------------------------------
// A persistent grid takes the 64-row blocks of x in dependency order from a
// ticket (forward: first block first; transposed: last block first), so every
// block a CTA waits for belongs to a CTA that is already running. The CTA of
// block i subtracts L_ij x_j (L_ji^T x_j when transposed) for each earlier block
// j as soon as that block is there, then multiplies by the diagonal block's
// inverse W_ii and writes x_i. Each thread visits the blocks in a
// fixed order, so the result does not depend on timing. Waits are bounded: when
// one runs out the kernel sets *err = 3 and every CTA leaves.
// x is filled with FLOW_EMPTY before the launch and its entries are their own flags: the
// load that finds an entry has it, with no fence, flag and second load between one block
// and the next (a solve of n = 3000, forward and transposed: 327 -> 203 us on average,
// n = 8192: 912 -> 544, with the transposed sums' 9 additions for 40). sync[0]: ticket;
// zeroed before the launch.
constexpr unsigned long long FLOW_EMPTY = ~0ull;  // a NaN that no instruction makes
constexpr int FLOW_BATCH = 8;  // earlier blocks applied per round

__global__ void __launch_bounds__(256) trsv_flow_kernel(const double *__restrict__ L, int64_t n, int64_t lda,
                                                        const double *__restrict__ Winv,
                                                        const double *__restrict__ b, double *x, int trans,
                                                        const int *__restrict__ status, unsigned *sync,
                                                        int *err, uint32_t polls) {
  __shared__ double Ws[NB][NB + 1];
  __shared__ double xs[FLOW_BATCH][NB];
  __shared__ double vs[NB];
  __shared__ double red[4][NB + 1];
  __shared__ int64_t step_sh;
  __shared__ int there[FLOW_BATCH];
  if (*(volatile const int *)status != 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t nblk = (n + NB - 1) / NB;
  static_assert(FLOW_BATCH == 8, "a block to a warp");
  for (;;) {
    __syncthreads();
    if (tid == 0) step_sh = (int64_t)atomicAdd(sync, 1u);
    __syncthreads();
    const int64_t step = step_sh;
    if (step >= nblk) return;
    const int64_t blk = trans ? nblk - 1 - step : step;
    const int64_t k0 = blk * NB;
    const int kb = (int)((n - k0) < NB ? (n - k0) : NB);
    const double *W = Winv + blk * NB * NB;
    for (int idx = tid; idx < NB * NB; idx += 256) Ws[idx % NB][idx / NB] = W[idx];
    // forward: thread (r, p) takes row r of the block and columns 16p..16p+15 of
    // every earlier block; transposed: warp w takes columns 8w..8w+7 of this block
    // and lane l rows l, l + 32 of every later block
    double acc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] = 0.0;
    const int r = tid & 63, p = tid >> 6;
    const int64_t ndep = trans ? nblk - 1 - blk : blk;
    // This thread's 16 entries of the L tile of earlier block number d; the tile of
    // the next block is always in flight (loaded before the wait for its flag and
    // before the products with the current one).
    auto load_tile = [&](int64_t d, double (&t)[16]) {
      const int64_t j = trans ? nblk - 1 - d : d;
      const int64_t j0 = j * NB;
      const int jb = (int)((n - j0) < NB ? (n - j0) : NB);
      if (!trans) {
        const double *Lr = L + (k0 + r) + (j0 + 16 * p) * lda;
#pragma unroll
        for (int q = 0; q < 16; ++q) t[q] = (r < kb && 16 * p + q < jb) ? Lr[q * lda] : 0.0;
      } else {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int c = warp * 8 + q;
          const double *Lc = L + j0 + (k0 + c) * lda;
          t[2 * q] = (c < kb && lane < jb) ? Lc[lane] : 0.0;
          t[2 * q + 1] = (c < kb && lane + 32 < jb) ? Lc[lane + 32] : 0.0;
        }
      }
    };
    double tnext[16];
    if (ndep > 0) load_tile(0, tnext);
    // b's entry that this thread subtracts the sum from
    const int bc = trans ? warp * 8 + lane : tid;
    const double bv = (trans ? lane < 8 : tid < NB) && bc < kb ? b[k0 + bc] : 0.0;
    for (int64_t d0 = 0; d0 < ndep;) {
      // warp w looks for block d0 + w and takes it along; warp 0 waits for the next one
      const int64_t d = d0 + warp, j0 = (trans ? nblk - 1 - d : d) * NB;
      bool run = d < ndep;
      for (uint32_t it = 0; run; ++it) {
        unsigned long long e[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          e[h] = 0ull;
          if (j0 + lane + 32 * h < n)
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(e[h]) : "l"(x + j0 + lane + 32 * h));
        }
        const bool all = __all_sync(0xffffffffu, e[0] != FLOW_EMPTY && e[1] != FLOW_EMPTY);
        // (one outcome for the warp, whose lanes may see the error word at different times:
        // the vote above needs all of them)
        const bool last =
            warp > 0 || it >= polls || ((it & 1023u) == 1023u && __any_sync(0xffffffffu, *(volatile const int *)err != 0));
        if (all || last) {
          xs[warp][lane] = __longlong_as_double((long long)e[0]);
          xs[warp][lane + 32] = __longlong_as_double((long long)e[1]);
          if (lane == 0) {
            there[warp] = all;
            if (!all && warp == 0) atomicExch(err, 3);
          }
          run = false;
        }
      }
      if (d >= ndep && lane == 0) there[warp] = 0;
      __syncthreads();
      int k = 0;
      while (k < FLOW_BATCH && there[k]) ++k;
      if (k == 0) return;
      for (int dd = 0; dd < k; ++dd) {
        double tc[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) tc[q] = tnext[q];
        if (d0 + dd + 1 < ndep) load_tile(d0 + dd + 1, tnext);
        if (!trans) {
#pragma unroll
          for (int q = 0; q < 16; ++q) acc[q & 7] = fma(tc[q], xs[dd][16 * p + q], acc[q & 7]);
        } else {
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[q] += fma(tc[2 * q + 1], xs[dd][lane + 32], tc[2 * q] * xs[dd][lane]);
        }
      }
      __syncthreads();
      d0 += k;
    }
    // v = b_blk - (the sum over the earlier blocks)
    if (!trans) {
      double t = 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q) t += acc[q];
      red[p][r] = t;
      __syncthreads();
      if (tid < NB) vs[tid] = tid < kb ? bv - (((red[0][tid] + red[1][tid]) + red[2][tid]) + red[3][tid]) : 0.0;
    } else {
      // eight sums over the warp's lanes, each as a tree over lane ^ 16, ^ 8, .. ^ 1: after
      // the first three steps a lane goes on with one of them (9 additions, not 40)
#pragma unroll
      for (int o = 16, m = 4; m >= 1; o >>= 1, m >>= 1)
#pragma unroll
        for (int q = 0; q < m; ++q) {
          const bool up = lane & o;
          const double keep = up ? acc[q + m] : acc[q], give = up ? acc[q] : acc[q + m];
          acc[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
      // lane l has sum 4 [l & 16] + 2 [l & 8] + [l & 4]
      const double t = __shfl_sync(0xffffffffu, acc[0], ((lane & 4) << 2) | ((lane & 2) << 2) | ((lane & 1) << 2));
      if (lane < 8) vs[bc] = bc < kb ? bv - t : 0.0;
    }
    __syncthreads();
    // x_blk = W v (lower W) or W^T v: four threads per entry, partial sums by shuffles
    {
      const int row = tid >> 2, pp = tid & 3;
      double s0 = 0.0, s1 = 0.0;
      if (!trans) {
        for (int c = pp; c <= row && c < kb; c += 8) {
          s0 = fma(Ws[row][c], vs[c], s0);
          if (c + 4 <= row && c + 4 < kb) s1 = fma(Ws[row][c + 4], vs[c + 4], s1);
        }
      } else {
        for (int rr = row + pp; rr < kb; rr += 8) {
          s0 = fma(Ws[rr][row], vs[rr], s0);
          if (rr + 4 < kb) s1 = fma(Ws[rr + 4][row], vs[rr + 4], s1);
        }
      }
      double s = s0 + s1;
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      if (pp == 0 && row < kb) {
        unsigned long long e = (unsigned long long)__double_as_longlong(s);
        if (e == FLOW_EMPTY) e = 0x7FF8000000000000ull;
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(x + k0 + row), "l"(e) : "memory");
      }
    }
  }
}

__global__ void flow_clear_kernel(int64_t n, double *__restrict__ x, unsigned *__restrict__ sync) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i < n) x[i] = __longlong_as_double((long long)FLOW_EMPTY);
  if (i == 0) *sync = 0u;
}

// Small solves (n <= 512): one CTA walks the row blocks in order (a launch and a
// 64-row step cost less than the flags of the multi-CTA version at this size).
// Thread (r, p) sums the earlier (later, when transposed) blocks' columns
// c = p mod 4 for row r of the block; the block's inverse then gives x_blk. The inverse
// and b come to shared memory beside those sums, and the sums' loads go out eight at a
// time: between the blocks are a few FP64 chains and no loads (n = 200: 30 -> 25 us).
__global__ void __launch_bounds__(256) trsv_small_kernel(const double *__restrict__ L, int64_t n, int64_t lda,
                                                         const double *__restrict__ Winv,
                                                         const double *__restrict__ b, double *__restrict__ x,
                                                         int trans, const int *__restrict__ status) {
  __shared__ double xs[8 * NB];
  __shared__ double vs[NB];
  __shared__ double red[4][NB + 1];
  __shared__ double Ws[NB][NB + 1];  // [column][row]
  if (*(volatile const int *)status != 0) return;
  const int tid = threadIdx.x, r = tid & 63, p = tid >> 6;
  const int nblk = (int)((n + NB - 1) / NB);
  for (int st = 0; st < nblk; ++st) {
    const int blk = trans ? nblk - 1 - st : st;
    const int k0 = blk * NB;
    const int kb = (int)(n - k0 < NB ? n - k0 : NB);
    const double *W = Winv + (int64_t)blk * NB * NB;
    double wr[NB * NB / 256];
#pragma unroll
    for (int t = 0; t < NB * NB / 256; ++t) wr[t] = W[tid + 256 * t];
    const double bv = tid < kb ? b[k0 + tid] : 0.0;
    double acc = 0.0;
    if (r < kb) {
      if (!trans) {
#pragma unroll 8
        for (int c = p; c < k0; c += 4) acc = fma(L[(k0 + r) + (int64_t)c * lda], xs[c], acc);
      } else {
#pragma unroll 8
        for (int c = k0 + kb + p; c < n; c += 4) acc = fma(L[c + (int64_t)(k0 + r) * lda], xs[c], acc);
      }
    }
#pragma unroll
    for (int t = 0; t < NB * NB / 256; ++t) Ws[(tid + 256 * t) / NB][tid % NB] = wr[t];
    red[p][r] = acc;
    __syncthreads();
    if (tid < NB) vs[tid] = tid < kb ? bv - (((red[0][tid] + red[1][tid]) + red[2][tid]) + red[3][tid]) : 0.0;
    __syncthreads();
    if (tid < kb) {
      double s0 = 0.0, s1 = 0.0;
      if (!trans) {
        int c = 0;
        for (; c + 1 <= tid; c += 2) {
          s0 = fma(Ws[c][tid], vs[c], s0);
          s1 = fma(Ws[c + 1][tid], vs[c + 1], s1);
        }
        if (c <= tid) s0 = fma(Ws[c][tid], vs[c], s0);
      } else {
        int rr = tid;
        for (; rr + 1 < kb; rr += 2) {
          s0 = fma(Ws[tid][rr], vs[rr], s0);
          s1 = fma(Ws[tid][rr + 1], vs[rr + 1], s1);
        }
        if (rr < kb) s0 = fma(Ws[tid][rr], vs[rr], s0);
      }
      xs[k0 + tid] = s0 + s1;
      x[k0 + tid] = s0 + s1;
    }
    __syncthreads();
  }
}

void trsv_flow(cudaStream_t s, const double *L, int64_t n, int64_t lda, const double *Winv, const double *b,
               double *x, bool trans, const int *status, unsigned *sync, int *err) {
  if (n <= 0) return;
  const int g_sms = device_sms();
  const int64_t nblk = (n + NB - 1) / NB;
  if (nblk <= 8) {
    KTScope kts(GPGP_KPROF_TRSV, s, (double)n * (double)n);
    trsv_small_kernel<<<1, 256, 0, s>>>(L, n, lda, Winv, b, x, trans ? 1 : 0, status);
    GPGP_CHECK_LAUNCH();
    return;
  }
  flow_clear_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, x, sync);
  GPGP_CHECK_LAUNCH();
  const unsigned grid = (unsigned)std::min<int64_t>(nblk, g_sms);
  KTScope kts(GPGP_KPROF_TRSV, s, (double)n * (double)n);
  trsv_flow_kernel<<<grid, 256, 0, s>>>(L, n, lda, Winv, b, x, trans ? 1 : 0, status, sync, err,
                                        tl_wait.polls[GPGP_WAIT_FLOW]);
  GPGP_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// multi-RHS solve and triangular inverse
// ---------------------------------------------------------------------------
void trsm_lower(cudaStream_t s, const double *L, int64_t n, int64_t lda, const double *Winv,
                double *B, int64_t m, int64_t ldb, double *tmp, const int *status) {
  // right-looking: X_k = W_kk B_k; B_rest -= L_rest,k X_k. tmp holds NB x m.
  (void)status;
  for (int64_t k0 = 0, blk = 0; k0 < n; k0 += NB, ++blk) {
    const int kb = (int)std::min<int64_t>(NB, n - k0);
    double *Bk = B + k0;
    gemm64(s, false, false, kb, m, kb, 1.0, Winv + blk * NB * NB, NB, Bk, ldb, 0.0, tmp, NB);
    GPGP_CUDA(cudaMemcpy2DAsync(Bk, ldb * sizeof(double), tmp, NB * sizeof(double),
                                kb * sizeof(double), m, cudaMemcpyDeviceToDevice, s));
    const int64_t rest = n - k0 - kb;
    if (rest > 0)
      gemm64(s, false, false, rest, m, kb, -1.0, L + (k0 + kb) + k0 * lda, lda, tmp, NB, 1.0,
             B + k0 + kb, ldb);
  }
}

__global__ void set_identity_kernel(double *W, int64_t n, int64_t ldw) {
  for (int64_t j = blockIdx.y; j < n; j += gridDim.y)
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
      W[i + j * ldw] = (i == j) ? 1.0 : 0.0;
}

void trtri_lower(cudaStream_t s, const double *L, int64_t n, int64_t lda, const double *Winv,
                 double *Wout, int64_t ldw, double *tmp, const int *status) {
  // Wout = L^-1 by a triangular solve against I that skips the zero columns:
  // for block row k, X_k = W_kk B_k[:, 0:k0+kb] and B_rest[:, 0:k0+kb] -= L_rest,k X_k.
  // tmp holds NB x n. The strict upper triangle of Wout stays exactly zero.
  (void)status;
  if (n == 0) return;
  dim3 g((unsigned)std::min<int64_t>((n + 255) / 256, 64), (unsigned)std::min<int64_t>(n, 65535));
  set_identity_kernel<<<g, 256, 0, s>>>(Wout, n, ldw);
  GPGP_CHECK_LAUNCH();
  for (int64_t k0 = 0, blk = 0; k0 < n; k0 += NB, ++blk) {
    const int kb = (int)std::min<int64_t>(NB, n - k0);
    const int64_t ncol = k0 + kb;
    double *Bk = Wout + k0;
    gemm64(s, false, false, kb, ncol, kb, 1.0, Winv + blk * NB * NB, NB, Bk, ldw, 0.0, tmp, NB);
    GPGP_CUDA(cudaMemcpy2DAsync(Bk, ldw * sizeof(double), tmp, NB * sizeof(double),
                                kb * sizeof(double), ncol, cudaMemcpyDeviceToDevice, s));
    const int64_t rest = n - ncol;
    if (rest > 0)
      gemm64(s, false, false, rest, ncol, kb, -1.0, L + ncol + k0 * lda, lda, tmp, NB, 1.0,
             Wout + ncol, ldw);
  }
}

// column sums of squares of a lower-triangular W (diag of W^T W)
__global__ void col_sumsq_lower_kernel(const double *__restrict__ W, int64_t n, int64_t ldw,
                                       double *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= n) return;
  double s = 0.0;
  for (int64_t r = c + lane; r < n; r += 32) {
    double v = W[r + c * ldw];
    s = fma(v, v, s);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) out[c] = s;
}

void col_sumsq_lower(cudaStream_t s, const double *W, int64_t n, int64_t ldw, double *out) {
  if (n == 0) return;
  col_sumsq_lower_kernel<<<(unsigned)((n * 32 + 255) / 256), 256, 0, s>>>(W, n, ldw, out);
  GPGP_CHECK_LAUNCH();
}

__global__ void col_sumsq_kernel(const double *__restrict__ B, int64_t n, int64_t m, int64_t ldb,
                                 double *__restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= m) return;
  double s = 0.0;
  for (int64_t r = lane; r < n; r += 32) {
    double v = B[r + c * ldb];
    s = fma(v, v, s);
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) out[c] = s;
}

void col_sumsq(cudaStream_t s, const double *B, int64_t n, int64_t m, int64_t ldb, double *out) {
  if (m == 0) return;
  col_sumsq_kernel<<<(unsigned)((m * 32 + 255) / 256), 256, 0, s>>>(B, n, m, ldb, out);
  GPGP_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// GEMV with a deterministic two-stage reduction over column chunks
// ---------------------------------------------------------------------------
constexpr int GV_ROWS = 256, GV_COLS = 1024;

__global__ void gemv_n_kernel(int64_t M, int64_t N, const double *__restrict__ A, int64_t lda,
                              const double *__restrict__ x, double *__restrict__ part) {
  const int64_t r = (int64_t)blockIdx.x * GV_ROWS + threadIdx.x;
  const int64_t c0 = (int64_t)blockIdx.y * GV_COLS;
  const int64_t c1 = (c0 + GV_COLS < N) ? c0 + GV_COLS : N;
  if (r >= M) return;
  // four chains, so that the FP64 latency of one row's sum is hidden by its own loads
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  int64_t c = c0;
  for (; c + 4 <= c1; c += 4)
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = fma(A[r + (c + u) * lda], x[c + u], s[u]);
  for (; c < c1; ++c) s[0] = fma(A[r + c * lda], x[c], s[0]);
  part[r + blockIdx.y * M] = (s[0] + s[1]) + (s[2] + s[3]);
}

// A^T x of a tall A with too few columns for a warp each to fill the GPU: a warp takes
// GT_ROWS rows of a column, and the partials are summed in order (gemv_reduce_kernel).
// 65536 x 256: 452 us with one warp per column.
constexpr int64_t GT_ROWS = 2048;
__global__ void gemv_t_part_kernel(int64_t M, int64_t N, const double *__restrict__ A, int64_t lda,
                                   const double *__restrict__ x, double *__restrict__ part) {
  const int lane = threadIdx.x & 31;
  const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= N) return;
  const int64_t r0 = (int64_t)blockIdx.y * GT_ROWS;
  const int64_t r1 = r0 + GT_ROWS < M ? r0 + GT_ROWS : M;
  double s0 = 0.0, s1 = 0.0;
  int64_t r = r0 + lane;
  for (; r + 32 < r1; r += 64) {
    s0 = fma(A[r + c * lda], x[r], s0);
    s1 = fma(A[r + 32 + c * lda], x[r + 32], s1);
  }
  if (r < r1) s0 = fma(A[r + c * lda], x[r], s0);
  double s = s0 + s1;
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) part[c + blockIdx.y * N] = s;
}

__global__ void gemv_t_kernel(int64_t M, int64_t N, const double *__restrict__ A, int64_t lda,
                              const double *__restrict__ x, double *__restrict__ y, double alpha,
                              double beta) {
  // y[c] = alpha * sum_r A[r, c] x[r] + beta y[c]; one warp per column
  const int lane = threadIdx.x & 31;
  const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= N) return;
  double s = 0.0;
  for (int64_t r = lane; r < M; r += 32) s = fma(A[r + c * lda], x[r], s);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) y[c] = (beta == 0.0) ? alpha * s : alpha * s + beta * y[c];
}

__global__ void gemv_reduce_kernel(int64_t M, int nchunk, const double *__restrict__ part,
                                   double alpha, double beta, double *__restrict__ y) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= M) return;
  double s = 0.0;
  for (int k = 0; k < nchunk; ++k) s += part[r + k * M];
  y[r] = (beta == 0.0) ? alpha * s : alpha * s + beta * y[r];
}

// Lower-triangular W (n x n, strict upper zero): y = W x (column chunks above a row
// block are skipped) or y = W^T x (a column's warp starts at its diagonal's
// 32-row group). Half the FP64 work of a full gemv, which bounds it on this part.
__global__ void trmv_n_kernel(int64_t n, const double *__restrict__ W, int64_t ldw, const double *__restrict__ x,
                              double *__restrict__ part) {
  const int64_t r = (int64_t)blockIdx.x * GV_ROWS + threadIdx.x;
  const int64_t c0 = (int64_t)blockIdx.y * GV_COLS;
  const int64_t rmax = (int64_t)blockIdx.x * GV_ROWS + GV_ROWS;  // columns >= rmax are zero for this block
  int64_t c1 = (c0 + GV_COLS < n) ? c0 + GV_COLS : n;
  if (c1 > rmax) c1 = rmax;
  if (r >= n) return;
  double s = 0.0;
  for (int64_t c = c0; c < c1; ++c) s = fma(W[r + c * ldw], x[c], s);
  part[r + blockIdx.y * n] = s;
}

__global__ void trmv_t_kernel(int64_t n, const double *__restrict__ W, int64_t ldw, const double *__restrict__ x,
                              double *__restrict__ y) {
  const int lane = threadIdx.x & 31;
  const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= n) return;
  double s = 0.0;
  for (int64_t r = (c & ~(int64_t)31) + lane; r < n; r += 32) s = fma(W[r + c * ldw], x[r], s);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) y[c] = s;
}

void trmv_lower(cudaStream_t s, bool trans, int64_t n, const double *W, int64_t ldw, const double *x, double *y) {
  if (n <= 0) return;
  if (trans) {
    trmv_t_kernel<<<(unsigned)((n * 32 + 255) / 256), 256, 0, s>>>(n, W, ldw, x, y);
    GPGP_CHECK_LAUNCH();
    return;
  }
  const int nchunk = (int)std::max<int64_t>(1, (n + GV_COLS - 1) / GV_COLS);
  double *part = nullptr;
  GPGP_CUDA(cudaMallocAsync((void **)&part, (size_t)n * nchunk * sizeof(double), s));
  dim3 grid((unsigned)((n + GV_ROWS - 1) / GV_ROWS), (unsigned)nchunk);
  trmv_n_kernel<<<grid, GV_ROWS, 0, s>>>(n, W, ldw, x, part);
  GPGP_CHECK_LAUNCH();
  gemv_reduce_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, nchunk, part, 1.0, 0.0, y);
  GPGP_CHECK_LAUNCH();
  GPGP_CUDA(cudaFreeAsync(part, s));
}

void gemv64(cudaStream_t s, bool trans, int64_t M, int64_t N, double alpha, const double *A,
            int64_t lda, const double *x, double beta, double *y) {
  if (trans) {
    if (N == 0) return;
    if (M >= 4 * GT_ROWS && N < 8 * device_sms()) {  // fewer than two warps to a sub-partition
      const int64_t nch = (M + GT_ROWS - 1) / GT_ROWS;
      double *part = nullptr;
      GPGP_CUDA(cudaMallocAsync((void **)&part, (size_t)N * nch * sizeof(double), s));
      gemv_t_part_kernel<<<dim3((unsigned)((N * 32 + 255) / 256), (unsigned)nch), 256, 0, s>>>(M, N, A, lda, x, part);
      GPGP_CHECK_LAUNCH();
      gemv_reduce_kernel<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(N, (int)nch, part, alpha, beta, y);
      GPGP_CHECK_LAUNCH();
      GPGP_CUDA(cudaFreeAsync(part, s));
      return;
    }
    gemv_t_kernel<<<(unsigned)((N * 32 + 255) / 256), 256, 0, s>>>(M, N, A, lda, x, y, alpha, beta);
    GPGP_CHECK_LAUNCH();
    return;
  }
  if (M == 0) return;
  const int nchunk = (int)std::max<int64_t>(1, (N + GV_COLS - 1) / GV_COLS);
  // partial sums of the column chunks: stream-ordered scratch of this call
  double *part = nullptr;
  GPGP_CUDA(cudaMallocAsync((void **)&part, (size_t)M * nchunk * sizeof(double), s));
  dim3 grid((unsigned)((M + GV_ROWS - 1) / GV_ROWS), (unsigned)nchunk);
  gemv_n_kernel<<<grid, GV_ROWS, 0, s>>>(M, N, A, lda, x, part);
  GPGP_CHECK_LAUNCH();
  gemv_reduce_kernel<<<(unsigned)((M + 255) / 256), 256, 0, s>>>(M, nchunk, part, alpha,
                                                                  beta, y);
  GPGP_CHECK_LAUNCH();
  GPGP_CUDA(cudaFreeAsync(part, s));
}

// ---------------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------------
__global__ void sum_vec_kernel(const double *__restrict__ v, int64_t n, double *__restrict__ out) {
  __shared__ double red[256];
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += 256) s += v[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) red[threadIdx.x] += red[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = red[0];
}

void sum_vec(cudaStream_t s, const double *v, int64_t n, double *out) {
  sum_vec_kernel<<<1, 256, 0, s>>>(v, n, out);
  GPGP_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// LU with partial pivoting of a small general matrix (the symmetric indefinite
// Schur complement of the bad sites in the non-log-concave fits, where the
// reference takes Matrix::lu of K + diag(V), R/laplace.R:113, R/ep.R:128)
// ---------------------------------------------------------------------------
// Column k: one CTA picks the pivot (largest |A_ik|, i >= k, first index on
// ties), swaps rows k and p across all columns and divides the column below the
// pivot by it; a grid then applies the rank-1 update to the trailing block.
__global__ void __launch_bounds__(256) lu_pivot_kernel(double *__restrict__ A, int64_t n, int64_t lda,
                                                       int64_t k, int *__restrict__ piv,
                                                       int *__restrict__ status) {
  __shared__ double bv[256];
  __shared__ int64_t bi[256];
  if (*(volatile int *)status != 0) return;
  double best = -1.0;
  int64_t arg = k;
  for (int64_t i = k + threadIdx.x; i < n; i += 256) {
    const double v = fabs(A[i + k * lda]);
    if (v > best) {
      best = v;
      arg = i;
    }
  }
  bv[threadIdx.x] = best;
  bi[threadIdx.x] = arg;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) {
      const double o = bv[threadIdx.x + st];
      const int64_t oi = bi[threadIdx.x + st];
      if (o > bv[threadIdx.x] || (o == bv[threadIdx.x] && oi < bi[threadIdx.x])) {
        bv[threadIdx.x] = o;
        bi[threadIdx.x] = oi;
      }
    }
    __syncthreads();
  }
  const int64_t p = bi[0];
  if (!(bv[0] > 0.0)) {  // exactly singular (or NaN)
    if (threadIdx.x == 0) atomicCAS(status, 0, (int)(k + 1));
    return;
  }
  if (threadIdx.x == 0) piv[k] = (int)p;
  if (p != k)
    for (int64_t j = threadIdx.x; j < n; j += 256) {
      const double t = A[k + j * lda];
      A[k + j * lda] = A[p + j * lda];
      A[p + j * lda] = t;
    }
  __syncthreads();
  const double r = 1.0 / A[k + k * lda];
  for (int64_t i = k + 1 + threadIdx.x; i < n; i += 256) A[i + k * lda] *= r;
}

__global__ void lu_update_kernel(double *__restrict__ A, int64_t n, int64_t lda, int64_t k,
                                 const int *__restrict__ status) {
  if (*(volatile const int *)status != 0) return;
  const int64_t m = n - k - 1;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m * m;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = k + 1 + e % m, j = k + 1 + e / m;
    A[i + j * lda] -= A[i + k * lda] * A[k + j * lda];
  }
}

void getrf(cudaStream_t s, double *A, int64_t n, int64_t lda, int *piv, int *status) {
  for (int64_t k = 0; k < n; ++k) {
    lu_pivot_kernel<<<1, 256, 0, s>>>(A, n, lda, k, piv, status);
    GPGP_CHECK_LAUNCH();
    const int64_t m = n - k - 1;
    if (m > 0) {
      const unsigned g = (unsigned)std::min<int64_t>((m * m + 255) / 256, 4 * 152);
      lu_update_kernel<<<g, 256, 0, s>>>(A, n, lda, k, status);
      GPGP_CHECK_LAUNCH();
    }
  }
}

// X <- A^-1 X with the factors of getrf: the row interchanges in order, then the
// unit lower and the upper substitutions. One warp per right-hand side; the
// lanes share each row's dot product.
__global__ void getrs_kernel(const double *__restrict__ LU, int64_t n, int64_t lda, const int *__restrict__ piv,
                             double *__restrict__ X, int64_t m, int64_t ldx, const int *__restrict__ status) {
  const int64_t c = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
  const int lane = threadIdx.x & 31;
  if (c >= m || *(volatile const int *)status != 0) return;
  double *x = X + c * ldx;
  if (lane == 0)
    for (int64_t k = 0; k < n; ++k) {
      const int64_t p = piv[k];
      if (p != k) {
        const double t = x[k];
        x[k] = x[p];
        x[p] = t;
      }
    }
  __syncwarp();
  for (int64_t i = 1; i < n; ++i) {  // unit lower
    double acc = 0.0;
    for (int64_t j = lane; j < i; j += 32) acc = fma(LU[i + j * lda], x[j], acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) x[i] -= acc;
    __syncwarp();
  }
  for (int64_t i = n - 1; i >= 0; --i) {  // upper
    double acc = 0.0;
    for (int64_t j = i + 1 + lane; j < n; j += 32) acc = fma(LU[i + j * lda], x[j], acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) x[i] = (x[i] - acc) / LU[i + i * lda];
    __syncwarp();
  }
}

void getrs(cudaStream_t s, const double *LU, int64_t n, int64_t lda, const int *piv, double *X, int64_t m,
           int64_t ldx, const int *status) {
  if (n <= 0 || m <= 0) return;
  getrs_kernel<<<(unsigned)((m + 7) / 8), 256, 0, s>>>(LU, n, lda, piv, X, m, ldx, status);
  GPGP_CHECK_LAUNCH();
}

}  // namespace gpgp
