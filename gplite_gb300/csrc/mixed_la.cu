// Blocked algorithms built on the sliced tensor-core GEMM (mixed.cu): Cholesky,
// triangular inverse, B^-1 = L^-T L^-1, the predictive variance's solve or product, and Gram
// products. Outputs have the same meaning and layout as the FP64 routines of dense.cu; only
// the contractions differ: products of fixed-point row slices, accumulated exactly and
// summed in FP64, of 32 bits (S = 4, the mixed precision) or 63 (S = OZ_FP64, the FP64 path
// of large n).
//
// Cholesky is two-level right-looking: outer panels of NBO columns (384: faster
// at n = 16384 than 256 or 512), each factored in 64-wide blocks (factor_panel); one
// sliced SYRK with K = NBO then updates the trailing matrix, so every trailing element is
// rewritten in FP64 once per outer panel.
#include <math.h>

#include <algorithm>
#include <vector>

#include "common.cuh"
#include "model.cuh"

namespace gpgp {

// potrf_panel_inv_kernel lives in dense.cu
__global__ void potrf_panel_inv_kernel(double *__restrict__ A21, int64_t m, int kb, int64_t lda,
                                       const double *__restrict__ W, const int *__restrict__ status);

namespace {

#ifndef GPGP_NBO
#define GPGP_NBO 384
#endif
constexpr int64_t NBO = GPGP_NBO;  // outer panel width of the Cholesky (a build-time tuning knob)
static_assert(NBO % NB == 0, "an outer panel is whole blocks wherever rows lie below it");
// Lookahead: a trailing update of at least LOOK_MIN_ROWS rows leaves LOOK_PANEL_SMS
// SMs to the next panel's factorisation, whose GEMMs are capped to them.
// The panel's rows below (panel_block) take most of that share, and the chain's clusters
// need four free SMs of one GPC: mixed step n = 16384 with 20 / 32 / 48 / 56 / 72 SMs left:
// 92.9 / 82.6 / 78.6 / 77.9 / 80.6 ms, mixed Laplace n = 8192 86.9 / 81.5 / 80.6 / 78.6 /
// 80.6, FP64 step n = 8192 33.2 / 31.8 / 31.7 / 30.8 / 31.7. From 3072 rows on: mixed
// Laplace 85.1 (32 SMs).
constexpr int64_t LOOK_MIN_ROWS = 6144;
constexpr int LOOK_PANEL_SMS = 56;

// The 64-wide blocks of the outer panel [k0, k0 + kbo). What the next diagonal block
// waits for is kept apart from the rest:
//  - chain (stream x): the factor and inverse W of the diagonal block, the panel's rows
//    L_p = A_p W^T and the next diagonal block's update by its own rows, on the FP64 pipe;
//  - the rest of the panel (stream z, after the panel's rows): the update of the panel's
//    lower triangle beside that block. The chain waits for it after its next diagonal
//    block;
//  - bulk (stream y, after the panel's rows): the rows below the panel, L_b = A_b W^T,
//    and their update of the panel's remaining columns (panel_block).
// x, y and z may be the same stream (the single-stream schedule; same products in the
// same order, so the same factor). With more streams the bulk takes no status word: the
// chain's diagonal kernels may set it while they run.
void factor_panel(cudaStream_t x, cudaStream_t y, cudaStream_t z, const SideStream *sd, double *A, int64_t n,
                  int64_t lda, double *Winv, double *logdet_part, int *status, int *err, int64_t k0, int64_t kbo,
                  int S) {
  const bool two = x != y;
  const int64_t pend = k0 + kbo;  // first row / column after the panel
  const int64_t mb = n - pend;    // rows below the panel
  const int *sst = two ? nullptr : status;
  bool rest = false;              // the block before left work on z
  for (int64_t j0 = k0; j0 < pend; j0 += NB) {
    const int jb = (int)std::min<int64_t>(NB, pend - j0);
    const int64_t blk = j0 / NB;
    double *Wb = Winv + blk * NB * NB;
    potrf_diag(x, A + j0 + j0 * lda, jb, lda, Wb, logdet_part + blk, status, j0, 0, 0, 0, 1);
    const int64_t mp = pend - (j0 + jb);  // panel rows below the block
    double *Ln = A + (j0 + NB) + j0 * lda;
    if (mp > 0) {
      if (two && rest) GPGP_CUDA(cudaStreamWaitEvent(x, sd->e, 0));
      potrf_panel_inv_kernel<<<(unsigned)((mp + 3) / 4), 256, 0, x>>>(Ln, mp, jb, lda, Wb, status);
      GPGP_CHECK_LAUNCH();
    }
    rest = mp > NB;
    if (two) {
      GPGP_CUDA(cudaEventRecord(sd->c, x));
      if (rest) GPGP_CUDA(cudaStreamWaitEvent(z, sd->c, 0));
      if (mb > 0) GPGP_CUDA(cudaStreamWaitEvent(y, sd->c, 0));
    }
    if (mp > 0) syrk_block(x, Ln, lda, (int)std::min<int64_t>(NB, mp), A + (j0 + NB) * (lda + 1));
    if (rest) {
      const int64_t mr = mp - NB, i0 = j0 + 2 * NB;  // rows from i0 on
      double *Lr = A + i0 + j0 * lda;
      gemm64(z, false, true, mr, NB, jb, -1.0, Lr, lda, Ln, lda, 1.0, A + i0 + (j0 + NB) * lda, lda, false, 0);
      gemm64(z, false, true, mr, mr, jb, -1.0, Lr, lda, Lr, lda, 1.0, A + i0 + i0 * lda, lda, true, 0);
      if (two) GPGP_CUDA(cudaEventRecord(sd->e, z));
    }
    if (mb > 0) panel_block(y, S, A, lda, pend, n, j0, Wb, (int)(mp / NB), err, sst);
  }
  if (two) {  // the panel is complete on x once the bulk is (z's work precedes it or x's)
    GPGP_CUDA(cudaEventRecord(sd->b, y));
    GPGP_CUDA(cudaStreamWaitEvent(x, sd->b, 0));
  }
}

}  // namespace

thread_local bool tl_lean = false;

void potrf_mixed(cudaStream_t s, double *A, int64_t n, int64_t lda, double *Winv,
                 double *logdet_part, int *status, int *err, const SideStream *side, int S) {
  SplitBuf a(s);  // the panel as the trailing update's operand
  if (S == OZ_FP64) {
    if (!with_scratch([&] { a.bind(n, NBO, S); })) {
      potrf(s, A, n, lda, Winv, logdet_part, status, 1);
      return;
    }
  } else {
    a.bind(n, NBO, S);
  }
  cudaStreamCaptureStatus cap_st = cudaStreamCaptureStatusNone;
  GPGP_CUDA(cudaStreamIsCapturing(s, &cap_st));
  // Per-kernel timers (tl_kt) time each launch alone, so a profiled call runs the
  // single-stream schedule.
  if (!side || !side->s3 || n <= 2 * NBO || cap_st != cudaStreamCaptureStatusNone || tl_kt) {
    for (int64_t k0 = 0; k0 < n; k0 += NBO) {
      const int64_t kbo = std::min<int64_t>(NBO, n - k0);
      factor_panel(s, s, s, nullptr, A, n, lda, Winv, logdet_part, status, err, k0, kbo, S);
      const int64_t m2 = n - k0 - kbo;
      if (m2 > 0) {
        double *P = A + (k0 + kbo) + k0 * lda;
        oz_split(s, P, lda, 0, m2, kbo, &a.sp);
        oz_gemm(s, a.sp, 0, a.sp, 0, m2, m2, 0, (kbo + 63) / 64, 0, -1.0, 1.0,
                A + (k0 + kbo) + (k0 + kbo) * lda, lda, true, err, status);
      }
    }
    return;
  }
  // Lookahead. The side stream factors the panels; the main stream applies each
  // finished panel p to the next panel's columns first, releases the side stream
  // (event a), and then applies p to the rest of the trailing matrix while panel
  // p + 1 is factored beside it (the two touch disjoint columns). Every product
  // is the one the plain schedule computes, so the factor is the same.
  cudaStream_t x = side->s;
  GPGP_CUDA(cudaEventRecord(side->fork, s));
  GPGP_CUDA(cudaStreamWaitEvent(x, side->fork, 0));
  // The main stream waits for the side stream before the buffers above are freed,
  // also when an error leaves the loop early (destroyed before them).
  struct Join {
    const SideStream *sd;
    cudaStream_t main;
    ~Join() {
      for (cudaStream_t o : {sd->s2, sd->s3}) {  // (an error may leave the panel loop early)
        cudaEventRecord(sd->b, o);
        cudaStreamWaitEvent(sd->s, sd->b, 0);
      }
      cudaEventRecord(sd->l, sd->s);
      cudaStreamWaitEvent(main, sd->l, 0);
    }
  } join{side, s};
  const int sms = oz_sms();
  int panel_cap = 0;
  for (int64_t k0 = 0; k0 < n; k0 += NBO) {
    const int64_t kbo = std::min<int64_t>(NBO, n - k0);
    {
      OzGridCap cap(panel_cap);
      factor_panel(x, side->s2, side->s3, side, A, n, lda, Winv, logdet_part, status, err, k0, kbo, S);
    }
    GPGP_CUDA(cudaEventRecord(side->l, x));
    GPGP_CUDA(cudaStreamWaitEvent(s, side->l, 0));
    const int64_t m2 = n - k0 - kbo;
    if (m2 <= 0) break;
    double *P = A + (k0 + kbo) + k0 * lda;
    double *C = A + (k0 + kbo) + (k0 + kbo) * lda;
    oz_split(s, P, lda, 0, m2, kbo, &a.sp);
    const int64_t nb2 = std::min<int64_t>(NBO, m2);
    oz_gemm(s, a.sp, 0, a.sp, 0, m2, nb2, 0, (kbo + 63) / 64, 0, -1.0, 1.0, C, lda, true, err, status);
    GPGP_CUDA(cudaEventRecord(side->a, s));
    GPGP_CUDA(cudaStreamWaitEvent(x, side->a, 0));
    const int64_t m3 = m2 - nb2;
    panel_cap = 0;
    if (m3 > 0) {
      const bool share = m3 >= LOOK_MIN_ROWS && sms > 2 * LOOK_PANEL_SMS;
      if (share) panel_cap = LOOK_PANEL_SMS;
      OzGridCap cap(share ? sms - LOOK_PANEL_SMS : 0);
      // no status word: the side stream's diagonal kernels may set it while this
      // launch runs, and every role of a GEMM CTA must see the same value
      oz_gemm(s, a.sp, nb2, a.sp, nb2, m3, m3, 0, (kbo + 63) / 64, 0, -1.0, 1.0, C + nb2 + nb2 * lda, lda,
              true, err, nullptr);
    }
  }
}

// ---------------------------------------------------------------------------
// recursive triangular inverse: W = L^-1, W21 = -W22 (L21 W11)
// ---------------------------------------------------------------------------
// every 64 x 64 diagonal-block inverse into W's diagonal, one kernel
__global__ void put_diag_inverses_kernel(const double *__restrict__ Winv, int64_t n, double *__restrict__ W,
                                         int64_t ldw) {
  const int64_t blk = blockIdx.x, k0 = blk * NB;
  const int kb = (int)((n - k0) < NB ? (n - k0) : NB);
  const double *src = Winv + blk * NB * NB;
  for (int idx = threadIdx.x; idx < NB * NB; idx += blockDim.x) {
    const int r = idx % NB, c = idx / NB;
    if (r < kb && c < kb) W[(k0 + r) + (k0 + c) * ldw] = src[r + c * NB];
  }
}

constexpr int64_t TRTRI_BASE = 512;  // diagonal blocks inverted level by level, batched

// Batched scratch for a level: `count` split operands of rows x K each.
static size_t split_batch_bytes(int64_t rows, int64_t K, int S) {
  return (oz_split_bytes(rows, K, S) + 1023) / 1024 * 1024;
}
struct SplitBatch {
  void *p = nullptr;
  cudaStream_t s = nullptr;
  OzSplit sp;
  SplitBatch(cudaStream_t st, int64_t rows, int64_t K, int64_t count, int S) : s(st) {
    const size_t per = split_batch_bytes(rows, K, S);
    if (cudaMallocAsync(&p, per * count, st) != cudaSuccess) {
      p = nullptr;
      (void)cudaGetLastError();
      throw std::bad_alloc();
    }
    oz_split_bind(p, rows, K, &sp, S);
    sp.bstride_ex = (int64_t)(per / sizeof(int));
    sp.bstride_sl = (int64_t)(per / sizeof(uint16_t));
  }
  ~SplitBatch() {
    if (p) cudaFreeAsync(p, s);
  }
};

// One level of the blocked inverse for every full b x b diagonal block at
// offsets k b (k < count), whose two halves are already inverted:
// W21 = -W22 (L21 W11), all blocks of the level in two batched GEMMs.
static void trtri_level(cudaStream_t s, const double *L, int64_t lda, double *W, int64_t ldw, int64_t b,
                        int64_t count, double *T, int *err, int S) {
  const int64_t h = b / 2;
  {
    SplitBatch a(s, h, h, count, S), bb(s, h, h, count, S);
    oz_split_batched(s, L + h, lda, b * (lda + 1), 0, h, h, &a.sp, count);
    oz_split_batched(s, W, ldw, b * (ldw + 1), 1, h, h, &bb.sp, count);
    oz_gemm_batched(s, a.sp, 0, bb.sp, 0, h, h, 0, bb.sp.nkb, 2, 1.0, 0.0, T, h, h * h, false, err, nullptr, 0,
                    count);
  }
  {
    SplitBatch a(s, h, h, count, S), bb(s, h, h, count, S);
    oz_split_batched(s, W + h + h * ldw, ldw, b * (ldw + 1), 0, h, h, &a.sp, count);
    oz_split_batched(s, T, h, h * h, 1, h, h, &bb.sp, count);
    oz_gemm_batched(s, a.sp, 0, bb.sp, 0, h, h, 0, a.sp.nkb, 3, -1.0, 0.0, W + h, ldw, b * (ldw + 1), false, err,
                    nullptr, 0, count);
  }
}

// recursive triangular inverse: W = L^-1, W21 = -W22 (L21 W11). Nodes already
// inverted (64-blocks from the factorisation, and full aligned 128 / 256 / 512
// blocks from the batched levels) are skipped; above the base the split points
// are multiples of the base so that its blocks line up.
static void trtri_rec(cudaStream_t s, const double *L, int64_t n, int64_t lda, int64_t off, int64_t ntot,
                      double *W, int64_t ldw, double *T, int *err, int S) {
  if (n <= NB) return;
  if ((n == 128 || n == 256 || n == TRTRI_BASE) && off % n == 0 && off + n <= ntot) return;
  const int64_t g = n > TRTRI_BASE ? TRTRI_BASE : NB;
  const int64_t n1 = ((n / 2) + g - 1) / g * g;
  const int64_t n2 = n - n1;
  trtri_rec(s, L, n1, lda, off, ntot, W, ldw, T, err, S);
  trtri_rec(s, L + n1 + n1 * lda, n2, lda, off + n1, ntot, W + n1 + n1 * ldw, ldw, T, err, S);
  // T = L21 W11  (n2 x n1): A = L21 (rows n2, K n1), B rows j = columns of W11 (W11[k, j], k >= j)
  {
    SplitBuf a(s, n2, n1, S), b(s, n1, n1, S);
    oz_split(s, L + n1, lda, 0, n2, n1, &a.sp);
    oz_split(s, W, ldw, 1, n1, n1, &b.sp);
    oz_gemm(s, a.sp, 0, b.sp, 0, n2, n1, 0, b.sp.nkb, 2, 1.0, 0.0, T, n2, false, err);
  }
  // W21 = -W22 T  (n2 x n1): A = W22 (rows n2, K n2, lower: k <= i), B rows j = columns of T
  {
    SplitBuf a(s, n2, n2, S), b(s, n1, n2, S);
    oz_split(s, W + n1 + n1 * ldw, ldw, 0, n2, n2, &a.sp);
    oz_split(s, T, n2, 1, n1, n2, &b.sp);
    oz_gemm(s, a.sp, 0, b.sp, 0, n2, n1, 0, a.sp.nkb, 3, -1.0, 0.0, W + n1, ldw, false, err);
  }
}

__global__ void zero_upper_kernel(double *W, int64_t n, int64_t ldw) {
  for (int64_t j = blockIdx.y; j < n; j += gridDim.y)
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < j;
         i += (int64_t)gridDim.x * blockDim.x)
      W[i + j * ldw] = 0.0;
}

void trtri_mixed(cudaStream_t s, const double *L, int64_t n, int64_t lda, const double *Winv,
                 double *W, int64_t ldw, int *err, int S) {
  if (n <= 0) return;
  dim3 g((unsigned)std::min<int64_t>((n + 255) / 256, 64), (unsigned)std::min<int64_t>(n, 65535));
  zero_upper_kernel<<<g, 256, 0, s>>>(W, n, ldw);
  GPGP_CHECK_LAUNCH();
  put_diag_inverses_kernel<<<(unsigned)((n + NB - 1) / NB), 256, 0, s>>>(Winv, n, W, ldw);
  GPGP_CHECK_LAUNCH();
  double *T = nullptr;
  const int64_t h = (n / 2 + TRTRI_BASE) * (n / 2 + TRTRI_BASE);
  if (cudaMallocAsync((void **)&T, (size_t)h * sizeof(double), s) != cudaSuccess) {
    (void)cudaGetLastError();
    throw std::bad_alloc();
  }
  try {
    // the full aligned diagonal blocks of 128, 256 and 512, all blocks of a size at once
    for (int64_t b = 2 * NB; b <= TRTRI_BASE; b *= 2)
      if (n / b > 0) trtri_level(s, L, lda, W, ldw, b, n / b, T, err, S);
    trtri_rec(s, L, n, lda, 0, n, W, ldw, T, err, S);
  } catch (...) {
    cudaFreeAsync(T, s);
    throw;
  }
  GPGP_CUDA(cudaFreeAsync(T, s));
}

void lauum_mixed(cudaStream_t s, const double *W, int64_t n, int64_t ldw, double *Binv,
                 int64_t ldb, int *err, int S) {
  // Binv_ij = sum_k W_ki W_kj (k >= max(i, j)); operand rows = columns of W
  SplitBuf a(s, n, n, S);
  oz_split(s, W, ldw, 1, n, n, &a.sp);
  oz_gemm(s, a.sp, 0, a.sp, 0, n, n, 0, a.sp.nkb, 1, 1.0, 0.0, Binv, ldb, true, err);
}

// X = L^-1 R in place (n x m), right-looking on two levels: a 64-row block is
// multiplied by its diagonal block's inverse and updates the rest of its outer block of
// TRSM_OUTER rows (K = 64); the rows below take one product with K = TRSM_OUTER, so
// that they are rewritten n / TRSM_OUTER times. Inverses of larger diagonal blocks would
// need fewer launches, but 128-row ones made the predictive variance 1.6 times and
// 512-row ones 4 times less accurate.
constexpr int64_t TRSM_OUTER = 512;

// For few right-hand sides the FP64 pipe's products are small ones (gemm64_small_kernel, up to
// 151 tiles of 64 x 64), and the sliced solve's five launches to a block cost more: gp_pred
// with variance, FP64 pipe against slices, at the last m on the one side of 180 tiles and the
// first measured on the other:
//   n = 900   m = 555 (135 tiles) 0.83 / 0.99 ms   777 (195) 1.32 / 1.07
//   n = 2000  m = 300 (160)       1.94 / 2.04      350 (192) 2.43 / 2.06
//   n = 4500  m = 111 (142)       3.97 / 4.30      133 (213) 5.87 / 4.35
//   n = 10000 m = 1 (157)         6.31 / 8.63, n = 12000 m = 16 (188) 11.83 / 11.32
constexpr int64_t TRSM_TILES = 180;
bool trsm_takes_slices(int64_t n, int64_t m) {
  return n >= SLICED_MIN && ((n + 63) / 64) * ((m + 63) / 64) >= TRSM_TILES;
}

size_t trsm_sliced_bytes(int64_t n, int64_t m, int S) {
  return (size_t)((n + NB - 1) / NB) * split_batch_bytes(NB, NB, S) + oz_split_bytes(n, TRSM_OUTER, S) +
         oz_split_bytes(m, TRSM_OUTER, S);
}

void trsm_sliced(cudaStream_t s, const double *L, int64_t n, int64_t lda, const double *Winv, double *R, int64_t m,
                 int64_t ldr, int *err, int S) {
  if (n <= 0 || m <= 0) return;
  const int64_t nblk = (n + NB - 1) / NB;
  SplitBatch w(s, NB, NB, nblk, S);  // the diagonal blocks' inverses, split at once
  oz_split_batched(s, Winv, NB, NB * NB, 0, NB, NB, &w.sp, nblk);
  SplitBuf a(s, n, TRSM_OUTER, S), x(s, m, TRSM_OUTER, S);
  for (int64_t o0 = 0; o0 < n; o0 += TRSM_OUTER) {
    const int64_t oend = std::min<int64_t>(o0 + TRSM_OUTER, n);
    for (int64_t k0 = o0; k0 < oend; k0 += NB) {
      const int64_t kb = std::min<int64_t>(NB, n - k0), rest = oend - k0 - kb;
      OzSplit wk = w.sp;
      wk.ex += k0 / NB * wk.bstride_ex;
      wk.sl += k0 / NB * wk.bstride_sl;
      oz_split(s, R + k0, ldr, 1, m, kb, &x.sp);
      oz_gemm(s, wk, 0, x.sp, 0, kb, m, 0, 1, 0, 1.0, 0.0, R + k0, ldr, false, err);
      if (rest <= 0) break;
      oz_split(s, R + k0, ldr, 1, m, kb, &x.sp);
      oz_split(s, L + (k0 + kb) + k0 * lda, lda, 0, rest, kb, &a.sp);
      oz_gemm(s, a.sp, 0, x.sp, 0, rest, m, 0, 1, 0, -1.0, 1.0, R + k0 + kb, ldr, false, err);
    }
    const int64_t below = n - oend;
    if (below <= 0) break;
    oz_split(s, R + o0, ldr, 1, m, oend - o0, &x.sp);
    oz_split(s, L + oend + o0 * lda, lda, 0, below, oend - o0, &a.sp);
    oz_gemm(s, a.sp, 0, x.sp, 0, below, m, 0, a.sp.nkb, 0, -1.0, 1.0, R + oend, ldr, false, err);
  }
}

// The Gram products of FITC and of the random features: few output tiles, long K. K is
// cut into as many ranges as give every SM a tile (each with exponents of its own), the
// ranges are one batched product, and the partials are added in order. 65536 x 256: the
// FP64 pipe took 7.0 ms, this 0.45 ms, most of it the two splits.
// The partials are kept in as many slots as 128 MB hold (at least one) and added whenever
// the slots are full, so that they do not grow with n (M = 4096, n = 65536: 37 partials
// of 134 MB each).
constexpr int64_t GRAM_PASS_BYTES = (int64_t)1 << 27;

struct GramPlan {
  int64_t kc, full, rem, nz;  // K of a range, full ranges, rows after them, ranges
  int64_t pass, slots;        // ranges to a product, partials kept
};
static GramPlan gram_plan(int64_t n, int64_t M, int64_t N, int sms) {
  GramPlan g;
  const int64_t tiles = ((M + 127) / 128) * ((N + 63) / 64);
  const int64_t want = std::max<int64_t>(1, sms / tiles);
  // a range: a multiple of the 256 K that are summed exactly, and small enough that the
  // split operands of one pass over the SMs stay below 128 MB each
  const int64_t krow = (int64_t)oz_split_bytes(std::max(M, N), 256, OZ_FP64) / 256;  // bytes per K
  g.kc = ((n + want - 1) / want + 255) / 256 * 256;
  g.kc = std::max<int64_t>(256, std::min<int64_t>(g.kc, GRAM_PASS_BYTES / (krow * want) / 256 * 256));
  g.full = n / g.kc;
  g.rem = n - g.full * g.kc;
  g.nz = g.full + (g.rem > 0 ? 1 : 0);
  g.pass = std::max<int64_t>(1, GRAM_PASS_BYTES / (krow * g.kc));
  g.slots = std::min(g.nz, std::max<int64_t>(1, GRAM_PASS_BYTES / (int64_t)sizeof(double) / (M * N)));
  return g;
}

size_t gram_sliced_bytes(int64_t n, int64_t M, int64_t N, int sms) {
  const GramPlan g = gram_plan(n, M, N, sms);
  const int64_t cnt = std::min(std::min(g.pass, g.slots), std::max<int64_t>(g.full, 1));
  return (size_t)cnt * (split_batch_bytes(M, g.kc, OZ_FP64) + split_batch_bytes(N, g.kc, OZ_FP64)) +
         (size_t)(g.slots * M * N) * sizeof(double);
}

void gram_sliced(cudaStream_t s, const double *A, int64_t lda, const double *B, int64_t ldb, int64_t n, int64_t M,
                 int64_t N, double *C, int64_t ldc, int *err) {
  if (M <= 0 || N <= 0) return;
  const GramPlan g = gram_plan(n, M, N, oz_sms());
  const int64_t kc = g.kc;
  DBuf P;
  P.alloc(s, (size_t)g.slots * M * N);
  int64_t used = 0;
  bool go_on = false;
  auto flush = [&] {
    splitk_reduce(s, M, N, (int)used, P.p, 1.0, 0.0, C, ldc, false, go_on);
    used = 0;
    go_on = true;
  };
  for (int64_t z0 = 0, cnt; z0 < g.full; z0 += cnt) {
    cnt = std::min(std::min(g.pass, g.full - z0), g.slots - used);
    SplitBatch a(s, M, kc, cnt, OZ_FP64), b(s, N, kc, cnt, OZ_FP64);
    oz_split_batched(s, A + z0 * kc, lda, kc, 1, M, kc, &a.sp, cnt);
    oz_split_batched(s, B + z0 * kc, ldb, kc, 1, N, kc, &b.sp, cnt);
    oz_gemm_batched(s, a.sp, 0, b.sp, 0, M, N, 0, kc / 64, 0, 1.0, 0.0, P.p + used * M * N, M, M * N, false, err,
                    nullptr, 0, cnt);
    used += cnt;
    if (used == g.slots) flush();
  }
  if (g.rem > 0) {
    SplitBuf a(s, M, g.rem, OZ_FP64), b(s, N, g.rem, OZ_FP64);
    oz_split(s, A + g.full * kc, lda, 1, M, g.rem, &a.sp);
    oz_split(s, B + g.full * kc, ldb, 1, N, g.rem, &b.sp);
    oz_gemm(s, a.sp, 0, b.sp, 0, M, N, 0, a.sp.nkb, 0, 1.0, 0.0, P.p + used * M * N, M, false, err);
    ++used;
  }
  if (used > 0) flush();
}

void trmv_sumsq_mixed(cudaStream_t s, const double *W, int64_t n, int64_t ldw, const double *R,
                      int64_t m, int64_t ldr, double *out, int *err) {
  // T = W R (n x m): A = W (rows n, K n, k <= i), B rows j = columns of R
  double *T = nullptr;
  if (cudaMallocAsync((void **)&T, (size_t)n * m * sizeof(double), s) != cudaSuccess) {
    (void)cudaGetLastError();
    throw std::bad_alloc();
  }
  {
    SplitBuf a(s, n, n, 4), b(s, m, n, 4);
    oz_split(s, W, ldw, 0, n, n, &a.sp);
    oz_split(s, R, ldr, 1, m, n, &b.sp);
    oz_gemm(s, a.sp, 0, b.sp, 0, n, m, 0, a.sp.nkb, 3, 1.0, 0.0, T, n, false, err);
  }
  col_sumsq(s, T, n, m, n, out);
  GPGP_CUDA(cudaFreeAsync(T, s));
}

}  // namespace gpgp

// ---------------------------------------------------------------------------
// self-test entry point: sliced GEMM against the FP64 GEMM on random data
// ---------------------------------------------------------------------------
namespace {
__global__ void fill_random_kernel(double *a, int64_t n, uint64_t seed, double scale_spread) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * (uint64_t)(i + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    const double u = (double)(z >> 11) * (1.0 / 9007199254740992.0) - 0.5;
    // entries of varying magnitude exercise the per-row scaling
    const double mag = exp2(scale_spread * (double)((z >> 3) & 7) / 7.0 - scale_spread / 2);
    a[i] = u * mag;
  }
}

__global__ void max_abs_kernel(const double *a, const double *b, int64_t n, double *out) {
  __shared__ double sd[256], sm[256];
  double d = 0.0, m = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += 256) {
    d = fmax(d, fabs(a[i] - b[i]));
    m = fmax(m, fabs(b[i]));
  }
  sd[threadIdx.x] = d;
  sm[threadIdx.x] = m;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (threadIdx.x < st) {
      sd[threadIdx.x] = fmax(sd[threadIdx.x], sd[threadIdx.x + st]);
      sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + st]);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = sd[0];
    out[1] = sm[0];
  }
}
}  // namespace

extern "C" gpgp_status gpgp_mixed_selftest(gpgp_ctx *ctx, int64_t M, int64_t N, int64_t K,
                                           int32_t slices, double *max_rel_err) {
  using namespace gpgp;
  if (!ctx || M < 1 || N < 1 || K < 1 || !max_rel_err || (slices != 4 && slices != 5 && slices != OZ_FP64))
    return GPGP_EINVAL;
  cudaStream_t s = (cudaStream_t)gpgp_stream(ctx);
  KTBind bind(ctx);
  try {
    double *A = nullptr, *B = nullptr, *C1 = nullptr, *C2 = nullptr, *red = nullptr;
    int *err = nullptr;
    GPGP_CUDA(cudaMallocAsync((void **)&A, M * K * sizeof(double), s));
    GPGP_CUDA(cudaMallocAsync((void **)&B, N * K * sizeof(double), s));
    GPGP_CUDA(cudaMallocAsync((void **)&C1, M * N * sizeof(double), s));
    GPGP_CUDA(cudaMallocAsync((void **)&C2, M * N * sizeof(double), s));
    GPGP_CUDA(cudaMallocAsync((void **)&red, 4 * sizeof(double), s));
    GPGP_CUDA(cudaMallocAsync((void **)&err, sizeof(int), s));
    GPGP_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
    fill_random_kernel<<<256, 256, 0, s>>>(A, M * K, 12345, 8.0);
    fill_random_kernel<<<256, 256, 0, s>>>(B, N * K, 777, 8.0);
    fill_random_kernel<<<256, 256, 0, s>>>(C1, M * N, 99, 0.0);
    GPGP_CUDA(cudaMemcpyAsync(C2, C1, M * N * sizeof(double), cudaMemcpyDeviceToDevice, s));
    {
      void *pa = nullptr, *pb = nullptr;
      GPGP_CUDA(cudaMallocAsync(&pa, oz_split_bytes(M, K, slices), s));
      GPGP_CUDA(cudaMallocAsync(&pb, oz_split_bytes(N, K, slices), s));
      OzSplit sa, sb;
      oz_split_bind(pa, M, K, &sa, slices);
      oz_split_bind(pb, N, K, &sb, slices);
      oz_split(s, A, M, 0, M, K, &sa);
      oz_split(s, B, N, 0, N, K, &sb);
      // C1 = -A B^T + C1 (sliced) ; C2 = -A B^T + C2 (FP64)
      oz_gemm(s, sa, 0, sb, 0, M, N, 0, sa.nkb, 0, -1.0, 1.0, C1, M, false, err);
      gemm64(s, false, true, M, N, K, -1.0, A, M, B, N, 1.0, C2, M);
      max_abs_kernel<<<1, 256, 0, s>>>(C1, C2, M * N, red);
      cudaFreeAsync(pa, s);
      cudaFreeAsync(pb, s);
    }
    double h[2];
    int herr = 0;
    GPGP_CUDA(cudaMemcpyAsync(h, red, 2 * sizeof(double), cudaMemcpyDeviceToHost, s));
    GPGP_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s));
    GPGP_CUDA(cudaStreamSynchronize(s));
    cudaFreeAsync(A, s);
    cudaFreeAsync(B, s);
    cudaFreeAsync(C1, s);
    cudaFreeAsync(C2, s);
    cudaFreeAsync(red, s);
    cudaFreeAsync(err, s);
    GPGP_CUDA(cudaStreamSynchronize(s));
    *max_rel_err = h[0] / (h[1] > 0 ? h[1] : 1.0);
    if (herr) return GPGP_ETIMEOUT;
    return GPGP_OK;
  } catch (const CudaError &e) {
    (void)cudaGetLastError();
    return fail(ctx, GPGP_ECUDA, std::string("CUDA error ") + cudaGetErrorString(e.err) + " in " + e.what);
  } catch (const std::bad_alloc &) {
    return GPGP_EOOM;
  }
}

extern "C" gpgp_status gpgp_sliced_product_selftest(gpgp_ctx *ctx, int64_t M, int64_t N, int64_t K, int32_t slices,
                                                    const double *A, const double *B, double *C) {
  using namespace gpgp;
  if (!ctx || M < 1 || N < 1 || K < 1 || !A || !B || !C || (slices != 4 && slices != 5 && slices != OZ_FP64))
    return fail(ctx, GPGP_EINVAL, "invalid argument");
  return guarded(ctx, [&]() -> gpgp_status {
    GPGP_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    DBuf dA, dB, dC;
    IBuf err;
    copy_in(s, dA, A, (size_t)(M * K), false);
    copy_in(s, dB, B, (size_t)(N * K), false);
    dC.alloc(s, (size_t)(M * N));
    err.alloc(s, 1);
    GPGP_CUDA(cudaMemsetAsync(err.p, 0, sizeof(int), s));
    SplitBuf a(s, M, K, slices), b(s, N, K, slices);
    oz_split(s, dA.p, M, 0, M, K, &a.sp);
    oz_split(s, dB.p, N, 0, N, K, &b.sp);
    oz_gemm(s, a.sp, 0, b.sp, 0, M, N, 0, a.sp.nkb, 0, 1.0, 0.0, dC.p, M, false, err.p);
    int herr = 0;
    GPGP_CUDA(cudaMemcpyAsync(&herr, err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    GPGP_CUDA(cudaMemcpyAsync(C, dC.p, (size_t)(M * N) * sizeof(double), cudaMemcpyDeviceToHost, s));
    GPGP_CUDA(cudaStreamSynchronize(s));
    if (herr) throw WaitTimeout{};
    return GPGP_OK;
  });
}

extern "C" gpgp_status gpgp_tri_rows_selftest(gpgp_ctx *ctx, int64_t n, int64_t M, const double *L, const double *B,
                                              int32_t mode, double *X) {
  using namespace gpgp;
  if (!ctx || n < 1 || M < 1 || !L || !B || !X || (mode != 0 && mode != 1))
    return fail(ctx, GPGP_EINVAL, "invalid argument");
  return guarded(ctx, [&]() -> gpgp_status {
    GPGP_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    DBuf dL, dX;
    IBuf err;
    copy_in(s, dL, L, (size_t)(M * M), false);
    copy_in(s, dX, B, (size_t)(n * M), false);
    err.alloc(s, 1);
    GPGP_CUDA(cudaMemsetAsync(err.p, 0, sizeof(int), s));
    tri_rows(s, dL.p, M, M, dX.p, n, dX.p, n, n, mode, err.p);
    int herr = 0;
    GPGP_CUDA(cudaMemcpyAsync(&herr, err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    GPGP_CUDA(cudaMemcpyAsync(X, dX.p, (size_t)(n * M) * sizeof(double), cudaMemcpyDeviceToHost, s));
    GPGP_CUDA(cudaStreamSynchronize(s));
    if (herr) throw WaitTimeout{};
    return GPGP_OK;
  });
}
