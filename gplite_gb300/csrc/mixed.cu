// Dense products on the tcgen05 tensor cores through exact BF16 slicing (an
// Ozaki-style split), at the accuracy the slice count gives: S = 4 and 5 for the mixed
// precision, S = 8 for the FP64 path of large n.
//
// Every operand row is scaled by a power of two so that its largest entry is
// in [0.5, 1) and then cut into S 8-bit fixed-point slices (this paragraph and the next:
// S = 4 or 5)
//   x = 2^e * sum_t q_t 2^-8(t+1),  q_t integers in [-256, 256].
// Slice t is stored as the BF16 value q_t 2^-8t (exact: an 8-bit integer times
// a power of two), so the product of slices t and u already carries its level
// weight 2^-8(t+u) and products of different levels can share an accumulator.
// Levels 0, 1 and 2 get their own FP32 accumulators in TMEM, levels 3.. share
// a fourth: a level-l sum of up to 256 products has 24 significant bits for
// l <= 2, so those sums are exact in FP32; the shared deeper levels round at
// 2^-50 of the result. After every 256-wide K group the four accumulators are
// added into a double-float (hi, lo) pair; at the end of the tile the pair is
// turned into a double with integer instructions and added to C (one FP64 add):
//   (A B^T)_ij = 2^(e_i + f_j - 16) (P_0 + P_1 + P_2 + P_3+).
// The truncation error is ~2^-(8S+1) of the row maxima.
//
// The products are issued as few, wide instructions: the B slices are adjacent in
// shared memory, and A_t times B slices 0..3-t is one MMA of N = 64 (4 - t) whose
// column blocks are the accumulators of levels t..3. S = 4 takes 7 instructions per K
// step instead of 13, S = 5 takes 13 instead of 19. The tensor pipe runs N >= 128 at
// its full rate (4080 multiply-adds per clock; N = 64 takes 48 cycles, N = 128 64,
// N = 256 128), so a K step of S = 4 is 476 cycles at least. What bounds the kernel:
// at long K the MMAs (1.37 to 1.5 PFLOP/s at 4096^2 x 4096, S = 4; 1.15 with the issue
// loop inside one lane's branch), at K <= 384 the epilogue's integer work and C
// traffic (8192^2, lower-only off: K = 384 0.52 ms, K = 256 0.41, K = 64 0.41; 0.70,
// 0.60 and 0.63 with 64-bit tile arithmetic in every warp and a branch per converted
// output).
//
// Data path: slices are stored pre-tiled in the canonical no-swizzle K-major
// UMMA layout (8-row x 16-byte core matrices, 64-row x 32-K tiles), so one
// cp.async.bulk per slice moves a chunk to shared memory. The GEMM kernel is
// persistent and warp-specialised: a producer warp streams K chunks of the
// CTA's output tiles through a ring of shared-memory stages, an MMA warp
// issues tcgen05.mma into one of two TMEM accumulator sets and commits to
// mbarriers, and sixteen epilogue warps drain the other set with tcgen05.ld
// and update C while the next group accumulates. Every wait is bounded: on
// timeout the kernel records an error, drains what it issued, releases TMEM
// and returns.
#include <limits.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "bulk.cuh"
#include "common.cuh"
#include "dfloat.cuh"
#include "model.cuh"

namespace gpgp {

constexpr int OZ_GROUP_K = 256;         // K of an exactly accumulated group
constexpr int OZ_TR = 64;               // rows per slice tile
constexpr int OZ_BM = 128, OZ_BN = 64;  // output tile
constexpr int OZ_EPI_WARPS = 16;  // four per TMEM lane quarter, 16 columns each
constexpr int OZ_EPI_COLS = OZ_BN / (OZ_EPI_WARPS / 4);
constexpr int OZ_THREADS = 32 * (2 + OZ_EPI_WARPS);  // producer, MMA, epilogue

// S slices per operand. S = 4 and 5 (8S-bit fixed point): levels t + u <= S are kept
// (13 products, truncation 2^-33; 19 products, 2^-41), levels >= 3 in one accumulator.
// S = 8 (OZ_FP64; 63-bit fixed point, digits of at most 128): the products of levels
// 0..7 (36), each level in an accumulator of its own, all 512 columns of TMEM. An
// operand entry keeps its 53 bits down to 2^-10 of its row's largest, the sums are
// exact to 2^-62 of the product of both rows' scales (unless the digits of 256 products
// line up: a level's sum beyond 2^24, possible from the fifth on, rounds to units of 2^-46
// and finer), and the outputs of fits of 1000
// to 3000 points are as far from 64-bit references as with the FP64 pipe's products
// (prediction mean 4.1e-14 against 4.4e-14, variance 9.8e-14 / 9.8e-14, gradient
// 1.53e-12 / 1.54e-12: geometric means over 36 and 24 fits). With 7 slices, which are
// 14% faster at K = 384, the gradient's error was 1.3 times the FP64 pipe's.
template <int S>
struct OzCfg {
  static constexpr bool FP64 = S == OZ_FP64;
  static constexpr int BITS = FP64 ? 8 * S - 1 : 8 * S;  // fixed-point bits below the row's power of two
  static constexpr int TK = FP64 ? 16 : 32;       // K chunk (one pipeline stage)
  static constexpr int TILE = OZ_TR * TK;         // bf16 elements per slice tile
  static constexpr int GROUP = OZ_GROUP_K / TK;   // chunks per exactly accumulated group
  static constexpr int NACC = FP64 ? S : 4;       // accumulators (levels 0, 1, 2, >= 3; or one each)
  static constexpr int NSET = FP64 ? 1 : 2;       // accumulator sets in TMEM
  static constexpr int A_SL = OZ_BM * TK * 2;     // bytes of one A slice chunk
  static constexpr int B_SL = OZ_BN * TK * 2;
  static constexpr int STAGE = S * (A_SL + B_SL);
  static constexpr int NST = S == 5 ? 3 : 4;      // pipeline stages
  static constexpr int SMEM = NST * STAGE + 1024 + 1024;   // + barriers + alignment
  static constexpr uint32_t TMEM_COLS = 512;
  static constexpr int PRODUCTS = S == 4 ? 13 : S == 5 ? 19 : 36;
};
static_assert(OzCfg<4>::NSET * OzCfg<4>::NACC * OZ_BN <= 512 && OzCfg<OZ_FP64>::NACC * OZ_BN <= 512, "TMEM columns");

static int oz_tk(int S) { return S == OZ_FP64 ? OzCfg<OZ_FP64>::TK : OzCfg<4>::TK; }

// ---------------------------------------------------------------------------
// split: FP64 rows -> S BF16 slices (canonical layout) + per-row exponents
// ---------------------------------------------------------------------------
// Element (r, k) of the logical rows x K operand is P[r + k*ld] (trans = 0)
// or P[k + r*ld] (trans = 1). Tiles: [slice][kc][rb], 64 rows x TK K each
// (kc counts TK-wide chunks, 64 / TK per 64-wide K block); within a tile, (r, k)
// lives at (r/8)*8 TK + (k/8)*64 + (r%8)*8 + (k%8) elements.
__device__ __forceinline__ double oz_elem(const double *P, int64_t ld, int trans, int64_t r,
                                          int64_t k, int64_t rows, int64_t K) {
  if (r >= rows || k >= K) return 0.0;
  return trans ? P[k + r * ld] : P[r + k * ld];
}

// Row exponents and slices are computed from the FP64 bit patterns with integer and FP32
// instructions only (the FP64 pipe of this part is slow).

// Two neighbouring entries v0, v1 of a row with power of two e, as the S slices' packed
// BF16 pairs. |x| 2^BITS (rounded to nearest) of x = v 2^-e is written in balanced
// base-256 digits d0..d(S-1) (|d0| <= 256, of S = 8 <= 128; the others in [-128, 127])
// carrying the sign of v; slice t holds d_t 2^-8t (S = 8: d_t, as every level has its own
// accumulator). With 128 added to every byte but the first, the digits are the bytes
// minus 128, and a byte under the exponent of 2^23 is a float: two instructions a digit
// where a count of leading zeros and shifts took ten.
template <int S>
__device__ __forceinline__ void oz_pair(double v0, double v1, int e, uint32_t (&out)[S]) {
  constexpr int BITS = OzCfg<S>::BITS;
  // the top digit at byte S - 1
  constexpr unsigned long long BIAS = 0x8080808080808080ull >> (8 * (9 - S));
  uint32_t half[2][S];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(i ? v1 : v0);
    const int E = (int)((b >> 52) & 0x7FF);
    unsigned long long X = 0ull;
    if (E != 0 && E != 2047) {
      const unsigned long long mnt = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
      const int rsh = 1075 + e - E - BITS;  // >= 53 - BITS because |v| < 2^e
      if (BITS > 52 && rsh <= 0) X = mnt << -rsh;
      else if (rsh < 64) X = (mnt + (1ull << (rsh - 1))) >> rsh;
    }
    X += BIAS;
    const uint32_t lo = (uint32_t)X, hi = (uint32_t)(X >> 32);
    const uint32_t sgn = (uint32_t)(b >> 63) << 31;
#pragma unroll
    for (int t = 0; t < S; ++t) {
      const int byte = S - 1 - t;
      float f;
      if (t == 0) {
        // the top digit, up to 256 (S = 4: 32-bit numbers and one more)
        f = (float)(int)(X >> (8 * (S - 1)));
      } else {
        const uint32_t w = byte >= 4 ? hi : lo;
        f = __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650u | (byte & 3))) - 8388736.0f;
      }
      if (!OzCfg<S>::FP64 && t > 0) f *= __uint_as_float((uint32_t)(127 - 8 * t) << 23);
      half[i][t] = __float_as_uint(f) ^ sgn;
    }
  }
#pragma unroll
  for (int t = 0; t < S; ++t) out[t] = __byte_perm(half[0][t], half[1][t], 0x7632);
}

// The exponent of a row from its largest biased exponent field E: the row's largest
// element is 0.1m x 2^e. Zero and subnormal rows get 0; so do non-finite ones, except
// that the FP64-accurate product marks them and its outputs are NaN there, as the FP64
// pipe's would be (a factorisation must not pass over a NaN entry of its matrix).
constexpr int OZ_NONFINITE = 1 << 20;
template <int S>
__device__ __forceinline__ int oz_exponent(int E) {
  if (E == 2047) return OzCfg<S>::FP64 ? OZ_NONFINITE : 0;
  return E == 0 ? 0 : E - 1022;
}

// One-pass split: a block takes 32 rows, finds their maxima (coalesced for either
// layout: lanes over rows when columns are contiguous, over K when rows are),
// then writes every slice of those rows.
template <int S>
__global__ void __launch_bounds__(256) oz_split_kernel(const double *__restrict__ P, int64_t ld, int trans,
                                                       int64_t rows, int64_t K, int64_t nrb, int64_t nkb,
                                                       int *__restrict__ ex, uint16_t *__restrict__ sl,
                                                       int64_t sP, int64_t sE, int64_t sS) {
  P += blockIdx.y * sP;
  ex += blockIdx.y * sE;
  sl += blockIdx.y * sS;
  __shared__ unsigned long long part[8][32];
  __shared__ int exs[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t r0 = (int64_t)blockIdx.x * 32;
  if (!trans) {
    const int64_t r = r0 + lane;
    unsigned long long mx = 0ull;
    if (r < rows)
      for (int64_t k = warp; k < K; k += 8) {
        const unsigned long long b = (unsigned long long)__double_as_longlong(P[r + k * ld]) & 0x7FFFFFFFFFFFFFFFull;
        mx = b > mx ? b : mx;
      }
    part[warp][lane] = mx;
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int rl = warp * 4 + q;
      const int64_t r = r0 + rl;
      unsigned long long mx = 0ull;
      if (r < rows)
        for (int64_t k = lane; k < K; k += 32) {
          const unsigned long long b = (unsigned long long)__double_as_longlong(P[k + r * ld]) & 0x7FFFFFFFFFFFFFFFull;
          mx = b > mx ? b : mx;
        }
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = t > mx ? t : mx;
      }
      if (lane == 0) part[0][rl] = mx;
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    unsigned long long mx = part[0][lane];
    if (!trans)
#pragma unroll
      for (int w = 1; w < 8; ++w) mx = part[w][lane] > mx ? part[w][lane] : mx;
    const int e = oz_exponent<S>((int)(mx >> 52));
    exs[lane] = e;
    if (r0 + lane < nrb * OZ_TR) ex[r0 + lane] = e;
  }
  __syncthreads();
  // The block's 32 rows go through shared memory 64 K at a time, read along the
  // operand's contiguous direction (rows for trans = 0, K for trans = 1), so that
  // the slices are written with consecutive lanes on consecutive rows in either
  // layout (four full 128-byte lines per store).
  __shared__ double T[32][65];
  constexpr int TK = OzCfg<S>::TK;
  const int64_t nkc = (64 / TK) * nkb;
  const int rl = threadIdx.x & 31, gl = threadIdx.x >> 5;  // row, 8-wide K group of the chunk
  const int64_t r = r0 + rl;
  const int e = exs[rl];
  for (int64_t kb0 = 0; kb0 < nkb * 64; kb0 += 64) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int idx = threadIdx.x + 256 * q;
      const int ar = trans ? idx / 64 : idx % 32, ak = trans ? idx % 64 : idx / 32;
      T[ar][ak] = oz_elem(P, ld, trans, r0 + ar, kb0 + ak, rows, K);
    }
    __syncthreads();
    if (r >= nrb * OZ_TR) continue;
    const int64_t k0 = kb0 + 8 * gl;
    uint32_t packed[S][4];
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      uint32_t w[S];
      oz_pair<S>(T[rl][8 * gl + j], T[rl][8 * gl + j + 1], e, w);
#pragma unroll
      for (int t = 0; t < S; ++t) packed[t][j / 2] = w[t];
    }
    const int64_t rb = r / OZ_TR, rr = r % OZ_TR;
    const int64_t kc = k0 / TK, kk = k0 % TK;
    const int64_t within = (rr / 8) * (8 * TK) + (kk / 8) * 64 + (rr % 8) * 8;
#pragma unroll
    for (int t = 0; t < S; ++t) {
      const int64_t tile = ((int64_t)t * nkc + kc) * nrb + rb;
      *reinterpret_cast<uint4 *>(sl + tile * OzCfg<S>::TILE + within) =
          make_uint4(packed[t][0], packed[t][1], packed[t][2], packed[t][3]);
    }
  }
}

// Two-pass split for operands with too few 32-row groups to fill the GPU: pass 1
// takes the biased exponent field E of every element of 32 rows x 256 K and
// atomically maximises it per row (E is monotonic in |x|, so the row's largest E
// is that of its largest element; 0 and 2047 mark zero / subnormal and
// non-finite rows as in the one-pass kernel); pass 2 writes the slices of one
// 64-wide K block of 32 rows per CTA.
constexpr int OZ_EK = 256;  // K per pass-1 CTA

__global__ void __launch_bounds__(256) oz_rowexp_kernel(const double *__restrict__ P, int64_t ld, int trans,
                                                        int64_t rows, int64_t K, int *__restrict__ Emax,
                                                        int64_t sP, int64_t sM) {
  P += blockIdx.z * sP;
  Emax += blockIdx.z * sM;
  __shared__ int part[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t r0 = (int64_t)blockIdx.x * 32;
  const int64_t k0 = (int64_t)blockIdx.y * OZ_EK;
  const int64_t k1 = k0 + OZ_EK < K ? k0 + OZ_EK : K;
  if (!trans) {
    const int64_t r = r0 + lane;
    int mx = 0;
    if (r < rows)
      for (int64_t k = k0 + warp; k < k1; k += 8) {
        const int E = (int)(((unsigned long long)__double_as_longlong(P[r + k * ld]) >> 52) & 0x7FF);
        mx = E > mx ? E : mx;
      }
    part[warp][lane] = mx;
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int rl = warp * 4 + q;
      const int64_t r = r0 + rl;
      int mx = 0;
      if (r < rows)
        for (int64_t k = k0 + lane; k < k1; k += 32) {
          const int E = (int)(((unsigned long long)__double_as_longlong(P[k + r * ld]) >> 52) & 0x7FF);
          mx = E > mx ? E : mx;
        }
      for (int o = 16; o > 0; o >>= 1) {
        const int t = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = t > mx ? t : mx;
      }
      if (lane == 0) part[0][rl] = mx;
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int mx = part[0][lane];
    if (!trans)
#pragma unroll
      for (int w = 1; w < 8; ++w) mx = part[w][lane] > mx ? part[w][lane] : mx;
    if (r0 + lane < rows && mx > 0) atomicMax(Emax + r0 + lane, mx);
  }
}

template <int S>
__global__ void __launch_bounds__(256) oz_slice_kernel(const double *__restrict__ P, int64_t ld, int trans,
                                                       int64_t rows, int64_t K, int64_t nrb, int64_t nkb,
                                                       const int *__restrict__ Emax, int *__restrict__ ex,
                                                       uint16_t *__restrict__ sl, int64_t sP, int64_t sE,
                                                       int64_t sS, int64_t sM) {
  P += blockIdx.z * sP;
  ex += blockIdx.z * sE;
  sl += blockIdx.z * sS;
  Emax += blockIdx.z * sM;
  __shared__ double T[32][65];
  const int64_t r0 = (int64_t)blockIdx.x * 32;
  const int rl = threadIdx.x & 31, gl = threadIdx.x >> 5;
  const int64_t r = r0 + rl;
  const int e = oz_exponent<S>(r < rows ? Emax[r] : 0);
  if (blockIdx.y == 0 && gl == 0 && r < nrb * OZ_TR) ex[r] = e;
  const int64_t kb0 = (int64_t)blockIdx.y * 64;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int idx = threadIdx.x + 256 * q;
    const int ar = trans ? idx / 64 : idx % 32, ak = trans ? idx % 64 : idx / 32;
    T[ar][ak] = oz_elem(P, ld, trans, r0 + ar, kb0 + ak, rows, K);
  }
  __syncthreads();
  if (r >= nrb * OZ_TR) return;
  const int64_t k0 = kb0 + 8 * gl;
  uint32_t packed[S][4];
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    uint32_t w[S];
    oz_pair<S>(T[rl][8 * gl + j], T[rl][8 * gl + j + 1], e, w);
#pragma unroll
    for (int t = 0; t < S; ++t) packed[t][j / 2] = w[t];
  }
  constexpr int TK = OzCfg<S>::TK;
  const int64_t nkc = (64 / TK) * nkb;
  const int64_t rb = r / OZ_TR, rr = r % OZ_TR;
  const int64_t kc = k0 / TK, kk = k0 % TK;
  const int64_t within = (rr / 8) * (8 * TK) + (kk / 8) * 64 + (rr % 8) * 8;
#pragma unroll
  for (int t = 0; t < S; ++t) {
    const int64_t tile = ((int64_t)t * nkc + kc) * nrb + rb;
    *reinterpret_cast<uint4 *>(sl + tile * OzCfg<S>::TILE + within) =
        make_uint4(packed[t][0], packed[t][1], packed[t][2], packed[t][3]);
  }
}

// 64-row tiles of a split operand: one more than the rows need, rounded up to
// an even count, so that a 128-row A tile starting at any 64-row offset inside
// the operand stays inside the buffer.
int64_t oz_nrb(int64_t rows) {
  const int64_t t = (rows + OZ_TR - 1) / OZ_TR + 1;
  return (t + 1) / 2 * 2;
}

void oz_split_batched(cudaStream_t s, const double *P, int64_t ld, int64_t sP, int trans, int64_t rows,
                      int64_t K, OzSplit *out, int64_t batch) {
  const int64_t nrb = oz_nrb(rows);
  const int64_t nkb = (K + 63) / 64;
  out->rows = rows;
  out->K = K;
  out->nrb = nrb;
  out->nkb = nkb;
  const int64_t rows_pad = nrb * OZ_TR;
  const int64_t sE = out->bstride_ex, sS = out->bstride_sl;
  KTScope kts(GPGP_KPROF_OZ_SPLIT, s, 0.0);
  const int64_t groups = rows_pad / 32;
  if (groups * batch < 2 * (int64_t)device_sms() && nkb >= 2 && batch <= 65535) {
    // too few row groups for one CTA each to fill the GPU: two passes over a 2-D grid
    int *Emax = nullptr;
    GPGP_CUDA(cudaMallocAsync((void **)&Emax, (size_t)rows_pad * batch * sizeof(int), s));
    GPGP_CUDA(cudaMemsetAsync(Emax, 0, (size_t)rows_pad * batch * sizeof(int), s));
    dim3 g1((unsigned)groups, (unsigned)((K + OZ_EK - 1) / OZ_EK), (unsigned)batch);
    oz_rowexp_kernel<<<g1, 256, 0, s>>>(P, ld, trans, rows, K, Emax, sP, rows_pad);
    GPGP_CHECK_LAUNCH();
    dim3 g2((unsigned)groups, (unsigned)nkb, (unsigned)batch);
    auto kern = out->S == OZ_FP64 ? oz_slice_kernel<OZ_FP64> : out->S == 5 ? oz_slice_kernel<5> : oz_slice_kernel<4>;
    kern<<<g2, 256, 0, s>>>(P, ld, trans, rows, K, nrb, nkb, Emax, out->ex, out->sl, sP, sE, sS, rows_pad);
    GPGP_CHECK_LAUNCH();
    GPGP_CUDA(cudaFreeAsync(Emax, s));
    return;
  }
  dim3 g((unsigned)groups, (unsigned)batch);
  auto kern = out->S == OZ_FP64 ? oz_split_kernel<OZ_FP64> : out->S == 5 ? oz_split_kernel<5> : oz_split_kernel<4>;
  kern<<<g, 256, 0, s>>>(P, ld, trans, rows, K, nrb, nkb, out->ex, out->sl, sP, sE, sS);
  GPGP_CHECK_LAUNCH();
}

void oz_split(cudaStream_t s, const double *P, int64_t ld, int trans, int64_t rows, int64_t K,
              OzSplit *out) {
  oz_split_batched(s, P, ld, 0, trans, rows, K, out, 1);
}

size_t oz_split_bytes(int64_t rows, int64_t K, int S) {
  const int64_t nrb = oz_nrb(rows);
  const int64_t nkb = (K + 63) / 64;
  return (size_t)nrb * OZ_TR * sizeof(int) + 256 + (size_t)S * nkb * nrb * OZ_TR * 64 * 2;
}

void oz_split_bind(void *mem, int64_t rows, int64_t K, OzSplit *out, int S) {
  const int64_t nrb = oz_nrb(rows);
  (void)K;
  out->S = S;
  char *p = (char *)mem;
  out->ex = (int *)p;
  size_t exb = ((size_t)nrb * OZ_TR * sizeof(int) + 255) / 256 * 256;
  out->sl = (uint16_t *)(p + exb);
}

// ---------------------------------------------------------------------------
// PTX helpers (tcgen05, mbarrier, bulk copy)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version for tcgen05
  // base offset 0, lbo mode 0, layout type 0 (no swizzle)
  return d;
}

__device__ __forceinline__ void umma_bf16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum));
}

// one lane of a converged warp (the predicate stays uniform for the compiler)
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                 "=r"(r[7])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// double-float accumulation of v into (hi, lo) with an error-free TwoSum
__device__ __forceinline__ void df_add(float &hi, float &lo, float v) {
  const float s = __fadd_rn(hi, v);
  const float bp = __fsub_rn(s, hi);
  const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(v, bp));
  hi = s;
  lo = __fadd_rn(lo, e);
}

// The slice products of KS K steps (16 K each, 256 bytes apart in an operand) into the
// accumulators at column d0: ad, bd describe slice 0 of the operands, a_sl and b_sl are the
// bytes from slice to slice. acc 0: overwrite the accumulators.
template <int S, int KS>
__device__ __forceinline__ void oz_issue(uint64_t ad0, uint64_t bd0, int a_sl, int b_sl, uint32_t d0, uint32_t acc) {
  using Cfg = OzCfg<S>;
  constexpr int NACC = Cfg::NACC;
  // D F32, A/B BF16, K-major both, M = 128; N is set per instruction
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(OZ_BM >> 4) << 24);
#pragma unroll
  for (int kk = 0; kk < KS; ++kk) {
#pragma unroll
    for (int ti = 0; ti < S; ++ti) {
      const uint64_t ad = ad0 + (uint64_t)((ti * a_sl + kk * 256) >> 4);
      // The B slices lie back to back with one 8-row stride, so slices
      // 0..NACC-1-ti read as one operand of 64 (NACC - ti) rows: an MMA puts
      // A_ti B_u^T (level ti + u) into accumulators ti.., which are adjacent
      // column blocks (N of at most 256: two MMAs where there are more). The
      // first slice's, first in a group, overwrite all of them.
#pragma unroll
      for (int o = 0; o < OZ_BN * (NACC - ti); o += 256) {
        const int nn = OZ_BN * (NACC - ti) - o < 256 ? OZ_BN * (NACC - ti) - o : 256;
        umma_bf16(d0 + (uint32_t)(ti * OZ_BN + o), ad, bd0 + (uint64_t)((o / OZ_BN * b_sl + kk * 256) >> 4),
                  idesc | ((uint32_t)(nn >> 3) << 17), (kk == 0 && ti == 0) ? acc : 1u);
      }
      // S = 4, 5: the remaining products of levels > 3 go one by one into the
      // last accumulator
      if (!Cfg::FP64)
#pragma unroll
        for (int ui = ti < NACC ? NACC - ti : 0; ui < S; ++ui) {
          if (ti + ui > S) continue;
          umma_bf16(d0 + (uint32_t)((NACC - 1) * OZ_BN), ad, bd0 + (uint64_t)((ui * b_sl + kk * 256) >> 4),
                    idesc | ((uint32_t)(OZ_BN >> 3) << 17), 1u);
        }
    }
  }
}

// The sum over one exactly accumulated group of NC columns: added to hi, lo (double-float,
// level-0 units; of S = 8 fixed point, hi in units of level 3, lo, 0 <= lo < 2^24, of level 6)
template <int S>
struct OzSum {
  using Hi = typename std::conditional<OzCfg<S>::FP64, long long, float>::type;
  using Lo = typename std::conditional<OzCfg<S>::FP64, int, float>::type;
};
template <int S, int NC>
__device__ __forceinline__ void oz_drain(uint32_t ta, typename OzSum<S>::Hi *hi, typename OzSum<S>::Lo *lo) {
  constexpr int NACC = OzCfg<S>::NACC;
  if constexpr (OzCfg<S>::FP64) {
#pragma unroll
    for (int cb = 0; cb < NC; cb += 4) {
      // an accumulator of level l holds an integer of at most (l + 1) 2^22: levels
      // 0..3 exactly, the deeper ones to a unit of theirs
      uint32_t r[4][4];
#pragma unroll
      for (int l = 0; l < 4; ++l) tmem_ld4(ta + (uint32_t)(l * OZ_BN + cb), r[l]);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        long long x = hi[cb + j] + __float2int_rn(__uint_as_float(r[3][j]));
        x += (long long)__float2int_rn(__uint_as_float(r[2][j])) * 256;
        x += (long long)__float2int_rn(__uint_as_float(r[1][j])) * 65536;
        x += (long long)__float2int_rn(__uint_as_float(r[0][j])) * 16777216;
        hi[cb + j] = x;
      }
#pragma unroll
      for (int l = 4; l < NACC; ++l) tmem_ld4(ta + (uint32_t)(l * OZ_BN + cb), r[l - 4]);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int i4 = __float2int_rn(__uint_as_float(r[0][j])), i5 = __float2int_rn(__uint_as_float(r[1][j]));
        int y = lo[cb + j] + ((i4 & 255) << 16) + ((i5 & 65535) << 8) + __float2int_rn(__uint_as_float(r[2][j]));
        y += __float2int_rn(__uint_as_float(r[3][j]) * 0x1p-8f);
        hi[cb + j] += (i4 >> 8) + (i5 >> 16) + (y >> 24);
        lo[cb + j] = y & 0xFFFFFF;
      }
    }
  } else {
#pragma unroll
    for (int cb = 0; cb < NC; cb += 8)
#pragma unroll
      for (int ac = 0; ac < NACC; ac += 2) {  // two accumulators at a time: 16 registers
        uint32_t r[2][8];
        tmem_ld8(ta + (uint32_t)(ac * OZ_BN + cb), r[0]);
        tmem_ld8(ta + (uint32_t)((ac + 1) * OZ_BN + cb), r[1]);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          df_add(hi[cb + j], lo[cb + j], __uint_as_float(r[0][j]));
          df_add(hi[cb + j], lo[cb + j], __uint_as_float(r[1][j]));
        }
      }
  }
}

// ---------------------------------------------------------------------------
// the GEMM: C = alpha A B^T + beta C over the given K range (alpha 1 or -1, beta 0 or 1)
// ---------------------------------------------------------------------------
struct OzGemmArgs {
  const uint16_t *a_sl;
  const int *a_ex;
  int a_nrb, a_nkc, a_rb0;  // slice-tile geometry (TK-wide K chunks); first 64-row tile
  const uint16_t *b_sl;
  const int *b_ex;
  int b_nrb, b_nkc, b_rb0;
  int M, N;
  int kc0, kc1;  // TK-wide K chunks [kc0, kc1) of both operands
  int kmode;     // 0 all; 1 start at max(row,col); 2 start at col; 3 end after row
  double alpha, beta;
  double *C;
  int64_t ldc;
  int lower_only;
  int *err;
  const int *status;  // optional: skip a problem whose factorisation already failed
  int64_t a_bs_sl, a_bs_ex, b_bs_sl, b_bs_ex, c_bs;  // per-problem strides
  int64_t status_bs;
  int gx, gy;       // tiles per problem along M and N
  int order;        // OzOrder
  int per, ntiles;  // tiles per problem and in the launch
  uint32_t polls;   // TEST only: bound of every wait ..
  int chunks;       // .. and K chunks after which a CTA's producer falls silent
};

// The order in which a problem's tiles are dealt to the CTAs, longest K range first
// where the ranges differ (kmode 1 and 3), so that the last round of the persistent
// grid holds the short ones:
//  OZ_COLS        columns of tiles, left to right
//  OZ_ROWS_UP     rows of tiles, last row first (kmode 3: the range ends after the row)
//  OZ_LOWER       the tiles that meet the lower triangle only, row by row (kmode 1: the
//                 range starts at the row). Tiles above the diagonal are not dealt: in a
//                 square product they are half of the list, and skipping them in turn
//                 left the CTAs with unequal counts.
enum OzOrder { OZ_COLS = 0, OZ_ROWS_UP = 1, OZ_LOWER = 2 };

struct OzTile {
  int z, row0, col0, c0, nch;
};

// Tiles of the lower triangle: row bx has min(2 bx + 2, gy) of them.
__host__ __device__ __forceinline__ int oz_lower_tiles(int gx, int gy) {
  const int q = gy / 2;  // rows below q have 2 bx + 2 <= gy tiles
  return gx <= q ? gx * (gx + 1) : q * (q + 1) + (gx - q) * gy;
}

// Position r of a problem's tile list -> tile coordinates (bx, by)
__host__ __device__ __forceinline__ void oz_tile_xy(int order, int gx, int gy, int r, int *bx, int *by) {
  if (order == OZ_LOWER) {
    const int q = gy / 2, cq = q * (q + 1);
    if (r < cq) {
      int b = (int)((sqrtf(4.0f * (float)r + 1.0f) - 1.0f) * 0.5f);
      while (b * (b + 1) > r) --b;
      while ((b + 1) * (b + 2) <= r) ++b;
      *bx = b;
      *by = r - b * (b + 1);
    } else {
      const int o = (r - cq) / gy;
      *bx = q + o;
      *by = (r - cq) - o * gy;
    }
  } else if (order == OZ_ROWS_UP) {
    const int o = r / gy;
    *bx = gx - 1 - o;
    *by = r - o * gy;
  } else {
    const int o = r / gx;
    *by = o;
    *bx = r - o * gx;
  }
}

// The K chunks [k0, k1) of the tile at (row0, col0)
__host__ __device__ __forceinline__ void oz_krange(int tk, int kmode, int grow0, int gcol0, int kc0, int kc1,
                                                   int *k0, int *k1) {
  if (kmode == 1) kc0 = max(kc0, max(grow0, gcol0) / tk);
  if (kmode == 2) kc0 = max(kc0, gcol0 / tk);
  if (kmode == 3) kc1 = min(kc1, (grow0 + OZ_BM + tk - 1) / tk);
  *k0 = kc0;
  *k1 = kc1;
}

// The work of position L (identical in every role): false when its problem has failed.
// All 32-bit: 64-bit divisions here cost every epilogue warp more than the tile's
// TMEM reads.
template <int S>
__device__ __forceinline__ bool oz_tile_at(const OzGemmArgs &g, int L, OzTile &t) {
  t.z = g.per == g.ntiles ? 0 : L / g.per;
  int bx, by;
  oz_tile_xy(g.order, g.gx, g.gy, L - t.z * g.per, &bx, &by);
  t.row0 = bx * OZ_BM;
  t.col0 = by * OZ_BN;
  if (g.status && *(volatile const int *)(g.status + t.z * g.status_bs) != 0) return false;
  int k0, k1;
  oz_krange(OzCfg<S>::TK, g.kmode, g.a_rb0 * OZ_TR + t.row0, g.b_rb0 * OZ_TR + t.col0, g.kc0, g.kc1, &k0, &k1);
  t.c0 = k0;
  t.nch = k1 > k0 ? k1 - k0 : 0;
  return true;
}

// Bounded wait that also gives up when another role has aborted.
__device__ __forceinline__ bool oz_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, uint32_t polls) {
  for (uint32_t it = 0; it < polls; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255u) == 255u && *abort_flag) return false;
  }
  return false;
}

// TEST: with the bounds of gpgp_wait_bound (as arguments of the one kernel they cost 7%)
template <int S, bool TEST>
// 576 threads: the register cap keeps the block inside one SM's register file
__global__ void __maxnreg__(96) oz_gemm_kernel(const OzGemmArgs g) {
  using Cfg = OzCfg<S>;
  constexpr int NST = Cfg::NST;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *bars = (uint64_t *)(smem + NST * Cfg::STAGE);
  __shared__ uint32_t tmem_base_sh;
  __shared__ int abort_sh;
  volatile int *abort_flag = &abort_sh;
  const uint32_t polls = TEST ? g.polls : WAIT_POLLS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // barriers: full[NST] (operands landed), empty[NST] (MMAs that read a stage done),
  // tfull[NSET] (an accumulator set is ready), tempty[NSET] (the epilogue drained it), drain
  constexpr int NSET = Cfg::NSET, NACC = Cfg::NACC, GROUP = Cfg::GROUP;
  constexpr int FULL = 0, EMPTY = NST, TFULL = 2 * NST, TEMPTY = 2 * NST + 2, DRAIN = 2 * NST + 4;
  auto bar = [&](int i) { return smem_u32(&bars[i]); };
  if (threadIdx.x == 0) {
    for (int i = 0; i < NST; ++i) {
      mbar_init(bar(FULL + i), 1);
      mbar_init(bar(EMPTY + i), 1);
    }
    for (int i = 0; i < NSET; ++i) {
      mbar_init(bar(TFULL + i), 1);
      mbar_init(bar(TEMPTY + i), OZ_EPI_WARPS);
    }
    mbar_init(bar(DRAIN), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_sh = 0;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_base_sh)),
                 "r"(Cfg::TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_sh;
  const int ntiles = g.ntiles;
  int last_full_parity[NST];
#pragma unroll
  for (int i = 0; i < NST; ++i) last_full_parity[i] = -1;
  bool mma_issued = false;

  if (warp == 0) {
    // ---- producer: K chunks of this CTA's tiles into the stage ring ----
    if (lane == 0) {
      int st = 0, left = TEST ? g.chunks : 0;
      uint32_t ph = 0;
      for (int L = blockIdx.x; L < ntiles; L += gridDim.x) {
        OzTile t;
        if (!oz_tile_at<S>(g, L, t) || t.nch == 0) continue;
        const uint16_t *ap = g.a_sl + t.z * g.a_bs_sl +
                             ((int64_t)t.c0 * g.a_nrb + g.a_rb0 + t.row0 / OZ_TR) * Cfg::TILE;
        const uint16_t *bp = g.b_sl + t.z * g.b_bs_sl +
                             ((int64_t)t.c0 * g.b_nrb + g.b_rb0 + t.col0 / OZ_TR) * Cfg::TILE;
        const int64_t asl = (int64_t)g.a_nkc * g.a_nrb * Cfg::TILE, bsl = (int64_t)g.b_nkc * g.b_nrb * Cfg::TILE;
        for (int c = 0; c < t.nch; ++c) {
          if (TEST && --left < 0) goto producer_done;
          if (!oz_wait(bar(EMPTY + st), ph ^ 1u, abort_flag, polls)) {
            if (!*abort_flag) atomicExch(g.err, 1);
            abort_sh = 1;
            goto producer_done;
          }
          const uint32_t base = smem_u32(smem + st * Cfg::STAGE);
          mbar_expect_tx(bar(FULL + st), Cfg::STAGE);
#pragma unroll
          for (int s = 0; s < S; ++s) {
            bulk_g2s(base + s * Cfg::A_SL, ap + s * asl, Cfg::A_SL, bar(FULL + st));
            bulk_g2s(base + S * Cfg::A_SL + s * Cfg::B_SL, bp + s * bsl, Cfg::B_SL, bar(FULL + st));
          }
          ap += (int64_t)g.a_nrb * Cfg::TILE;
          bp += (int64_t)g.b_nrb * Cfg::TILE;
          last_full_parity[st] = (int)ph;
          if (++st == NST) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
    producer_done:;
    }
  } else if (warp == 1) {
    // ---- MMA issuer: the whole warp walks the chunks, one elected lane issues ----
    // (Warp-uniform control flow keeps descriptors and barrier addresses in uniform
    // registers; with everything inside one lane's branch an instruction took 84 to
    // 100 cycles to issue, longer than the tensor pipe takes to run it.)
    // no-swizzle K-major: core matrices of 8 rows x 16 bytes; LBO steps K (128 B),
    // SBO steps 8 rows (8 x TK x 2 B). Slices, K steps and stages are offsets
    // in 16-byte units (shared addresses stay below 2^18, so the 14-bit address field
    // never carries).
    const uint64_t adesc = umma_desc(smem_u32(smem), 128u, 16u * Cfg::TK);
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    // Whether a wait gives up depends on a lane's own polls and on when it sees the abort
    // flag, but the lanes must stay together (the barriers need all 32): a lane's outcome
    // only keeps the leader from issuing, and the warp leaves the loop by a vote. The vote
    // stands after the issue, off the way from the operands to their products: there the
    // loop is also 2 to 5% faster than with a branch at each wait (4096^2 x 4096, S = 4 /
    // 8: 1.24 / 2.96 ms; a branch 1.26 / 3.12, a vote at each wait 1.31 / 3.18, lane 0's
    // outcome shuffled to the others 1.38 / 3.35).
    const bool leader = elect_one();
    bool ok = true;
    int st = 0, b = 0;
    uint32_t ph = 0, tph = 0;  // tph bit b: parity of accumulator set b
    for (int L = blockIdx.x; L < ntiles; L += gridDim.x) {
      OzTile t;
      if (!oz_tile_at<S>(g, L, t) || t.nch == 0) continue;
      uint32_t acc = 0;  // 0 while the group's accumulators are still to be overwritten
      for (int c = 0; c < t.nch; ++c) {
        const bool gend = ((c + 1) & (GROUP - 1)) == 0 || c == t.nch - 1;
        if ((c & (GROUP - 1)) == 0) {
          ok &= oz_wait(bar(TEMPTY + b), ((tph >> b) & 1u) ^ 1u, abort_flag, polls);
          acc = 0;
        }
        ok &= oz_wait(bar(FULL + st), ph, abort_flag, polls);
        tc_fence_after();
        const uint64_t ad0 = adesc + (uint64_t)((uint32_t)st * (uint32_t)(Cfg::STAGE >> 4));
        const uint64_t bd0 = ad0 + (uint64_t)((S * Cfg::A_SL) >> 4);
        const uint32_t d0 = tm + (uint32_t)(b * NACC * OZ_BN);
        if (leader && ok) {
          oz_issue<S, Cfg::TK / 16>(ad0, bd0, Cfg::A_SL, Cfg::B_SL, d0, acc);
          umma_commit(bar(EMPTY + st));
          if (gend) umma_commit(bar(TFULL + b));
        }
        acc = 1u;
        mma_issued = true;
        if (!__all_sync(0xffffffffu, ok)) {
          if (!*abort_flag) atomicExch(g.err, 2);
          abort_sh = 1;
          goto mma_done;
        }
        if (++st == NST) {
          st = 0;
          ph ^= 1u;
        }
        if (gend) {
          tph ^= 1u << b;
          b ^= NSET - 1;
        }
      }
    }
  mma_done:;
  } else {
    // ---- epilogue: warps 2..17 drain TMEM lanes 32 (warp % 4).., 16 columns each ----
    const int quarter = warp & 3, part = (warp - 2) >> 2;
    int b = 0;
    uint32_t tph[2] = {0u, 0u};
    // alpha is 1 or -1 and beta 0 or 1 (checked on the host): the sum's sign is flipped on
    // its bits and C takes one FP64 addition (that pipe is the scarce unit, and even a
    // multiplication that is predicated off holds it)
    const bool beta0 = g.beta == 0.0;
    const uint32_t negmask = g.alpha < 0.0 ? 0x80000000u : 0u;
    for (int L = blockIdx.x; L < ntiles; L += gridDim.x) {
      OzTile t;
      if (!oz_tile_at<S>(g, L, t)) continue;
      const int my_row = t.row0 + quarter * 32 + lane;
      const int col_base = t.col0 + part * OZ_EPI_COLS;
      // this thread's columns: those inside C and, of a lower-only product, left of
      // the diagonal (0 outside the rows)
      int ncol = my_row < g.M ? min(OZ_EPI_COLS, g.N - col_base) : 0;
      if (g.lower_only) ncol = min(ncol, my_row - col_base + 1);
      double *cp = g.C + t.z * g.c_bs + my_row + (int64_t)col_base * g.ldc;
      // The first half of this thread's C values is loaded before the accumulators are
      // ready, so that the loads overlap the MMAs; the second half is only brought to
      // L2 (16 values at a time would not leave the accumulation its registers).
      constexpr int HALF = Cfg::FP64 ? 4 : OZ_EPI_COLS / 2;
      double cv[HALF];
      auto load_c = [&](int j0) {
        const double *cr = cp + j0 * g.ldc;
#pragma unroll
        for (int j = 0; j < HALF; ++j) {
          cv[j] = j0 + j < ncol ? *cr : 0.0;
          cr += g.ldc;
        }
      };
      if (!beta0) {
        load_c(0);
        const double *cr = cp + HALF * g.ldc;
#pragma unroll
        for (int j = 0; j < OZ_EPI_COLS - HALF; ++j) {
          if (HALF + j < ncol) asm volatile("prefetch.global.L2 [%0];" ::"l"(cr));
          cr += g.ldc;
        }
      }
      if (t.nch == 0) {  // nothing accumulated: C = 0 or C
        if (beta0)
          for (int j = 0; j < ncol; ++j) cp[j * g.ldc] = 0.0;
        continue;
      }
      // exponents: the row's, and the 16 columns' one to a lane
      const int ea = my_row < g.M ? g.a_ex[t.z * g.a_bs_ex + g.a_rb0 * OZ_TR + my_row] : 0;
      const int eb = lane < OZ_EPI_COLS && col_base + lane < g.N
                         ? g.b_ex[t.z * g.b_bs_ex + g.b_rb0 * OZ_TR + col_base + lane] : 0;
      const int ngr = (t.nch + GROUP - 1) / GROUP;
      // the tile's sum over its K groups
      typename OzSum<S>::Hi hi[OZ_EPI_COLS];
      typename OzSum<S>::Lo lo[OZ_EPI_COLS];
#pragma unroll
      for (int j = 0; j < OZ_EPI_COLS; ++j) {
        hi[j] = 0;
        lo[j] = 0;
      }
      for (int gi = 0; gi < ngr; ++gi) {
        int ok = 1;
        if (lane == 0) ok = oz_wait(bar(TFULL + b), tph[b], abort_flag, polls) ? 1 : 0;
        ok = __shfl_sync(0xffffffffu, ok, 0);
        if (!ok) {
          if (lane == 0) {
            if (!*abort_flag) atomicExch(g.err, 3);
            abort_sh = 1;
          }
          goto epi_done;
        }
        tc_fence_after();
        const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(b * NACC * OZ_BN + part * OZ_EPI_COLS);
        oz_drain<S, OZ_EPI_COLS>(ta, hi, lo);
        // every load of this set has completed: hand it back to the MMA warp
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(TEMPTY + b));
        tph[b] ^= 1u;
        b ^= NSET - 1;
      }
      // C = alpha 2^(e_i + f_j) (sum) + beta C, EC columns at a time without a branch
      // between them, so that their conversions overlap; a value outside the fast range
      // (subnormal, overflow) sends them through the general conversion
      constexpr int EC = 4;
      double *cw = cp;
#pragma unroll
      for (int j0 = 0; j0 < OZ_EPI_COLS; j0 += EC) {
        if (j0 > 0 && j0 % HALF == 0 && !beta0) load_c(j0);
        double v[EC];
        bool slow = false;
#pragma unroll
        for (int j = 0; j < EC; ++j) {
          const int sh = ea + __shfl_sync(0xffffffffu, eb, j0 + j);
          if constexpr (Cfg::FP64) {
            v[j] = fixed_to_double(hi[j0 + j], lo[j0 + j], sh, negmask, slow);
          } else {
            // the sign of alpha goes onto the FP32 pair
            hi[j0 + j] = __uint_as_float(__float_as_uint(hi[j0 + j]) ^ negmask);
            lo[j0 + j] = __uint_as_float(__float_as_uint(lo[j0 + j]) ^ negmask);
            v[j] = df2d_try(hi[j0 + j], lo[j0 + j], sh - 16, slow);
          }
        }
        if (__any_sync(0xffffffffu, slow)) {
#pragma unroll
          for (int j = 0; j < EC; ++j) {
            const int sh = ea + __shfl_sync(0xffffffffu, eb, j0 + j);
            if constexpr (Cfg::FP64) v[j] = fixed_to_double_slow(hi[j0 + j], lo[j0 + j], sh, negmask);
            else v[j] = df2d_scaled(hi[j0 + j], lo[j0 + j], sh - 16);
          }
        }
#pragma unroll
        for (int j = 0; j < EC; ++j) {
          if (!beta0) v[j] = cv[(j0 + j) % HALF] + v[j];
          if (j0 + j < ncol) *cw = v[j];
          cw += g.ldc;
        }
      }
    }
  epi_done:;
  }

  __syncthreads();
  if (abort_sh) {
    // a wait ran out: let what was issued land (bounded) before the shared memory
    // and TMEM are released
    if (warp == 1 && mma_issued && elect_one()) {  // (the same lane as issued)
      umma_commit(bar(DRAIN));
      mbar_wait_bounded(bar(DRAIN), 0);
    }
    if (warp == 0 && lane == 0)
      for (int i = 0; i < NST; ++i)
        if (last_full_parity[i] >= 0) mbar_wait_bounded(bar(FULL + i), (uint32_t)last_full_parity[i]);
  }
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::TMEM_COLS));
  }
}

thread_local int tl_oz_grid_cap = 0;

static const WaitBounds kWaitDefault = {{WAIT_POLLS, WAIT_POLLS, WAIT_POLLS, FLOW_POLLS}, INT_MAX};
thread_local WaitBounds tl_wait = kWaitDefault;

template <int S>
static void launch_oz_gemm(cudaStream_t s, int grid, const OzGemmArgs &g) {
  static PerDevice attr;
  per_device(attr, [] {
    GPGP_CUDA(cudaFuncSetAttribute(oz_gemm_kernel<S, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   OzCfg<S>::SMEM));
    GPGP_CUDA(cudaFuncSetAttribute(oz_gemm_kernel<S, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   OzCfg<S>::SMEM));
    return 1;
  });
  if (g.polls == WAIT_POLLS && g.chunks == INT_MAX)
    oz_gemm_kernel<S, false><<<(unsigned)grid, OZ_THREADS, OzCfg<S>::SMEM, s>>>(g);
  else
    oz_gemm_kernel<S, true><<<(unsigned)grid, OZ_THREADS, OzCfg<S>::SMEM, s>>>(g);
}

static int oz_sm_count() { return device_sms(); }

void oz_gemm_batched(cudaStream_t s, const OzSplit &A, int64_t a_row0, const OzSplit &B, int64_t b_row0,
                     int64_t M, int64_t N, int64_t kc0, int64_t kc1, int kmode, double alpha,
                     double beta, double *C, int64_t ldc, int64_t sC, bool lower_only, int *err,
                     const int *status, int64_t status_bs, int64_t batch) {
  if (M <= 0 || N <= 0 || batch <= 0) return;
  if ((alpha != 1.0 && alpha != -1.0) || (beta != 0.0 && beta != 1.0))
    throw CudaError{cudaErrorInvalidValue, "oz_gemm: alpha must be 1 or -1, beta 0 or 1", __LINE__};
  if (A.S != B.S) throw CudaError{cudaErrorInvalidValue, "oz_gemm: operands split to different slice counts", __LINE__};
  OzGemmArgs g;
  g.a_sl = A.sl;
  g.a_ex = A.ex;
  g.a_nrb = (int)A.nrb;
  const int tk = oz_tk(A.S), per64 = 64 / tk;
  g.a_nkc = (int)(per64 * A.nkb);
  g.a_rb0 = (int)(a_row0 / OZ_TR);
  g.b_sl = B.sl;
  g.b_ex = B.ex;
  g.b_nrb = (int)B.nrb;
  g.b_nkc = (int)(per64 * B.nkb);
  g.b_rb0 = (int)(b_row0 / OZ_TR);
  g.M = (int)M;
  g.N = (int)N;
  // callers count K in 64-wide blocks; the kernel in TK-wide chunks
  g.kc0 = (int)(per64 * kc0);
  g.kc1 = (int)std::min<int64_t>(per64 * kc1, std::min(g.a_nkc, g.b_nkc));
  g.kmode = kmode;
  g.alpha = alpha;
  g.beta = beta;
  g.C = C;
  g.ldc = ldc;
  g.lower_only = lower_only ? 1 : 0;
  g.err = err;
  g.status = status;
  g.a_bs_sl = A.bstride_sl;
  g.a_bs_ex = A.bstride_ex;
  g.b_bs_sl = B.bstride_sl;
  g.b_bs_ex = B.bstride_ex;
  g.c_bs = sC;
  g.status_bs = status_bs;
  const int64_t gx = (M + OZ_BM - 1) / OZ_BM, gy = (N + OZ_BN - 1) / OZ_BN;
  if (gx * gy * batch >= (int64_t)1 << 31 || M >= (int64_t)1 << 30 || N >= (int64_t)1 << 30)
    throw CudaError{cudaErrorInvalidValue, "oz_gemm: too many tiles", __LINE__};
  g.gx = (int)gx;
  g.gy = (int)gy;
  g.order = lower_only ? OZ_LOWER : kmode == 3 ? OZ_ROWS_UP : OZ_COLS;
  g.per = lower_only ? oz_lower_tiles(g.gx, g.gy) : g.gx * g.gy;
  g.ntiles = (int)(g.per * batch);
  g.polls = tl_wait.polls[GPGP_WAIT_GEMM];
  g.chunks = tl_wait.gemm_chunks;
  const int cap = tl_oz_grid_cap > 0 ? std::min(tl_oz_grid_cap, oz_sm_count()) : oz_sm_count();
  const int grid = std::min(g.ntiles, cap);
  double fl = 0.0;
  if (tl_kt) {
    // executed MMA arithmetic of the tiles the launch runs (failed problems are not
    // known on the host)
    const int prods = A.S == OZ_FP64 ? OzCfg<OZ_FP64>::PRODUCTS : A.S == 5 ? OzCfg<5>::PRODUCTS : OzCfg<4>::PRODUCTS;
    for (int r = 0; r < g.per; ++r) {
      int bx, by, k0, k1;
      oz_tile_xy(g.order, g.gx, g.gy, r, &bx, &by);
      oz_krange(tk, kmode, g.a_rb0 * OZ_TR + bx * OZ_BM, g.b_rb0 * OZ_TR + by * OZ_BN, g.kc0, g.kc1, &k0, &k1);
      if (k1 > k0) fl += 2.0 * OZ_BM * OZ_BN * tk * (double)(k1 - k0) * prods;
    }
    fl *= (double)batch;
  }
  {
    KTScope kts(GPGP_KPROF_OZ_GEMM, s, fl);
    if (A.S == OZ_FP64) launch_oz_gemm<OZ_FP64>(s, grid, g);
    else if (A.S == 5) launch_oz_gemm<5>(s, grid, g);
    else launch_oz_gemm<4>(s, grid, g);
  }
  GPGP_CHECK_LAUNCH();
}

int oz_sms() { return oz_sm_count(); }

void oz_gemm(cudaStream_t s, const OzSplit &A, int64_t a_row0, const OzSplit &B, int64_t b_row0,
             int64_t M, int64_t N, int64_t kc0, int64_t kc1, int kmode, double alpha, double beta,
             double *C, int64_t ldc, bool lower_only, int *err, const int *status) {
  oz_gemm_batched(s, A, a_row0, B, b_row0, M, N, kc0, kc1, kmode, alpha, beta, C, ldc, 0, lower_only,
                  err, status, 0, 1);
}

// ---------------------------------------------------------------------------
// a 64-wide block column of the Cholesky's outer panel, in one kernel
// ---------------------------------------------------------------------------
// Rows [r0, r1) of the block column at j0, 128 to a CTA:
//   L = A W^T (W: the diagonal block's inverse), written over A, then
//   A_q -= L L_q^T for the panel's next q1 64-wide column blocks, L_q the rows j0 + 64 (q + 1)
//   .. of the block column (finished before).
// Every operand is 64 K wide, so it is split where it is used: the rows' exponents and
// slices go from registers to shared memory and on to the tensor cores, and neither the
// slices nor L in slices pass through memory. As split, split, product, split, split,
// product the block took six launches and ~280 us of a 32-SM share at n = 16384 for work
// of ~20 us. The products, their order and their rounding are those of oz_split and
// oz_gemm. (One loop body serves every
// round: its phases run once or a few times, and with a copy for each product the warps
// spent 44% of their time waiting for instructions.)
// A round takes ~15 us, most of it latency, so where there are fewer tiles than SMs a tile
// gets a cluster of `group` CTAs: each forms L for itself, the first one writes it (when
// all have read A), and the column blocks are dealt between them: with 21 tiles the first
// block of a panel takes 37 us instead of 95, the six 170 instead of 350, and the panel no
// longer waits for them (n = 3000, FP64: 3.49 -> 3.23 ms for the factorisation).
constexpr int PB_THREADS = 512;
constexpr int PB_SBO = 1024;  // 8 rows x 64 K x 2 bytes
constexpr int PB_LEAVE = 40;  // SMs that groups leave

template <int S>
struct PbCfg {
  static constexpr int A_SL = OZ_BM * 64 * 2, B_SL = OZ_BN * 64 * 2;  // a slice of 64 K
  static constexpr int SMEM = S * (A_SL + B_SL) + 1024;
  static constexpr uint32_t TMEM_COLS = OzCfg<S>::NACC * OZ_BN;  // 256 or 512
};

// NV entries (a multiple of 8) of row r, K 8 kg0 .., as slices at base. Rolled over the
// pairs: the kernel's phases run once or a few times each, and with everything unrolled
// its warps spent 44% of their time waiting for instructions.
template <int S, int NV>
__device__ __forceinline__ void pb_put(uint8_t *base, int sl, int r, int kg0, const double *v, int e) {
  uint8_t *dst = base + (r >> 3) * PB_SBO + kg0 * 128 + (r & 7) * 16;
#pragma unroll
  for (int g = 0; g < NV / 8; ++g)
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      uint32_t w[S];
      oz_pair<S>(v[8 * g + j], v[8 * g + j + 1], e, w);
#pragma unroll
      for (int t = 0; t < S; ++t) *reinterpret_cast<uint32_t *>(dst + t * sl + g * 128 + 2 * j) = w[t];
    }
}

__device__ __forceinline__ int pb_field(double v) {
  return (int)(((unsigned long long)__double_as_longlong(v) >> 52) & 0x7FF);
}

template <int S>
__global__ void __launch_bounds__(PB_THREADS) panel_block_kernel(double *__restrict__ A, int64_t lda, int64_t r0,
                                                                 int64_t r1, int64_t j0,
                                                                 const double *__restrict__ W, int q1, int group,
                                                                 int *err, const int *__restrict__ status,
                                                                 uint32_t polls) {
  using Cfg = PbCfg<S>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *As = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023), *Bs = As + S * Cfg::A_SL;
  __shared__ int amax[OZ_BM], bmax[OZ_BN];
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_sh;
  if (status && *(volatile const int *)status != 0) return;
  const int tid = threadIdx.x, warp = tid >> 5;
  if (tid == 0) {
    mbar_init(smem_u32(&bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_sh)),
                 "r"(Cfg::TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_sh;
  // this thread's row of the tile and its 16 columns of a 64-wide block; in the second
  // operand its row and 8 columns
  const int row = tid & 127, part = tid >> 7, brow = tid & 63, bpart = tid >> 6;
  const uint32_t ta = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(part * 16);
  const uint64_t ad = umma_desc(smem_u32(As), 128u, PB_SBO), bd = umma_desc(smem_u32(Bs), 128u, PB_SBO);
  uint32_t ph = 0;
  bool ok = true;
  // operands in shared memory -> products in TMEM (false: the wait ran out)
  auto product = [&]() -> bool {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
      tc_fence_after();
      if (elect_one()) {
        oz_issue<S, 4>(ad, bd, Cfg::A_SL, Cfg::B_SL, tmem, 0u);
        umma_commit(smem_u32(&bar));
      }
      __syncwarp();
    }
    const bool done = mbar_wait_bounded(smem_u32(&bar), ph, polls);
    ph ^= 1u;
    tc_fence_after();
    return !__syncthreads_or(!done);
  };
  // TMEM -> 16 doubles of this thread's row (power of two ea) and columns (bmax)
  auto results = [&](double (&v)[16], int ea, uint32_t negmask) {
#pragma unroll
    for (int h = 0; h < 16; h += 8) {
      typename OzSum<S>::Hi hi[8];
      typename OzSum<S>::Lo lo[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        hi[j] = 0;
        lo[j] = 0;
      }
      oz_drain<S, 8>(ta + (uint32_t)h, hi, lo);
      bool slow = false;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int sh = ea + oz_exponent<S>(bmax[part * 16 + h + j]);
        if constexpr (OzCfg<S>::FP64) {
          v[h + j] = fixed_to_double(hi[j], lo[j], sh, negmask, slow);
        } else {
          hi[j] = __uint_as_float(__float_as_uint(hi[j]) ^ negmask);
          lo[j] = __uint_as_float(__float_as_uint(lo[j]) ^ negmask);
          v[h + j] = df2d_try(hi[j], lo[j], sh - 16, slow);
        }
      }
      if (__any_sync(0xffffffffu, slow)) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int sh = ea + oz_exponent<S>(bmax[part * 16 + h + j]);
          if constexpr (OzCfg<S>::FP64) v[h + j] = fixed_to_double_slow(hi[j], lo[j], sh, negmask);
          else v[h + j] = df2d_scaled(hi[j], lo[j], sh - 16);
        }
      }
    }
    tc_fence_before();
  };
  // the second operand: 64 rows of P (leading dimension ld)
  auto load_b = [&](const double *P, int64_t ld) {
    double b[8];
    int mx = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      b[k] = P[brow + (8 * bpart + k) * ld];
      mx = max(mx, pb_field(b[k]));
    }
    atomicMax(&bmax[brow], mx);
    __syncthreads();
    pb_put<S, 8>(Bs, Cfg::B_SL, brow, bpart, b, oz_exponent<S>(bmax[brow]));
  };
  // the first operand: this thread's 16 entries of its row; returns the row's power of two
  auto put_a = [&](const double (&v)[16]) -> int {
    int mx = 0;
#pragma unroll
    for (int k = 0; k < 16; ++k) mx = max(mx, pb_field(v[k]));
    atomicMax(&amax[row], mx);
    __syncthreads();
    const int e = oz_exponent<S>(amax[row]);
    pb_put<S, 16>(As, Cfg::A_SL, row, 2 * part, v, e);
    return e;
  };
  const int tiles = (int)gridDim.x / group, g = (int)blockIdx.x % group;  // (the cluster of CTAs has this tile's rows)
  for (int64_t t0 = r0 + (int64_t)(blockIdx.x / group) * OZ_BM; ok && t0 < r1; t0 += (int64_t)tiles * OZ_BM) {
    const int64_t gr = t0 + row;
    const bool in = gr < r1;
    double v[16];
    double *ar = A + gr + (j0 + 16 * part) * lda;
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = in ? ar[k * lda] : 0.0;
    // every CTA of the cluster has read A before the first writes L over it (a cluster has
    // one tile, so its CTAs come here together and once)
    if (group > 1) cluster_arrive();
    int ea = 0;
    // round -1: L = A W^T; round q: the update of column block q
#pragma unroll 1
    for (int q = -1; q < q1; q = q < 0 ? g : q + group) {
      __syncthreads();
      if (tid < OZ_BN) bmax[tid] = 0;
      const bool newa = q <= g;  // A, then L as the first operand
      if (newa && tid >= 128 && tid < 128 + OZ_BM) amax[tid - 128] = 0;
      __syncthreads();
      if (newa) ea = put_a(v);
      const double *P = q < 0 ? W : A + j0 + 64 * (q + 1) + j0 * lda;
      load_b(P, q < 0 ? NB : lda);
      double *cr = A + gr + (j0 + 64 * (q + 1) + 16 * part) * lda;
      double c[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) c[k] = q >= 0 && in ? cr[k * lda] : 0.0;
      const bool done = product();
      if (q < 0 && group > 1) cluster_wait();
      ok = done;
      if (!ok) break;
      double u[16];
      results(u, ea, q < 0 ? 0u : 0x80000000u);
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        if (q < 0) v[k] = u[k];
        else u[k] += c[k];
        if (in && (q >= 0 || g == 0)) cr[k * lda] = u[k];
      }
    }
  }
  if (!ok && tid == 0) {
    atomicExch(err, 5);
    // the products that were waited for land (bounded) before their operands' shared memory
    // and their TMEM are released
    mbar_wait_bounded(smem_u32(&bar), ph ^ 1u);
  }
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::TMEM_COLS));
  }
}

template <int S>
static void launch_panel_block(cudaStream_t s, double *A, int64_t lda, int64_t r0, int64_t r1, int64_t j0,
                               const double *W, int q1, int *err, const int *status) {
  static PerDevice attr;
  per_device(attr, [] {
    GPGP_CUDA(cudaFuncSetAttribute(panel_block_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   PbCfg<S>::SMEM));
    return 1;
  });
  const int cap = tl_oz_grid_cap > 0 ? std::min(tl_oz_grid_cap, oz_sm_count()) : oz_sm_count();
  const int64_t tiles = (r1 - r0 + OZ_BM - 1) / OZ_BM;
  const double fl = 2.0 * OZ_BM * OZ_BN * 64 * (double)tiles * (1 + q1) * OzCfg<S>::PRODUCTS;
  KTScope kts(GPGP_KPROF_OZ_GEMM, s, fl);
  // the smallest group with the fewest rounds that leaves the chain's kernels some SMs
  const int64_t room = cap - PB_LEAVE;
  int group = 1;
  for (int g = 2; g <= q1 && g <= 8 && tiles * g <= room; ++g)
    if ((q1 + g - 1) / g < (q1 + group - 1) / group) group = g;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim = {(unsigned)group, 1, 1};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(group > 1 ? tiles * group : std::min<int64_t>(tiles, cap)));
  cfg.blockDim = dim3(PB_THREADS);
  cfg.dynamicSmemBytes = PbCfg<S>::SMEM;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  GPGP_CUDA(cudaLaunchKernelEx(&cfg, panel_block_kernel<S>, A, lda, r0, r1, j0, W, q1, group, err, status,
                               tl_wait.polls[GPGP_WAIT_PANEL]));
  GPGP_CHECK_LAUNCH();
}

void panel_block(cudaStream_t s, int S, double *A, int64_t lda, int64_t r0, int64_t r1, int64_t j0, const double *W,
                 int q1, int *err, const int *status) {
  if (r1 <= r0) return;
  if (S == OZ_FP64) launch_panel_block<OZ_FP64>(s, A, lda, r0, r1, j0, W, q1, err, status);
  else launch_panel_block<4>(s, A, lda, r0, r1, j0, W, q1, err, status);
}

}  // namespace gpgp

// ---------------------------------------------------------------------------
// bounded-wait self-test: an mbarrier that is never completed (two arrivals
// expected, one made), polled with the same loop as the GEMM's waits but with a
// caller-chosen bound; the kernel records the timeout and returns
// ---------------------------------------------------------------------------
namespace gpgp {
__global__ void wait_selftest_kernel(uint32_t polls, int *err) {
  __shared__ uint64_t bar;
  __shared__ int abort_sh;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar), 2);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    abort_sh = 0;
    mbar_arrive(smem_u32(&bar));
    bool done = false;
    for (uint32_t it = 0; it < polls && !done; ++it) done = mbar_try_wait(smem_u32(&bar), 0);
    if (!done) atomicExch(err, 4);
  }
  __syncthreads();
}
}  // namespace gpgp

extern "C" gpgp_status gpgp_wait_bound(int32_t kernel, int32_t polls, int32_t gemm_chunks) {
  using namespace gpgp;
  if (kernel < 0 || kernel >= GPGP_NWAIT) return GPGP_EINVAL;
  tl_wait.polls[kernel] = polls < 0 ? kWaitDefault.polls[kernel] : (uint32_t)polls;
  tl_wait.gemm_chunks = gemm_chunks < 0 ? kWaitDefault.gemm_chunks : gemm_chunks;
  return GPGP_OK;
}

extern "C" gpgp_status gpgp_wait_selftest(gpgp_ctx *ctx, int32_t polls) {
  if (!ctx || polls < 1) return GPGP_EINVAL;
  return gpgp::guarded(ctx, [&]() -> gpgp_status {
    GPGP_CUDA(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    gpgp::IBuf err;
    err.alloc(s, 1);
    GPGP_CUDA(cudaMemsetAsync(err.p, 0, sizeof(int), s));
    gpgp::wait_selftest_kernel<<<1, 32, 0, s>>>((uint32_t)polls, err.p);
    GPGP_CHECK_LAUNCH();
    int h = 0;
    GPGP_CUDA(cudaMemcpyAsync(&h, err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    GPGP_CUDA(cudaStreamSynchronize(s));
    if (h) return gpgp::fail(ctx, GPGP_ETIMEOUT, "a bounded device wait ran out (self-test)");
    return GPGP_OK;
  });
}
