// The Cholesky's diagonal block: factor and inverse of up to 64 x 64 FP64 entries, by a
// cluster of CTAs (one block) or by one CTA each (many blocks).
#include <math.h>

#include <algorithm>

#include "bulk.cuh"
#include "common.cuh"
#include "fp64math.cuh"

namespace gpgp {

// -x by flipping the sign bit (an integer instruction, not an FP64 one)
__device__ __forceinline__ double neg_bits(double x) {
  return __longlong_as_double(__double_as_longlong(x) ^ (long long)0x8000000000000000ull);
}

// ---------------------------------------------------------------------------
// one block: a cluster, a block column to each CTA
// ---------------------------------------------------------------------------
// On this part an FP64 warp instruction holds its SM sub-partition for 64 cycles (76 with
// all four busy, 1.7 multiply-adds a clock for the SM), and a dependent one waits as long.
// The block's factor and inverse, 2 x 43.7 k multiply-adds, are 52 k cycles of one SM's
// pipe, and the chain of the 64 pivots (an update, five instructions of the inverse square
// root, a scaling) another 40 k, in which nothing else may hold its sub-partition. So the
// chain moves on through segments of 4 columns, each in the registers of a warp of its
// own, one segment to a sub-partition of the four SMs of a cluster, and everything else is
// kept off the sub-partition whose turn it is:
//  - a chain warp holds its columns' rows 0..31 (from segment 8 on 32..63), a row to a
//    lane. It takes the columns before its segment one by one as they are published (own[]
//    of its CTA, col[] from the others, a barrier for each half column) and then pivots its
//    own. The next pivot's column is updated first, the others when the inverse square
//    root has been started (held()). Rows 32..63 of segments 0..7 are in the registers of
//    a second warp, which follows.
//  - one warp sends the finished columns to the CTAs after this one (st.async, counted
//    by the receiver's barrier), another forms V's first terms and sends those to the CTAs
//    before it.
//  - the inverse W = D^-1 V, D = diag(L), V the unit lower triangular inverse of L D^-1:
//      V(i, c) = -sum_{k=c..i-1} (L(i, k) / L(k, k)) V(k, c),  V(c, c) = 1,
//    term k = c from the pivot, the others in the order in which the columns arrive. The
//    warps of a segment that is done build its columns, beside the others' pivots.
// 43 us a block: ~650 cycles from pivot to pivot, 85 for each update on the way, 300 from
// one segment's warp to the next. One CTA with a barrier per column took 66 us; with the
// products of 16 x 16 blocks in fixed point on the integer pipe, 51. (Segments of 8 in two
// warps to a CTA 47 us, a cluster of 8 with the columns dealt to four warps in turn 49.)
// Every entry takes the same operations in the same order as in the one-CTA kernel below,
// so the two give the same bits. That matters to the mixed precision: its updates cut
// their operands to 32 bits, so any other rounding here draws the whole truncation anew
// (predicted variances, whose error is 2e-8 of their scale, moved by 2e-9 of it).
constexpr int DIAG_C = 4;         // CTAs of the cluster
constexpr int DCW = NB / DIAG_C;  // columns of a CTA
constexpr int DSEG = 4;           // columns of a segment
constexpr int DCT = 320;          // threads: eight compute warps and two that send

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// 8 or 16 bytes to a peer's shared memory, counted by the peer's barrier
__device__ __forceinline__ void send8(uint32_t dst, double v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void send16(uint32_t dst, double2 v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
               "l"(__double_as_longlong(v.x)), "l"(__double_as_longlong(v.y)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  cluster_arrive();
  cluster_wait();
}
// Bounded wait for phase 0 of a barrier that another CTA completes (a second or so)
__device__ __forceinline__ bool wait_peer(uint32_t bar, uint32_t polls = WAIT_POLLS) {
  for (uint32_t it = 0; it < polls; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// x, in a form that the compiler must take to depend on `after`: keeps FP64 instructions
// out of the pivot chain's way until `after` is known (sel is 0x3210)
__device__ __forceinline__ double held(double x, double after, uint32_t sel) {
  return __hiloint2double(__double2hiint(x), __byte_perm(__double2loint(x), __double2hiint(after), sel));
}

// TEST: waits of max_polls polls (gpgp_wait_bound)
template <bool TEST>
__global__ void __cluster_dims__(DIAG_C, 1, 1) __launch_bounds__(DCT)
    potrf_diag_kernel(double *__restrict__ A, int kb, int64_t lda, double *__restrict__ Winv,
                      double *__restrict__ logdet_part, int *__restrict__ status, int64_t k0, int64_t sA, int64_t sW,
                      int64_t sL, uint32_t max_polls) {
  const uint32_t polls = TEST ? max_polls : WAIT_POLLS;
  constexpr int C = DIAG_C, PW = DCW;
  static_assert(NB == 64 && PW == 4 * DSEG, "a segment to a sub-partition");
  __shared__ __align__(16) double col[NB][NB];  // column k < base: L(:, k); else V's first terms -L(:, k) / L(k, k)
  __shared__ __align__(16) double own[PW][NB];  // this CTA's columns of L
  __shared__ double rd[NB];                     // 1 / L(k, k)
  __shared__ double lg[NB];                     // rank 0: the logarithms of the diagonal
  // rows 0..31 and 32..63 of column k are here (k >= base + PW: V's are, all rows by the
  // second); each used once
  __shared__ uint64_t full[2][NB];
  __shared__ uint64_t vown[PW];  // V's first terms of this CTA's columns
  __shared__ int failc, fails[C];
  const int64_t prob = blockIdx.x / C;  // batched: strides sA, sW, sL; one status word per problem
  A += prob * sA;
  Winv += prob * sW;
  logdet_part += prob * sL;
  status += prob;
  if (*(volatile int *)status != 0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)cluster_rank(), base = rank * PW;
  // a compute warp's segment and rows: warps 0..3 pivot, 4..7 follow with rows 32..63 where
  // the pivots lie above them, segment f's on sub-partition f + 1 (f's pivots are on f, and
  // those after f come when f's follower is done)
  const bool chain = warp < 4;
  const int sb = base + DSEG * (chain ? warp : (warp + 3) & 3), half = chain ? sb >> 5 : 1, row = 32 * half + lane;
  const bool compute = warp < 8 && sb < kb && (chain || sb < 32);
  double a[DSEG];
#pragma unroll
  for (int q = 0; q < DSEG; ++q)
    a[q] = compute && row >= sb + q && row < kb && sb + q < kb ? A[row + (sb + q) * lda] : 0.0;
  if (tid < kb) {
    const uint32_t b0 = smem_u32(&full[0][tid]), b1 = smem_u32(&full[1][tid]);
    mbar_init(b0, 1);
    mbar_init(b1, 1);
    if (tid < PW) mbar_init(smem_u32(&vown[tid]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (tid < base) {
      if (base < 32) mbar_expect_tx(b0, (32 - base) * 8);
      mbar_expect_tx(b1, (NB - max(32, base)) * 8);
    } else if (tid >= base + PW) {
      mbar_expect_tx(b1, (NB - tid / PW * PW + 1) * 8);
    }
  }
  if (tid < NB) lg[tid] = 0.0;
  if (tid == 0) failc = NB;
  __syncthreads();
  cluster_sync();
  const uint32_t col_a = smem_u32(col), full_a = smem_u32(full), rd_a = smem_u32(rd);
  auto bar = [&](int h, int k) { return full_a + (uint32_t)(h * NB + k) * 8; };
  bool ok = true;
  const int kown = min(base + PW, kb);  // own columns end
  auto wait = [&](int h, int k) {
    if (ok && !(k >= base && k < kown ? mbar_wait_bounded(bar(h, k), 0, polls) : wait_peer(bar(h, k), polls))) {
      ok = false;
      atomicMin(&failc, -1);
    }
  };
  if (compute) {
    double lp = 0.0, lc[DSEG];  // the column before and its entries at the rows of this segment's columns
#pragma unroll
    for (int q = 0; q < DSEG; ++q) lc[q] = 0.0;
    auto receive = [&](int k) {
      wait(half, k);
      if (!chain) wait(0, k);
      const double *c = k < base ? col[k] : own[k - base];
      lp = c[row];
#pragma unroll
      for (int q = 0; q < DSEG; ++q) lc[q] = c[sb + q];
      a[0] = fma(-lp, lc[0], a[0]);
    };
#pragma unroll 1
    for (int k = 0; k + 1 < sb; ++k) {
      receive(k);
#pragma unroll
      for (int q = 1; q < DSEG; ++q) a[q] = fma(-lp, lc[q], a[q]);
    }
    if (sb > 0) receive(sb - 1);
    const int n = min(DSEG, kb - sb);
    if (chain) {
      const int pl = sb & 31;
      const bool odd = lane & 1;
      const double c0 = odd ? 0.5 : -0.0;
      const uint32_t sel = 0x3210u + ((uint32_t)kb >> 16);
#pragma unroll
      for (int j = 0; j < DSEG; ++j) {
        if (j >= n) break;
        const int k = sb + j;
        const double d = __shfl_sync(0xffffffffu, a[j], pl + j);
        // rsqrt_fast(d), with the updates that the pivot before left for now in its gaps
        const double y0 = rsqrt_seed(d);
        const double c1 = odd ? 0.375 : y0;
        const double l1 = held(lp, d, sel);
#pragma unroll
        for (int q = j + 1; q < DSEG && q < j + 2; ++q) a[q] = fma(-l1, lc[q], a[q]);
        const double e = fma(-(d * y0), y0, 1.0);
        const double z = fma(e, c1, c0);  // y0 e on even lanes, 3/8 e + 1/2 on odd ones
        double rp = fma(__shfl_sync(0xffffffffu, z, 0), __shfl_sync(0xffffffffu, z, 1), y0);
        // not positive (sign bit or zero) or not finite, tested on the bits
        const long long db = __double_as_longlong(d);
        const bool bad = db <= 0ll || (db >> 52) >= 0x7FFll;
        if (bad || !rsqrt_in_range(d)) rp = rsqrt_fast(bad ? 1.0 : d);
        const double l = a[j] * rp;
        const double l2 = held(lp, rp, sel);
#pragma unroll
        for (int q = j + 2; q < DSEG; ++q) a[q] = fma(-l2, lc[q], a[q]);
        if (j + 1 < DSEG) a[j + 1] = fma(-l, __shfl_sync(0xffffffffu, l, pl + j + 1), a[j + 1]);
        double *oc = own[k - base];
        oc[row] = l;
        if (lane == 0) {
          rd[k] = rp;
          if (bad) atomicMin(&failc, k);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(half, k));
        lp = l;
#pragma unroll
        for (int q = j + 2; q < DSEG; ++q) lc[q] = oc[sb + q];
      }
    } else {
      if (sb > 0)
#pragma unroll
        for (int q = 1; q < DSEG; ++q) a[q] = fma(-lp, lc[q], a[q]);
#pragma unroll 1
      for (int j = 0; j < n; ++j) {
        const int k = sb + j;
        double *oc = own[k - base];
        wait(0, k);
        const double l = a[0] * rd[k];
        oc[row] = l;
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(1, k));
#pragma unroll
        for (int q = 1; q < DSEG; ++q) a[q - 1] = q < DSEG - j ? fma(-l, oc[k + q], a[q]) : 0.0;
      }
    }
  } else if (warp == 8) {
    // the finished columns to the CTAs after this one that have columns
#pragma unroll 1
    for (int k = base; k < kown; ++k)
#pragma unroll 1
      for (int h = k >> 5; h < 2; ++h) {
        wait(h, k);
        const int r = 32 * h + 2 * lane;
        const double2 v = lane < 16 ? *reinterpret_cast<const double2 *>(&own[k - base][r]) : make_double2(0.0, 0.0);
        for (int dst = rank + 1; dst < C && dst * PW < min(kb, 32 * (h + 1)); ++dst)
          if (lane < 16 && r >= dst * PW)
            send16(peer_addr(col_a + (uint32_t)(k * NB + r) * 8, dst), v, peer_addr(bar(h, k), dst));
      }
    // the logarithms of the diagonal, to rank 0
    if (base + lane < kown) {
      const double l = log(own[lane][base + lane]);
      asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(peer_addr(smem_u32(&lg[base + lane]), 0)),
                   "l"(__double_as_longlong(l))
                   : "memory");
    }
  } else if (warp == 9) {
    // V's first terms, here and to the CTAs before this one
    const int r = 2 * lane;
#pragma unroll 1
    for (int k = base; k < kown; ++k) {
      if (k < 32) wait(0, k);
      wait(1, k);
      const double rp = rd[k];
      const double2 l = *reinterpret_cast<const double2 *>(&own[k - base][r]);
      const double2 v = make_double2(-(l.x * rp), -(l.y * rp));
      if (r >= base) {
        *reinterpret_cast<double2 *>(&col[k][r]) = v;
        for (int dst = 0; dst < rank; ++dst)
          send16(peer_addr(col_a + (uint32_t)(k * NB + r) * 8, dst), v, peer_addr(bar(1, k), dst));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&vown[k - base]));
      if (lane < rank) send8(peer_addr(rd_a + 8 * k, lane), rp, peer_addr(bar(1, k), lane));
    }
  }
  // the inverse: warps f and f + 4 take two columns each of segment f, whose sub-partition
  // is free from then on, a lane rows row0 and row1
  const int row0 = base + lane, row1 = row0 + 32;
  const bool in0 = row0 < NB, in1 = row1 < NB;
  const int cw = base + DSEG * (warp & 3) + 2 * (warp >> 2);
  double v[2][2];
  if (warp < 8 && cw < kb) {
    auto wait_v = [&](int k) {
      if (k >= kown) wait(1, k);
      else if (ok && !mbar_wait_bounded(smem_u32(&vown[k - base]), 0, polls)) {
        ok = false;
        atomicMin(&failc, -1);
      }
    };
    wait_v(cw);
    v[0][0] = in0 && row0 > cw ? col[cw][row0] : 0.0;
    v[0][1] = in1 ? col[cw][row1] : 0.0;
    v[1][0] = v[1][1] = 0.0;
#pragma unroll 1
    for (int k = cw + 1; k < kb; ++k) {
      const int lr = k - base;
      wait_v(k);
      const double f0 = in0 ? col[k][row0] : 0.0, f1 = in1 ? col[k][row1] : 0.0;
      double vk[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) vk[q] = __shfl_sync(0xffffffffu, lr < 32 ? v[q][0] : v[q][1], lr & 31);
      if (k == cw + 1) {
        v[1][0] = row0 > k ? f0 : 0.0;
        v[1][1] = f1;
      }
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (cw + q < k) {
          if (lr < 31) {
            const double t = fma(f0, vk[q], v[q][0]);
            v[q][0] = row0 > k ? t : v[q][0];
          }
          if (base < 32) {
            const double t = fma(f1, vk[q], v[q][1]);
            v[q][1] = row1 > k ? t : v[q][1];
          }
        }
    }
  }
  __syncthreads();
  if (tid < C)
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(peer_addr(smem_u32(&fails[rank]), tid)), "r"(failc)
                 : "memory");
  cluster_sync();
  int bad = NB;
#pragma unroll
  for (int r = 0; r < C; ++r) bad = min(bad, fails[r]);
  if (bad < NB) {
    // A wait ran out: every CTA still sends all it would have, and a CTA stays until what
    // is sent to it has landed (bounded).
    if (bad < 0 && tid < kb && base < kb && (tid < base || tid >= base + PW)) {
      if (tid < base && base < 32) wait_peer(bar(0, tid));
      wait_peer(bar(1, tid));
    }
    if (rank == 0 && tid == 0) atomicCAS(status, 0, bad < 0 ? STATUS_TIMEOUT : (int)(k0 + bad + 1));
    return;
  }
  for (int idx = tid; idx < PW * NB; idx += DCT) {
    const int r = idx % NB, cl = idx / NB, c = base + cl;
    if (c < kb && r >= c && r < kb) A[r + c * lda] = own[cl][r];
    if (r < base) Winv[r + c * NB] = 0.0;
  }
  if (warp < 8)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int c = cw + q;
      if (in0) Winv[row0 + c * NB] = row0 < kb && row0 >= c ? (row0 == c ? rd[c] : rd[row0] * v[q][0]) : 0.0;
      if (in1) Winv[row1 + c * NB] = row1 < kb && c < kb ? rd[row1] * v[q][1] : 0.0;
    }
  if (rank == 0 && warp == 8) {  // log det in a fixed order
    double l = lg[lane] + lg[lane + 32];
    for (int o = 16; o > 0; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
    if (lane == 0) *logdet_part = l;
  }
}

// ---------------------------------------------------------------------------
// many blocks: one CTA each
// ---------------------------------------------------------------------------
// On this part the FP64 pipe retires about 2 lane operations per clock per SM,
// and a warp instruction occupies it whether 1 or 32 lanes are active, so the
// kernel issues as few FP64 warp instructions as it can, each with all lanes on
// distinct entries, and runs the factor and the inverse in one loop with one
// barrier per column:
//  - factor, right-looking: warp 0 takes the pivots one column ahead (column
//    j+1 gets its update from column j, then its inverse square root,
//    rsqrt_fast) while the update warps apply the rank-1 update of column j to
//    the trailing triangle c >= j+2. The trailing triangle's entries are
//    numbered by column, last column first, so that step j's entries are the
//    first (kb-2-j)(kb-1-j)/2 of one fixed list. The warps that share warp 0's
//    sub-partition take no update work; the other twelve (three per
//    sub-partition, enough to cover the FP64 latency) share it evenly.
//  - inverse: W = L^-1 = D^-1 V with D = diag(L) and V the unit lower triangular
//    inverse of the column-scaled factor L D^-1:
//      V(i, c) = -sum_{k=c..i-1} (L(i, k) / L(k, k)) V(k, c),  V(c, c) = 1.
//    The k = c term is written by the pivot of column c (V(i, c) starts as
//    -L(i, c) / L(c, c)); the terms k > c are added right-looking, step k adding
//    V(i, k) V(k, c) to every (i > k, c < k) while V(i, k) still holds only its
//    first term. Step k needs column k of L and rows <= k of V final, so it runs
//    beside the factor's step k + 1 in the same loop iteration. Every inverse
//    entry costs one FMA; the row scaling by 1 / L(i, i) happens once, on the
//    way out.
//  - log L_jj summed in a fixed tree order.
constexpr int DIAG_THREADS = 512;

__device__ __forceinline__ int div_small(int e, int d, int magic) {
  // e / d for e < 4096, 1 <= d <= 64, magic = ceil(2^20 / d): exact on that range
  return (int)(((unsigned)e * (unsigned)magic) >> 20);
}

__global__ void __launch_bounds__(DIAG_THREADS) potrf_diag_many_kernel(double *__restrict__ A, int kb, int64_t lda,
                                                         double *__restrict__ Winv,
                                                         double *__restrict__ logdet_part,
                                                         int *__restrict__ status, int64_t k0,
                                                         int64_t sA, int64_t sW, int64_t sL) {
  // batched: problem blockIdx.x (strides sA, sW, sL; status has one word per problem)
  A += blockIdx.x * sA;
  Winv += blockIdx.x * sW;
  logdet_part += blockIdx.x * sL;
  status += blockIdx.x;
  __shared__ double S[NB][NB + 1];
  __shared__ double V[NB][NB + 1];
  __shared__ double rdiag[NB];
  __shared__ double lg[NB];
  __shared__ unsigned short pairs[NB * (NB + 1) / 2];  // (r | c << 8), column-major from the last column
  __shared__ int failed;
  if (*(volatile int *)status != 0) return;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  for (int idx = tid; idx < NB * NB; idx += DIAG_THREADS) {
    const int r = idx % NB, c = idx / NB;
    // held negated until its column is pivoted (see the update loop)
    S[r][c] = (r < kb && c < kb && r >= c) ? neg_bits(A[r + c * lda]) : 0.0;
    V[r][c] = 0.0;
  }
  // entry e of the kb x kb triangle: u = kb - 1 - c is the largest u with
  // u (u + 1) / 2 <= e; r = c + e - u (u + 1) / 2 (a partial block lists only its
  // own entries)
  for (int e = tid; e < kb * (kb + 1) / 2; e += DIAG_THREADS) {
    int u = (int)((sqrtf(8.0f * (float)e + 1.0f) - 1.0f) * 0.5f);
    while (u * (u + 1) / 2 > e) --u;
    while ((u + 1) * (u + 2) / 2 <= e) ++u;
    const int c = kb - 1 - u, r = c + (e - u * (u + 1) / 2);
    pairs[e] = (unsigned short)(r | (c << 8));
  }
  if (tid == 0) failed = 0;
  __syncthreads();
  // Warp 0 keeps the current scaled column in registers: lane l owns rows l and
  // l + 32, and lreg[u] holds L(l + 32 u, j) once column j is pivoted. Rows below
  // 32 drop out after column 31, so their FP64 work is skipped from then on (a
  // warp instruction costs the same with one lane or 32).
  double lreg[2] = {0.0, 0.0};
  // pivot of column j by warp 0 from t[u] = -S(l + 32 u, j) after all updates:
  // L_jj, the scaled column below it (stored positive, and kept in lreg) and the
  // first term of column j of V
  auto pivot = [&](int j, const double (&t)[2]) {
    const double dj = neg_bits(__shfl_sync(0xffffffffu, j < 32 ? t[0] : t[1], j & 31));
    // not positive (sign bit or zero) or not finite, tested on the bits
    const long long djb = __double_as_longlong(dj);
    if (djb <= 0ll || (djb >> 52) >= 0x7FFll) {
      if (lane == 0) {
        failed = 1;
        atomicCAS(status, 0, (int)(k0 + j + 1));
      }
      return;
    }
    const double rp = rsqrt_fast(dj);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (u == 1 || j < 31) {
        const int r = lane + 32 * u;
        if (r > j && r < kb) {
          const double l = -(t[u] * rp);
          S[r][j] = l;
          V[r][j] = -(l * rp);
          lreg[u] = l;
        }
      }
    }
    if (lane == (j & 31)) {
      S[j][j] = dj * rp;
      rdiag[j] = rp;
    }
  };
  if (warp == 0) {
    double t0[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) t0[u] = (lane + 32 * u < kb) ? S[lane + 32 * u][0] : 0.0;
    pivot(0, t0);
  }
  __syncthreads();
  if (failed) return;
  // update workers: every warp off sub-partition 0 (warps 4, 8, 12 share warp 0's)
  constexpr int NUPD = DIAG_THREADS / 32 - DIAG_THREADS / 128;  // 12 update warps
  const int uw = warp - 1 - (warp >> 2);
  const int ut = uw * 32 + lane;
  for (int j = 0; j < kb; ++j) {
    if (warp == 0) {
      if (j + 1 < kb) {
        // column j + 1 takes its last update, from column j, then its pivot
        const double l = __shfl_sync(0xffffffffu, (j + 1) < 32 ? lreg[0] : lreg[1], (j + 1) & 31);
        double t[2] = {0.0, 0.0};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (u == 1 || j < 31) {
            const int r = lane + 32 * u;
            if (r > j && r < kb) t[u] = fma(lreg[u], l, S[r][j + 1]);
          }
        }
        pivot(j + 1, t);
      }
    } else if ((warp & 3) != 0) {
      // factor step j: entries (r, c), c >= j + 2, of the fixed list; inverse step
      // k = j - 1: entries (i, c), k < i < kb, c < k, row-major by i. Both are
      // dst += a b with a, b >= sign-free operands (the trailing matrix is held
      // negated), so that each entry is exactly one FP64 instruction.
      const int cf = j < kb - 2 ? (kb - 2 - j) * (kb - 1 - j) / 2 : 0;
      const int k = j - 1;
      const int ci = k >= 1 ? (kb - 1 - k) * k : 0;
      const int magic = k >= 1 ? ((1 << 20) + k - 1) / k : 0;
      for (int e = ut; e < cf + ci; e += NUPD * 32) {
        const double *pa, *pb;
        double *dst;
        if (e < cf) {
          const unsigned short pc = pairs[e];
          const int r = pc & 0xFF, c = pc >> 8;
          dst = &S[r][c];
          pa = &S[r][j];
          pb = &S[c][j];
        } else {
          const int e2 = e - cf;
          const int q = div_small(e2, k, magic);
          const int c = e2 - q * k, i = k + 1 + q;
          dst = &V[i][c];
          pa = &V[i][k];
          pb = &V[k][c];
        }
        *dst = fma(*pa, *pb, *dst);
      }
    }
    __syncthreads();
    if (failed) return;
  }
  // write the factor back (lower part of the block)
  for (int idx = tid; idx < kb * kb; idx += DIAG_THREADS) {
    const int r = idx % kb, c = idx / kb;
    if (r >= c) A[r + c * lda] = S[r][c];
  }
  if (tid < NB) lg[tid] = tid < kb ? log(S[tid][tid]) : 0.0;
  __syncthreads();
  // W = D^-1 V
  for (int idx = tid; idx < NB * NB; idx += DIAG_THREADS) {
    const int r = idx % NB, c = idx / NB;
    double wv = 0.0;
    if (r < kb && c <= r) wv = (r == c) ? rdiag[r] : rdiag[r] * V[r][c];
    Winv[r + c * NB] = wv;
  }
  for (int st = NB / 2; st > 0; st >>= 1) {
    if (tid < st) lg[tid] += lg[tid + st];
    __syncthreads();
  }
  if (tid == 0) *logdet_part = lg[0];
}

// The cluster for as many blocks as are resident at once (four SMs each); from there on
// SM time counts, of which the one-CTA kernel takes 66 us a block and the cluster 172.
void potrf_diag(cudaStream_t s, double *A, int kb, int64_t lda, double *Winv, double *logdet_part, int *status,
                int64_t k0, int64_t sA, int64_t sW, int64_t sL, int64_t batch) {
  KTScope kts(GPGP_KPROF_POTRF_DIAG, s, 2.0 * kb * kb * kb / 3 * (double)batch);
  const uint32_t polls = tl_wait.polls[GPGP_WAIT_DIAG];
  if (batch * DIAG_C <= device_sms())
    (polls == WAIT_POLLS ? potrf_diag_kernel<false> : potrf_diag_kernel<true>)<<<(unsigned)(batch * DIAG_C), DCT, 0, s>>>(
        A, kb, lda, Winv, logdet_part, status, k0, sA, sW, sL, polls);
  else
    potrf_diag_many_kernel<<<(unsigned)batch, DIAG_THREADS, 0, s>>>(A, kb, lda, Winv, logdet_part, status, k0, sA, sW,
                                                                    sL);
  GPGP_CHECK_LAUNCH();
}

}  // namespace gpgp
