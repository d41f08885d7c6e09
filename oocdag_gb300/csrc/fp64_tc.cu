// FP64 trailing updates on the tensor cores: C -= X X^T in FP64 from exact products of
// integer digits (the error-free splitting of Ozaki, Ogita, Oishi and Rump, 2012).
//
// The FP64 pipe of this part does ~1.7 FMAs per clock per SM (1.05 TFLOP/s in all), the
// BF16 tensor pipe ~1900 times as much.  So a run of at most 128 columns of X is rewritten
// row by row in fixed point: with |x(i, k)| < 2^e(i) for the row's columns,
//     x(i, k) ~ 2^(e(i) - 55) X,   X = sum_s d_s 2^(8 (6 - s)),   s = 0..6,  |d_s| <= 128,
// seven balanced base-256 digits, each exact in BF16; |x| within 2^-3 of the row's largest
// is represented exactly, anything smaller to 2^-56 of 2^e(i).  Products of digits are
// integers of at most 2^14 and the products of one order g = s + t are summed over K <= 128
// and at most 7 pairs in one FP32 TMEM accumulator: at most 2^23.8, so every sum is exact.
// Orders 0..7 are kept (34 of the 49 products).  What is dropped is below 2^-60 of
// 2^(e(i) + e(j)) per term; rounding the smaller elements of a row to 2^-56 of its scale
// costs about as much as one FP64 rounding of the largest product, and the eight sums are
// put together in a 64-bit integer and rounded to FP64 once per run, where a chain of FP64
// FMAs rounds at every term.  Scaling by rows is what suits a Cholesky factor: |l(i, k)| <=
// sqrt(a(i, i)), and the error of an updated element stays below a small multiple of
// 2^-53 sqrt(a(i, i) a(j, j)), the bound of the usual componentwise analysis.
//
// k_digits writes the digit planes in the order the MMA kernel's shared memory holds them
// (64-byte-swizzled K-major tiles of 128 rows x 32 columns), so that operands arrive by
// plain bulk copies without tensor maps; k_digit_update is the update.
//
// An element whose row or column of X holds an infinity or NaN takes the plain FP64 sum.

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "fp64_tc.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr int ND = 7;                         // digits per element
constexpr int NG = 8;                         // product orders kept
constexpr int DR = 128;                       // rows per plane unit and output block
constexpr int DC = 64;                        // columns per output block
constexpr int DK = 32;                        // K per stage
constexpr int A_DIG = DR * DK * 2;            // 8 KB: one digit of 128 rows x 32 columns
constexpr int B_DIG = DC * DK * 2;            // 4 KB
constexpr int UNIT_STAGE = ND * A_DIG;        // 56 KB: one stage of a plane unit
constexpr int D_STAGE = ND * (A_DIG + B_DIG); // 84 KB
constexpr int D_STAGES = 2;
constexpr int D_EPI_WARPS = 8;                // two per TMEM lane quadrant, 32 columns each
constexpr int D_THREADS = 64 + 32 * D_EPI_WARPS;
constexpr int D_SMEM = D_STAGES * D_STAGE + 1024 /*align*/ + 256 /*barriers*/;
constexpr int EXP_NONFINITE = 1 << 28;        // row exponent of a row with an infinity or NaN
static_assert(NG * DC == 512, "the eight order sums fill the TMEM");

// ---- digits ----------------------------------------------------------------------
// CTA: 32 rows, thread (row, half stage of 16 columns).  Two passes over the thread's
// elements: the row's largest exponent (the eight threads of a row meet in shared memory),
// then the digits, eight columns at a time.  Integer arithmetic only.  Bound by HBM/L2:
// 8 B in and 14 B out per element.
__global__ void __launch_bounds__(256) k_digits(const double* __restrict__ X, i64 ldx, i64 stride, int nb, i64 org,
                                                int rows, int Kall, uint8_t* __restrict__ planes, size_t slot,
                                                const int* status) {
  pdl_wait();
  if (status && *(volatile const int*)status) return;
  const int K = min(DIGIT_K, Kall - (int)blockIdx.y * DIGIT_K);  // blockIdx.y: run
  const int nst = (K + DK - 1) / DK;
  X += (i64)blockIdx.y * DIGIT_K * ldx;
  planes += (size_t)blockIdx.y * slot;
  int* exps = reinterpret_cast<int*>(planes + (size_t)(gridDim.x / 4) * nst * UNIT_STAGE);
  constexpr int KT = DK / 2;  // columns per thread
  __shared__ int smax[8][32];
  const int rl = threadIdx.x & 31, cg = threadIdx.x >> 5, st = cg >> 1;
  const int row = blockIdx.x * 32 + rl;
  const bool live = row < rows && st < nst;
  const i64 r = org + (row < rows ? row : 0);
  const double* p = X + (r / nb) * stride + (r % nb) + (i64)cg * KT * ldx;
  const int kn = min(KT, K - cg * KT);
  unsigned long long v[KT];
  int bmax = 0;
#pragma unroll
  for (int k = 0; k < KT; k++) {
    v[k] = (live && k < kn) ? (unsigned long long)__double_as_longlong(p[(i64)k * ldx]) : 0ull;
  }
#pragma unroll
  for (int k = 0; k < KT; k++) bmax = max(bmax, (int)((v[k] >> 52) & 0x7FF));
  smax[cg][rl] = bmax;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; q++) bmax = max(bmax, smax[q][rl]);
  const int e = max(bmax, 1) - 1022;  // |x| < 2^e
  if (cg == 0) exps[row] = bmax == 0x7FF ? EXP_NONFINITE : e;
  if (st >= nst) return;
  uint8_t* base = planes + ((i64)(row >> 7) * nst + st) * UNIT_STAGE + (row & 127) * 64;
  const int swz = (row >> 1) & 3;  // 64-byte swizzle: 16-byte chunk c of a row sits at c ^ ((row / 2) % 4)
#pragma unroll
  for (int c = 0; c < 2; c++) {
    long long x[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const unsigned long long b = v[8 * c + j];
      const int be = (int)((b >> 52) & 0x7FF);
      unsigned long long m = b & 0xFFFFFFFFFFFFFull;
      if (be) m |= 1ull << 52;
      const int sh = max(be, 1) - 1020 - e;  // X = m 2^sh, sh <= 2
      if (sh >= 0) m <<= min(sh, 2);
      else m = sh < -55 ? 0ull : (m + (1ull << (-sh - 1))) >> (-sh);
      x[j] = (b >> 63) ? -(long long)m : (long long)m;
    }
#pragma unroll
    for (int s = ND - 1; s >= 0; s--) {
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        int d0, d1;
        if (s > 0) {
          d0 = (int)((x[j] + 128) & 255) - 128;
          d1 = (int)((x[j + 1] + 128) & 255) - 128;
          x[j] = (x[j] - d0) >> 8;
          x[j + 1] = (x[j + 1] - d1) >> 8;
        } else {
          d0 = (int)x[j];
          d1 = (int)x[j + 1];
        }
        // an integer of magnitude <= 128 is exact in BF16: the upper half of its FP32 encoding
        w[j / 2] = (__float_as_uint((float)d0) >> 16) | (__float_as_uint((float)d1) & 0xFFFF0000u);
      }
      *reinterpret_cast<uint4*>(base + s * A_DIG + (((2 * (cg & 1) + c) ^ swz) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// ---- update ----------------------------------------------------------------------
// One product shape throughout: M = 128 rows, N = 64 columns, K = 16, each MMA adding into
// one order's 64 TMEM columns, so that every pair of MMAs that shares an accumulator has
// the same accumulator and shape (the pairs the tensor core keeps in issue order).
constexpr uint32_t IDESC_D =
    (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(DC >> 3) << 17) | ((uint32_t)(DR >> 4) << 24);
struct Operand {
  const uint8_t* planes[DIGIT_RUNS];  // each run's planes and row exponents, at the update's first row
  const int* exps[DIGIT_RUNS];
  const double* X;                    // the runs' elements (non-finite rows)
  i64 ldx, stride, org;
  int nb, rows;
  __device__ const double* row(int r) const {
    const i64 g = org + r;
    return X + (g / nb) * stride + g % nb;
  }
};
struct UpdateArgs {
  Operand a, b;                       // rows and columns of C
  int nst[DIGIT_RUNS];                // a run's stages of DK columns
  int nrun, K;
  double alpha, beta;                 // general products only
  int mask;
};

// The eight order sums of one element put together: sum_g G_g 2^(8 (5 - g)) as a 64-bit integer
// (|G_0| <= 2^21, so it stays below 2^62).  Orders 5..7 are added in FP32 first, to within one
// unit of order 5, 2^-54 of 2^(e(i) + e(j)): an FP64 chain over the K products errs by several
// times that.
__device__ __forceinline__ long long digit_sum(const uint32_t* g, int stride) {
  auto f = [&](int o) { return __uint_as_float(g[o * stride]); };
  const int t = __float2int_rn(fmaf(f(7), 0x1.0p-16f, fmaf(f(6), 0x1.0p-8f, f(5))));
  // |G_0| <= 2^21 and |G_1| <= 2^22: an FP32 addition of 1.5 2^23 leaves the integer in the low bits
  // (a conversion instruction issues at a quarter of the rate)
  auto small_int = [](float x) { return __float_as_int(x + 12582912.f) - 0x4B400000; };
  const int a1 = small_int(f(0)) * 256 + small_int(f(1));  // < 2^30
  const int a2 = __float2int_rn(f(2)) * 256 + __float2int_rn(f(3));  // < 2^31
  return ((long long)a1 << 32) + ((long long)a2 * 65536 + ((long long)__float2int_rn(f(4)) * 256 + t));
}
// V 2^(es - 54) rounded to FP64 (es = e(i) + e(j)), on the integer pipe and without branches:
// `special` is raised where the result needs digit_value_special.
__device__ __forceinline__ double digit_value(long long V, int es, bool& special) {
  const unsigned long long sg = (unsigned long long)(V >> 63);
  const unsigned long long a = ((unsigned long long)V ^ sg) - sg;
  const int lz = __clzll((long long)a);
  const int be = es + 1023 + 9 - lz;  // V = 1.x 2^(63 - lz)
  special = special || (a != 0 && (unsigned)(be - 1) > 2044u) || es > EXP_NONFINITE / 2;
  const unsigned long long M = a << (lz & 63);
  const unsigned long long r = (M >> 11) + ((M >> 10) & 1u) + ((unsigned long long)(uint32_t)((be - 1) << 20) << 32);
  return a == 0 ? 0.0 : __longlong_as_double((long long)(r | (sg << 63)));
}
// The same where the result is subnormal or overflows, and the plain sum for non-finite rows.
__device__ __noinline__ double digit_value_special(long long V, int es, const UpdateArgs& X, int run, int r, int c) {
  if (es <= EXP_NONFINITE / 2) return scalbn((double)V, es - 54);
  if (r >= X.a.rows || c >= X.b.rows) return 0.0;
  const double* a = X.a.row(r) + (i64)run * DIGIT_K * X.a.ldx;
  const double* b = X.b.row(c) + (i64)run * DIGIT_K * X.b.ldx;
  double v = 0.0;
  for (int k = 0; k < X.nst[run] * DK && run * DIGIT_K + k < X.K; k++)
    v = fma(a[(i64)k * X.a.ldx], b[(i64)k * X.b.ldx], v);
  return v;
}

// C(r, c) -= sum_k X(r, k) X(c, k) for c in block columns [bj_lo, bj_hi) of 64 and r >= c,
// rows and columns counted from `org` of the tile map.  Warp 0: bulk copies into a two-stage
// ring of K = 32 (84 KB a stage); warp 1: 34 MMAs per K = 16; warps 2..9: the eight order
// sums of a block are read from TMEM and put together, the TMEM is handed back, and C is
// updated while the next block's MMAs run.  Measured per block and run of 128 columns: 17.0k
// clocks of MMAs (62 per 128 x 64 x 16 product, of which the tensor pipe needs 32), 6.0k until the
// sums are out of TMEM; C overlaps with the next block.  A 4096 x 4096 lower triangle with
// K = 128 takes 99 us (21.7 TFLOP/s of FP64 work); FP64 MMAs took 3.2 ms for K = 256.
// GENERAL: C = beta C + alpha A B^T on all of C or a triangle (mask) instead, T columns of blocks.
template <bool GENERAL>
__global__ void __launch_bounds__(D_THREADS, 1)
    k_digit_update(const __grid_constant__ UpdateArgs X, TileMap Cm, int T, int bj_lo, int bj_hi, i64 nblk,
                   int* status) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + D_STAGES * D_STAGE);
  uint64_t* empty = full + D_STAGES;
  uint64_t* tfull = empty + D_STAGES;
  uint64_t* tempty = tfull + 1;
  uint64_t* done = tempty + 1;
  uint32_t* tmem_slot = (uint32_t*)(done + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  volatile long long* n_issued = (volatile long long*)(tmem_slot + 2);
  volatile long long* n_consumed = n_issued + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < D_STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, D_EPI_WARPS);
    mbar_init(done, 1);
    *abort_flag = 0;
    *n_issued = 0;
    *n_consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                 "r"(NG * DC));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
  const uint32_t tmem = *tmem_slot;
  pdl_wait();  // (the set-up above touches no other kernel's data)
  if (*(volatile int*)status) nblk = 0;
  auto block_at = [&](i64 t, int* bi, int* bj) {
    if constexpr (GENERAL) {
      *bi = (int)(t / T);
      *bj = (int)(t % T);
    } else {
      strip2_decode(t, T, bj_lo, bj_hi, bi, bj);
    }
  };

  if (warp == 0) {
    if (lane == 0) {
      long long c = 0;
      bool ok = true;
      for (i64 t = blockIdx.x; ok && t < nblk; t += gridDim.x) {
        int bi, bj;
        block_at(t, &bi, &bj);
        for (int run = 0; ok && run < X.nrun; run++) {
          const int nst = X.nst[run];
          const uint8_t* ua = X.a.planes[run] + (i64)bi * nst * UNIT_STAGE;
          const uint8_t* ub = X.b.planes[run] + (i64)(bj >> 1) * nst * UNIT_STAGE + (bj & 1) * B_DIG;
          for (int kc = 0; kc < nst; kc++, c++) {
            const int s = (int)(c % D_STAGES);
            if (!mbar_wait(&empty[s], (uint32_t)((c / D_STAGES) & 1) ^ 1u, abort_flag)) {
              ok = false;
              break;
            }
            uint8_t* st = smem + s * D_STAGE;
            mbar_expect_tx(&full[s], D_STAGE);
            bulk_load(st, ua + (i64)kc * UNIT_STAGE, UNIT_STAGE, &full[s]);
            for (int q = 0; q < ND; q++)
              bulk_load(st + UNIT_STAGE + q * B_DIG, ub + (i64)kc * UNIT_STAGE + q * A_DIG, B_DIG, &full[s]);
            *n_issued = c + 1;
          }
        }
      }
      if (!ok) *abort_flag = 1;
    }
  } else if (warp == 1) {
    if (lane == 0) {
      long long c = 0;
      int tl = 0;
      bool ok = true;
      for (i64 u = blockIdx.x * (i64)X.nrun; ok && u < nblk * X.nrun; tl++) {  // u: (block, run)
        const int nst = X.nst[tl % X.nrun];
        u += (tl % X.nrun == X.nrun - 1) ? (i64)(gridDim.x - 1) * X.nrun + 1 : 1;
        if (!mbar_wait(tempty, (uint32_t)(tl & 1) ^ 1u, abort_flag)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
        for (int kc = 0; kc < nst; kc++, c++) {
          const int s = (int)(c % D_STAGES);
          if (!mbar_wait(&full[s], (uint32_t)((c / D_STAGES) & 1), abort_flag)) { ok = false; break; }
          *n_consumed = c + 1;
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
          const uint32_t a0 = smem_u32(smem + s * D_STAGE), b0 = a0 + UNIT_STAGE;
#pragma unroll
          for (int kk = 0; kk < DK / 16; kk++) {
#pragma unroll
            for (int p = 0; p < ND; p++)
#pragma unroll
              for (int q = 0; q < ND && p + q < NG; q++) {
                // an order's first product of the block overwrites its accumulator
                const bool first = kk == 0 && (p == 0 || (p == 1 && q == ND - 1));
                const uint32_t d = tmem + (uint32_t)((p + q) * DC);
                const uint64_t da = umma_desc_sw64(a0 + p * A_DIG + kk * 32), db = umma_desc_sw64(b0 + q * B_DIG + kk * 32);
                const uint32_t acc = (first && kc == 0) ? 0u : 1u;
                if (q == 0) umma_collect<0>(IDESC_D, d, da, db, acc);
                else if (q + 1 < ND && p + q + 1 < NG) umma_collect<1>(IDESC_D, d, da, db, acc);
                else umma_collect<2>(IDESC_D, d, da, db, acc);
              }
          }
          umma_commit(&empty[s]);
        }
        if (!ok) break;
        umma_commit(tfull);
      }
      if (!ok) *abort_flag = 1;
    }
  } else {
    const int quad = warp & 3;
    const int half = ((warp - 2) >> 2) * 32;  // this warp's 32 of the block's 64 columns
    const int nb = Cm.nb;
    int tl = 0;
    bool ok = true;
    for (i64 t = blockIdx.x; ok && t < nblk; t += gridDim.x) {
      int bi, bj;
      block_at(t, &bi, &bj);
      const int row = bi * DR + quad * 32 + lane, col0 = bj * DC + half;
      double v[32];  // the runs' sum
#pragma unroll
      for (int q = 0; q < 32; q++) v[q] = 0.0;
      for (int run = 0; run < X.nrun; run++, tl++) {
        const int* exps = X.b.exps[run];
        const int er = X.a.exps[run][row];
        const bool got = mbar_wait(tfull, (uint32_t)(tl & 1), abort_flag);
        if (!__all_sync(0xffffffffu, got)) {
          if (lane == 0) *abort_flag = 1;
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
#pragma unroll
        for (int b = 0; b < 4; b++) {  // eight columns at a time
          uint32_t g[NG][8];
#pragma unroll
          for (int o = 0; o < NG; o++)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                         : "=r"(g[o][0]), "=r"(g[o][1]), "=r"(g[o][2]), "=r"(g[o][3]), "=r"(g[o][4]), "=r"(g[o][5]),
                           "=r"(g[o][6]), "=r"(g[o][7])
                         : "r"(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(o * DC + half + 8 * b)));
          asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::);
          const int4 ea = *reinterpret_cast<const int4*>(exps + col0 + 8 * b);
          const int4 eb = *reinterpret_cast<const int4*>(exps + col0 + 8 * b + 4);
          const int ec[8] = {ea.x, ea.y, ea.z, ea.w, eb.x, eb.y, eb.z, eb.w};
          bool special = false;
          double w[8];
#pragma unroll
          for (int j = 0; j < 8; j++) w[j] = digit_value(digit_sum(&g[0][j], 8), er + ec[j], special);
          if (special) {
#pragma unroll
            for (int j = 0; j < 8; j++)
              w[j] = digit_value_special(digit_sum(&g[0][j], 8), er + ec[j], X, run, row, col0 + 8 * b + j);
          }
#pragma unroll
          for (int j = 0; j < 8; j++) v[8 * b + j] = run == 0 ? w[j] : v[8 * b + j] + w[j];
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty);  // the accumulators may be overwritten now
      }
      if (!ok) break;
      if constexpr (GENERAL) {
        if (row < X.a.rows) {
          const int q0 = X.mask == 2 ? max(0, row - col0) : 0;  // columns [q0, q1) of the warp's 32
          const int q1 = min(32, X.mask == 1 ? min(row + 1, X.b.rows) - col0 : X.b.rows - col0);
          double* p = Cm.base + row + (i64)col0 * Cm.ld;
#pragma unroll
          for (int h = 0; h < 2; h++) {
            double cv[16];
#pragma unroll
            for (int q = 0; q < 16; q++)
              cv[q] = X.beta != 0.0 && 16 * h + q >= q0 && 16 * h + q < q1 ? p[(i64)(16 * h + q) * Cm.ld] : 0.0;
#pragma unroll
            for (int q = 0; q < 16; q++)
              if (16 * h + q >= q0 && 16 * h + q < q1)
                p[(i64)(16 * h + q) * Cm.ld] =
                    X.beta == 0.0 ? X.alpha * v[16 * h + q] : fma(X.alpha, v[16 * h + q], X.beta * cv[q]);
          }
        }
      } else if (row < X.a.rows) {
        const i64 r = X.a.org + row, c = X.a.org + col0;
        const i64 ti = r / nb, tj = c / nb;  // a block column lies in one tile column (64 divides nb)
        double* p = (Cm.packed ? Cm.base + packed_tile_index((int)ti, (int)tj, Cm.Ym) * (i64)nb * nb + (r - ti * nb) +
                                     (c - tj * nb) * Cm.ld
                               : Cm.base + r + c * Cm.ld);
        const int nc = min(32, row - col0 + 1);  // r >= c
#pragma unroll
        for (int h = 0; h < 2; h++) {
          double cv[16];
#pragma unroll
          for (int q = 0; q < 16; q++) cv[q] = 16 * h + q < nc ? p[(i64)(16 * h + q) * Cm.ld] : 0.0;
#pragma unroll
          for (int q = 0; q < 16; q++)
            if (16 * h + q < nc) p[(i64)(16 * h + q) * Cm.ld] = cv[q] - v[16 * h + q];
        }
      }
    }
  }

  // ---- teardown
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) atomicCAS(status, 0, ERR_TIMEOUT_CODE);
    if (warp == 1 && lane == 0) {
      umma_commit(done);  // fires once every MMA this thread issued has completed
      (void)mbar_wait(done, 0, nullptr);
    }
    if (warp == 0 && lane == 0) {  // let copies in flight land (bounded) before the shared memory goes away
      for (long long c = *n_consumed; c < *n_issued; c++)
        (void)mbar_wait(&full[c % D_STAGES], (uint32_t)((c / D_STAGES) & 1), nullptr);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(NG * DC));
  }
}

}  // namespace

size_t digit_plane_bytes(i64 rows, int K) {
  const size_t units = (size_t)((rows + DR - 1) / DR);
  return units * (size_t)((K + DK - 1) / DK) * UNIT_STAGE + units * DR * sizeof(int);
}

int launch_digits(DigitRuns& X, const int* status, cudaStream_t s) {
  if (X.rows <= 0 || X.K <= 0) return OOC_OK;
  const int nrun = (X.K + DIGIT_K - 1) / DIGIT_K;
  if (nrun > DIGIT_RUNS || X.rows > (1 << 30)) return OOC_ERR_INTERNAL;
  for (int q = 0; q < nrun; q++) X.org_of[q] = X.org;
  OOC_CUDA_TRY(launch_pdl(k_digits, dim3(4 * (unsigned)((X.rows + DR - 1) / DR), nrun), 256, 0, s, X.X, X.ldx, X.stride,
                          X.nb, X.org, (int)X.rows, X.K, (uint8_t*)X.planes, X.slot, status));
  return OOC_OK;
}

// The runs of X as an operand whose first row is X.org.
static int operand_of(const DigitRuns& X, Operand* o, int* nst) {
  const int nrun = (X.K + DIGIT_K - 1) / DIGIT_K;
  if (nrun > DIGIT_RUNS || X.rows > (1 << 30)) return OOC_ERR_INTERNAL;
  for (int q = 0; q < nrun; q++) {
    const i64 up = X.org - X.org_of[q];
    if (up < 0 || up % DR != 0) return OOC_ERR_INTERNAL;
    const int K = std::min(DIGIT_K, X.K - q * DIGIT_K);
    const size_t units = (size_t)((X.rows + up + DR - 1) / DR);
    nst[q] = (K + DK - 1) / DK;
    const uint8_t* p = (const uint8_t*)X.planes + (size_t)q * X.slot;
    o->planes[q] = p + (size_t)(up / DR) * nst[q] * UNIT_STAGE;
    o->exps[q] = (const int*)(p + units * nst[q] * UNIT_STAGE) + up;
  }
  o->X = X.X;
  o->ldx = X.ldx;
  o->stride = X.stride;
  o->org = X.org;
  o->nb = X.nb;
  o->rows = (int)X.rows;
  return OOC_OK;
}

template <bool GENERAL>
static int launch_blocks(const UpdateArgs& a, const TileMap& C, int T, int lo, int hi, i64 nblk, int* status,
                         cudaStream_t s, int reserve_sms) {
  if (nblk <= 0) return OOC_OK;
  int dev = 0, nsm = 0;
  OOC_CUDA_TRY(cudaGetDevice(&dev));
  OOC_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  OOC_CUDA_TRY(cudaFuncSetAttribute(k_digit_update<GENERAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, D_SMEM));
  const i64 grid = std::max<i64>(1, std::min<i64>(nblk, std::max(1, nsm - std::max(0, reserve_sms))));
  OOC_CUDA_TRY(launch_pdl(k_digit_update<GENERAL>, dim3((unsigned)grid), D_THREADS, D_SMEM, s, a, C, T, lo, hi, nblk,
                          status));
  return OOC_OK;
}

int launch_digit_update(const DigitRuns& X, const TileMap& C, i64 c_lo, i64 c_hi, const int* status, cudaStream_t s,
                        int reserve_sms) {
  c_hi = std::min(c_hi, X.rows);
  if (X.rows <= 0 || X.K <= 0 || c_lo >= c_hi) return OOC_OK;
  if (!status || c_lo % DC != 0 || C.nb % DC != 0) return OOC_ERR_INTERNAL;
  UpdateArgs a{};
  int rc = operand_of(X, &a.a, a.nst);
  if (rc) return rc;
  a.b = a.a;
  a.nrun = (X.K + DIGIT_K - 1) / DIGIT_K;
  a.K = X.K;
  const int T = (int)((X.rows + DC - 1) / DC), lo = (int)(c_lo / DC), hi = (int)((c_hi + DC - 1) / DC);
  return launch_blocks<false>(a, C, T, lo, hi, count_blocks2(T, lo, hi), const_cast<int*>(status), s, reserve_sms);
}

int launch_digit_gemm(const DigitRuns& A, const DigitRuns& B, double* C, i64 ldc, double alpha, double beta, int mask,
                      int* status, cudaStream_t s) {
  if (A.rows <= 0 || B.rows <= 0 || A.K <= 0) return OOC_OK;
  if (!status || A.K != B.K) return OOC_ERR_INTERNAL;
  UpdateArgs a{};
  int rc = operand_of(A, &a.a, a.nst);
  if (!rc) rc = operand_of(B, &a.b, a.nst);
  if (rc) return rc;
  a.nrun = (A.K + DIGIT_K - 1) / DIGIT_K;
  a.K = A.K;
  a.alpha = alpha;
  a.beta = beta;
  a.mask = mask;
  const int T = (int)((B.rows + DC - 1) / DC);
  // (a triangle's blocks on the other side of the diagonal are computed and not stored)
  return launch_blocks<true>(a, TileMap{C, ldc, 0, 1, 0}, T, 0, 0, (A.rows + DR - 1) / DR * T, status, s, 0);
}
