// FP64 trailing updates on the tensor cores: C -= X X^T in FP64 from products of
// integer digits (the splitting of Ozaki, Ogita, Oishi and Rump, 2012).
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
//
// Operands that are not a Cholesky factor's panels are checked first (DigitCheck).  What digits lose is
// relative to the largest elements of the two rows, what an FP64 sum loses to sum |a| |b|, which may be far less:
// operands graded along k in opposite directions, (A D)(D^-1 B), meet large with small throughout.  So k_digits notes, for
// each row and run, which elements are within 2^-5 of the row's scale 2^e, and which columns are not all zero;
// k_uneven counts.  If both rows have 5/8 of the columns that matter (not all zero in either operand) there, at
// least a quarter of these have a product of at least 2^(e(i) + e(j) - 10), so the loss, 2^-55 of 2^(e(i) + e(j)) per
// column, stays below 2^-43 of sum |a| |b| whatever the values; for uniform and normal ones it is below what an FP64
// sum rounds off.  A last run of at most 32 columns is too short to count: after a run with 64 columns that matter its
// rows have to be within a factor of 2 of that run's, whose sum is then at least 16 2^(e(i) + e(j) - 10) and its loss below 2^-42 of
// it.  Where a row fails, the FP64 pipe takes the product.
// 2^-5 and 5/8: of 128 normally distributed elements 80 % or more are that large; a row that is mostly zeros, or a
// few large elements, fails.

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "digits.cuh"
#include "fp64_tc.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr int DR = 128;                       // rows per plane unit and output block
constexpr int DC = 64;                        // columns per output block
constexpr int DK = 32;                        // K per stage
constexpr int A_DIG = DR * DK * 2;            // 8 KB: one digit of 128 rows x 32 columns
constexpr int B_DIG = DC * DK * 2;            // 4 KB
constexpr int UNIT_STAGE = ND * A_DIG;        // 56 KB: one stage of a plane unit
constexpr int D_EPI_WARPS = 8;                // two per TMEM lane quadrant, 32 columns each
constexpr int D_THREADS = 64 + 32 * D_EPI_WARPS;
enum { UPDATE, GENERAL, NARROW };              // what a kernel computes (k_digit_update)
__host__ __device__ constexpr int stage_bytes(int mode) { return UNIT_STAGE + (mode == NARROW ? 2 * ND * 16 * DK * 2 : ND * B_DIG); }
__host__ __device__ constexpr int stages(int mode) { return mode == NARROW ? 3 : 2; }
__host__ __device__ constexpr int d_smem(int mode) { return stages(mode) * stage_bytes(mode) + 1024 /*align*/ + 256 /*barriers*/; }
// Of at most 16 columns (general products): the second operand's digits lie one below the other,
// 16 rows each, between 6 x 16 and 16 rows of zeros.
constexpr int NC = 16;                        // columns
constexpr int N_SLAB = NC * DK * 2;           // 1 KB: one digit's rows, or zeros
static_assert(NG * DC == 512, "the eight order sums fill the TMEM");
static_assert(stage_bytes(NARROW) == UNIT_STAGE + 2 * ND * N_SLAB, "six slabs of zeros, the digits, one of zeros");

// ---- digits ----------------------------------------------------------------------
// CTA: 32 rows x one run of 128 columns, thread (row, 8 columns): four lanes hold a row's 32
// columns of a stage, so a warp reads eight full sectors of each column and writes 512
// contiguous bytes per digit.  Two passes over the thread's elements: the row's largest
// exponent (shuffles, then shared memory across the stages), then the digits.  Integer
// arithmetic only, two instructions a digit and half a one to pack it: with 128 added at every
// digit at once, the digits are the bytes of the sum less 128.
// 16384 x 16384 elements of a symmetric matrix: 1.17 ms (5.0 TB/s of 8 B in and 14 B out per element), where a
// thread per 16 columns that peeled the digits off one by one took 1.9 ms.
struct DigitArgs {
  const double* X;
  i64 ldx, stride, org, k0;
  int nb, rows, K, ksign, sym;
  const int* kshift;
  const int* only_if;
  DigitCheck chk;
  uint8_t* planes;
  size_t slot;
};
constexpr int WIDE_BITS = 5;   // "large": at least 2^-5 of the row's scale
constexpr int SHORT_RUN = 32;  // columns of a run that is compared with the one before it

// 1023 + the exponent of the nonzero finite element with bits b, counting a subnormal's leading zeros.
__device__ __forceinline__ int true_exponent(unsigned long long b) {
  const int be = (int)((b >> 52) & 0x7FF);
  return be ? be : 12 - __clzll((long long)(b << 12 >> 12));
}

// SHIFT: exponents moved by kshift, and symmetric operands.  CHECK: the rows' large elements and the nonzero columns
// are noted.
template <bool SHIFT, bool CHECK>
__device__ __forceinline__ void digit_rows(const DigitArgs& a, int run) {
  constexpr int KT = 8;  // columns per thread
  __shared__ int smax[DIGIT_K / DK][32];
  const int K = min(DIGIT_K, a.K - run * DIGIT_K);
  const int nst = (K + DK - 1) / DK;
  uint8_t* planes = a.planes + (size_t)run * a.slot;
  int* exps = reinterpret_cast<int*>(planes + (size_t)(gridDim.x / 4) * nst * UNIT_STAGE);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rl = 8 * (warp & 3) + (lane >> 2), ch = lane & 3, st = warp >> 2;
  const int row = blockIdx.x * 32 + rl;
  const bool live = row < a.rows;
  const uint32_t r = (uint32_t)a.org + (live ? row : 0);
  const int kc = st * DK + ch * KT;                      // the thread's first column in the run
  const i64 kb = (i64)run * DIGIT_K + kc;
  const int kn = live ? min(KT, K - kc) : 0;
  const double* p = a.X + (a.sym ? 0 : (i64)(r / (uint32_t)a.nb) * a.stride + r % (uint32_t)a.nb + kb * a.ldx);
  unsigned long long v[KT];
  int sft[SHIFT ? KT : 1];
  int bmax = -(1 << 20);  // of the nonzero elements
  bool finite = true;
#pragma unroll
  for (int k = 0; k < KT; k++) {
    const double* q = p + (i64)k * a.ldx;
    if (SHIFT && a.sym) {
      const i64 c = a.k0 + kb + k;
      q = a.X + (r >= c ? r + c * a.ldx : c + r * a.ldx);
    }
    v[k] = k < kn ? (unsigned long long)__double_as_longlong(*q) : 0ull;
    if constexpr (SHIFT) sft[k] = k < kn ? a.ksign * a.kshift[a.k0 + kb + k] : 0;
  }
#pragma unroll
  for (int k = 0; k < KT; k++) {
    const int be = (int)((v[k] >> 52) & 0x7FF);
    if (v[k] << 1) bmax = max(bmax, (CHECK ? true_exponent(v[k]) : max(be, 1)) + (SHIFT ? sft[SHIFT ? k : 0] : 0));
    finite = finite && be != 0x7FF;
  }
  if (!finite) bmax = EXP_NONFINITE;
  bmax = max(bmax, __shfl_xor_sync(0xffffffffu, bmax, 1));
  bmax = max(bmax, __shfl_xor_sync(0xffffffffu, bmax, 2));
  __syncthreads();  // (the last run's are read)
  if (ch == 0) smax[st][rl] = bmax;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < DIGIT_K / DK; q++) bmax = max(bmax, smax[q][rl]);
  const int e = bmax < -(1 << 19) ? 0 : bmax - 1022;  // |x| < 2^e (a row of zeros: any scale)
  if (st == 0 && ch == 0) exps[row] = bmax >= EXP_NONFINITE ? EXP_NONFINITE : e;
  if constexpr (CHECK) {
    uint32_t large = 0, some = 0;
    int least = bmax;
#pragma unroll
    for (int k = 0; k < KT; k++)
      if (v[k] << 1) {
        some |= 1u << (KT * ch + k);
        const int ex = true_exponent(v[k]) + (SHIFT ? sft[SHIFT ? k : 0] : 0);
        if (ex > bmax - WIDE_BITS) large |= 1u << (KT * ch + k);
        least = min(least, ex);
      }
    if (bmax >= EXP_NONFINITE) large = ~0u;  // (plain sums: nothing to lose)
    else if (bmax - least >= a.chk.least) *a.chk.wide = 1;
    large |= __shfl_xor_sync(0xffffffffu, large, 1);
    large |= __shfl_xor_sync(0xffffffffu, large, 2);
    if (ch == 0) a.chk.large[((i64)run * (gridDim.x * 32) + row) * (DIGIT_K / DK) + st] = large;
    some = __reduce_or_sync(0xffffffffu, some);
    if (lane == 0 && some) atomicOr(a.chk.cols + run * (DIGIT_K / DK) + st, some);
  }
  if (st >= nst) return;
  unsigned long long x[KT];
#pragma unroll
  for (int j = 0; j < KT; j++) {
    x[j] = digit_fixed(v[j], (SHIFT ? sft[SHIFT ? j : 0] : 0) - e);
  }
  // 64-byte swizzle: 16-byte chunk c of a row sits at c ^ ((row / 2) % 4)
  put_digits<0>(x, planes + ((i64)(row >> 7) * nst + st) * UNIT_STAGE + (row & 127) * 64 + ((ch ^ ((row >> 1) & 3)) << 4),
                A_DIG);
}
template <bool SHIFT, bool CHECK>
__global__ void __launch_bounds__(512) k_digits(const __grid_constant__ DigitArgs a, const int* status) {
  pdl_wait();
  if (status && *(volatile const int*)status) return;
  if (SHIFT && a.only_if && !*(volatile const int*)a.only_if) return;
  for (int run = blockIdx.y; run * DIGIT_K < a.K; run += gridDim.y) digit_rows<SHIFT, CHECK>(a, run);
}

// Raises *wide where a row of A or B (blockIdx.z) is too uneven in run blockIdx.y.
struct UnevenArgs {
  const uint32_t* large[2];
  const int* exps[2];  // the first run's; `step` ints to the next one's, but the last run's sit at last_exps
  size_t step[2];
  const int* last_exps[2];
  const uint32_t* cols[2];
  int rows[2], pad[2];
  int nrun, K;
  int* wide;
};
__global__ void __launch_bounds__(128) k_uneven(const __grid_constant__ UnevenArgs a) {
  pdl_wait();
  constexpr int W = DIGIT_K / DK;
  const int row = blockIdx.x * 128 + threadIdx.x, run = blockIdx.y, z = blockIdx.z;
  if (row >= a.rows[z]) return;
  auto words = [&](int q) { return reinterpret_cast<const uint4*>(a.large[z])[(i64)q * a.pad[z] + row]; };
  const uint4 l = words(run);
  if (!(l.x | l.y | l.z | l.w)) return;  // a row of zeros
  // columns of run q that are not all zero in either operand, and how many of them `w` marks
  auto count = [&](int q, const uint4& w, int* marked) {
    const uint32_t lw[W] = {w.x, w.y, w.z, w.w};
    int n = 0;
    *marked = 0;
#pragma unroll
    for (int i = 0; i < W; i++) {
      const uint32_t both = a.cols[0][q * W + i] & a.cols[1][q * W + i];
      n += __popc(both);
      *marked += __popc(lw[i] & both);
    }
    return n;
  };
  int c;
  bool ok;
  const uint4 b = run > 0 ? words(run - 1) : make_uint4(0, 0, 0, 0);
  if (run > 0 && a.K - run * DIGIT_K <= SHORT_RUN && count(run - 1, b, &c) >= DIGIT_K / 2) {
    ok = (b.x | b.y | b.z | b.w) && a.last_exps[z][row] <= a.exps[z][(run - 1) * a.step[z] + row] + 1;
    ok = ok || a.last_exps[z][row] == EXP_NONFINITE;
  } else {
    const int n = count(run, l, &c);
    ok = 8 * c >= 5 * n;
  }
  if (!ok) *a.wide = 1;
}
static_assert(DIGIT_K / DK == 4, "a row's large elements in a run: one uint4");

// ---- update ----------------------------------------------------------------------
// One product shape throughout: M = 128 rows, N = 64 columns, K = 16, each MMA adding into
// one order's 64 TMEM columns, so that every pair of MMAs that shares an accumulator has
// the same accumulator and shape (the pairs the tensor core keeps in issue order).
__host__ __device__ constexpr uint32_t idesc_of(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(DR >> 4) << 24);
}
struct Operand {
  const uint8_t* planes[DIGIT_RUNS];  // each run's planes and row exponents, at the update's first row
  const int* exps[DIGIT_RUNS];
  const double* X;                    // the runs' elements (non-finite rows)
  i64 ldx, stride, org, k0;
  int nb, rows, sym, ksign;
  const int* kshift;
  size_t slot;                        // general products: bytes from one run's planes to the next
  __device__ double at(int r, i64 k) const {
    const i64 g = org + r, c = k0 + k;
    const double v = sym ? X[g >= c ? g + c * ldx : c + g * ldx] : X[(g / nb) * stride + g % nb + k * ldx];
    return kshift ? scalbn(v, ksign * kshift[c]) : v;
  }
};
struct UpdateArgs {
  Operand a, b;                       // rows and columns of C
  int nst[DIGIT_RUNS];                // a run's stages of DK columns (general products: 4, but in the last)
  int nrun, K;
  const int* unless;                  // nothing is done where this word is not 0 (may be null)
  double alpha, beta;                 // general products only
  int mask;
};

// The same where the result is subnormal or overflows, and the plain sum for non-finite rows.
__device__ __noinline__ double digit_value_special(long long V, int es, const UpdateArgs& X, int run, int r, int c) {
  if (es <= EXP_NONFINITE / 2) return scalbn((double)V, es - 54);
  if (r >= X.a.rows || c >= X.b.rows) return 0.0;
  double v = 0.0;
  const int k1 = min(X.K, (run + 1) * DIGIT_K);
  for (int k = run * DIGIT_K; k < k1; k++) v = fma(X.a.at(r, k), X.b.at(c, k), v);
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
// NARROW: the same for C of at most 16 columns.  Products narrower than 64 columns cost what 64 do, so
// one product takes digit p of A against the 128 rows of B from digit -p on, zeros standing for the
// digits there are not: column 16 g + j of the one accumulator is order g of column j.  7 products per
// K = 16 instead of 34; two accumulators, so that one run is put together beside the next one's
// products, and three stages of 70 KB.  16384 x 16 with K = 16384 (3.8 GB of planes): 525 us
// (7.2 TB/s, all that HBM gives), 1300 us as GENERAL.
template <int MODE>
__global__ void __launch_bounds__(D_THREADS, 1)
    k_digit_update(const __grid_constant__ UpdateArgs X, TileMap Cm, int T, int bj_lo, int bj_hi, i64 nblk,
                   int* status) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  constexpr int S_BYTES = stage_bytes(MODE), S_NUM = stages(MODE);
  constexpr int S_ACC = MODE == NARROW ? 2 : 1;  // sets of order sums
  uint64_t* full = (uint64_t*)(smem + S_NUM * S_BYTES);
  uint64_t* empty = full + S_NUM;
  uint64_t* tfull = empty + S_NUM;
  uint64_t* tempty = tfull + 2;
  uint64_t* done = tempty + 2;
  uint32_t* tmem_slot = (uint32_t*)(done + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  volatile long long* n_issued = (volatile long long*)(tmem_slot + 2);
  volatile long long* n_consumed = n_issued + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S_NUM; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < S_ACC; s++) {
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], D_EPI_WARPS);
    }
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
  if constexpr (MODE == NARROW) {  // the zeros around each stage's digits (and those, until they are loaded)
    constexpr int per = 2 * ND * N_SLAB / 16;
    for (int i = threadIdx.x; i < S_NUM * per; i += D_THREADS)
      *reinterpret_cast<uint4*>(smem + i / per * S_BYTES + UNIT_STAGE + i % per * 16) = make_uint4(0, 0, 0, 0);
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
  const uint32_t tmem = *tmem_slot;
  pdl_wait();  // (the set-up above touches no other kernel's data)
  // (one answer for all roles: a kernel beside this one may set the status)
  const int skip = *(volatile int*)status | (X.unless ? *(volatile const int*)X.unless : 0);
  if (__syncthreads_or(skip)) nblk = 0;
  auto run_stages = [&](int run) {
    return MODE == UPDATE ? X.nst[run] : run + 1 < X.nrun ? DIGIT_K / DK : (X.K - run * DIGIT_K + DK - 1) / DK;
  };
  auto run_planes = [&](const Operand& o, int run) { return MODE != UPDATE ? o.planes[0] + (size_t)run * o.slot : o.planes[run]; };
  auto run_exps = [&](const Operand& o, int run) {  // (the last run of a general product has fewer stages before them)
    if constexpr (MODE == UPDATE) return o.exps[run];
    const size_t units = (size_t)((o.rows + DR - 1) / DR);
    return (const int*)(run_planes(o, run) + units * run_stages(run) * UNIT_STAGE);
  };
  auto block_at = [&](i64 t, int* bi, int* bj) {
    if constexpr (MODE != UPDATE) {
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
          const int nst = run_stages(run);
          const uint8_t* ua = run_planes(X.a, run) + (i64)bi * nst * UNIT_STAGE;
          const uint8_t* ub = run_planes(X.b, run) + (i64)(bj >> 1) * nst * UNIT_STAGE + (bj & 1) * B_DIG;
          for (int kc = 0; kc < nst; kc++, c++) {
            const int s = (int)(c % S_NUM);
            if (!mbar_wait(&empty[s], (uint32_t)((c / S_NUM) & 1) ^ 1u, abort_flag)) {
              ok = false;
              break;
            }
            uint8_t* st = smem + s * S_BYTES;
            constexpr int bb = MODE == NARROW ? N_SLAB : B_DIG;
            uint8_t* sb = st + UNIT_STAGE + (MODE == NARROW ? (ND - 1) * N_SLAB : 0);
            mbar_expect_tx(&full[s], UNIT_STAGE + ND * bb);
            bulk_load(st, ua + (i64)kc * UNIT_STAGE, UNIT_STAGE, &full[s]);
            for (int q = 0; q < ND; q++)
              bulk_load(sb + q * bb, ub + (i64)kc * UNIT_STAGE + q * A_DIG, bb, &full[s]);
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
        const int nst = run_stages(tl % X.nrun);
        u += (tl % X.nrun == X.nrun - 1) ? (i64)(gridDim.x - 1) * X.nrun + 1 : 1;
        const int set = tl % S_ACC;
        if (!mbar_wait(&tempty[set], (uint32_t)((tl / S_ACC) & 1) ^ 1u, abort_flag)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
        for (int kc = 0; kc < nst; kc++, c++) {
          const int s = (int)(c % S_NUM);
          if (!mbar_wait(&full[s], (uint32_t)((c / S_NUM) & 1), abort_flag)) { ok = false; break; }
          *n_consumed = c + 1;
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
          const uint32_t a0 = smem_u32(smem + s * S_BYTES), b0 = a0 + UNIT_STAGE;
#pragma unroll
          for (int kk = 0; kk < DK / 16; kk++) {
            if constexpr (MODE == NARROW) {
#pragma unroll
              for (int p = 0; p < ND; p++)
                umma_collect<3>(idesc_of(NG * NC), tmem + (uint32_t)(set * NG * NC),
                                umma_desc_sw64(a0 + p * A_DIG + kk * 32),
                                umma_desc_sw64(b0 + (ND - 1 - p) * N_SLAB + kk * 32), kc == 0 && kk == 0 && p == 0 ? 0u : 1u);
              continue;
            }
#pragma unroll
            for (int p = 0; p < ND; p++)
#pragma unroll
              for (int q = 0; q < ND && p + q < NG; q++) {
                // an order's first product of the block overwrites its accumulator
                const bool first = kk == 0 && (p == 0 || (p == 1 && q == ND - 1));
                const uint32_t d = tmem + (uint32_t)((p + q) * DC);
                const uint64_t da = umma_desc_sw64(a0 + p * A_DIG + kk * 32), db = umma_desc_sw64(b0 + q * B_DIG + kk * 32);
                const uint32_t acc = (first && kc == 0) ? 0u : 1u;
                if (q == 0) umma_collect<0>(idesc_of(DC), d, da, db, acc);
                else if (q + 1 < ND && p + q + 1 < NG) umma_collect<1>(idesc_of(DC), d, da, db, acc);
                else umma_collect<2>(idesc_of(DC), d, da, db, acc);
              }
          }
          umma_commit(&empty[s]);
        }
        if (!ok) break;
        umma_commit(&tfull[set]);
      }
      if (!ok) *abort_flag = 1;
    }
  } else {
    const int quad = warp & 3;
    constexpr int W = MODE == NARROW ? NC / 2 : DC / 2;  // this warp's columns of the block
    const int half = ((warp - 2) >> 2) * W;
    const int nb = Cm.nb;
    int tl = 0;
    bool ok = true;
    for (i64 t = blockIdx.x; ok && t < nblk; t += gridDim.x) {
      int bi, bj;
      block_at(t, &bi, &bj);
      const int row = bi * DR + quad * 32 + lane, col0 = bj * DC + half;
      double v[W];  // the runs' sum
#pragma unroll
      for (int q = 0; q < W; q++) v[q] = 0.0;
      for (int run = 0; run < X.nrun; run++, tl++) {
        const int* exps = run_exps(X.b, run);
        const int er = run_exps(X.a, run)[row];
        const int set = tl % S_ACC;
        const bool got = mbar_wait(&tfull[set], (uint32_t)((tl / S_ACC) & 1), abort_flag);
        if (!__all_sync(0xffffffffu, got)) {
          if (lane == 0) *abort_flag = 1;
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
#pragma unroll
        for (int b = 0; b < W / 8; b++) {  // eight columns at a time
          if (MODE != UPDATE && col0 + 8 * b >= X.b.rows) break;
          uint32_t g[NG][8];
#pragma unroll
          for (int o = 0; o < NG; o++)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                         : "=r"(g[o][0]), "=r"(g[o][1]), "=r"(g[o][2]), "=r"(g[o][3]), "=r"(g[o][4]), "=r"(g[o][5]),
                           "=r"(g[o][6]), "=r"(g[o][7])
                         : "r"(tmem + ((uint32_t)(quad * 32) << 16) +
                               (uint32_t)((set * NG + o) * (MODE == NARROW ? NC : DC) + half + 8 * b)));
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
        if (lane == 0) mbar_arrive(&tempty[set]);  // the accumulators may be overwritten now
      }
      if (!ok) break;
      if constexpr (MODE != UPDATE) {
        if (row < X.a.rows) {
          const int q0 = X.mask == 2 ? max(0, row - col0) : 0;  // columns [q0, q1) of the warp's
          const int q1 = min(W, X.mask == 1 ? min(row + 1, X.b.rows) - col0 : X.b.rows - col0);
          constexpr int H = W < 16 ? W : 16;
          double* p = Cm.base + row + (i64)col0 * Cm.ld;
#pragma unroll
          for (int h = 0; h < W / H; h++) {
            double cv[H];
#pragma unroll
            for (int q = 0; q < H; q++)
              cv[q] = X.beta != 0.0 && H * h + q >= q0 && H * h + q < q1 ? p[(i64)(H * h + q) * Cm.ld] : 0.0;
#pragma unroll
            for (int q = 0; q < H; q++)
              if (H * h + q >= q0 && H * h + q < q1)
                p[(i64)(H * h + q) * Cm.ld] =
                    X.beta == 0.0 ? X.alpha * v[H * h + q] : fma(X.alpha, v[H * h + q], X.beta * cv[q]);
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
        (void)mbar_wait(&full[c % S_NUM], (uint32_t)((c / S_NUM) & 1), nullptr);
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
  if (X.rows > (1 << 30) || nrun > 65535) return OOC_ERR_INTERNAL;
  for (int q = 0; q < std::min(nrun, DIGIT_RUNS); q++) X.org_of[q] = X.org;
  const DigitArgs a{X.X, X.ldx, X.stride, X.org, X.k0, X.sym ? 1 : X.nb, (int)X.rows, X.K, X.ksign, X.sym, X.kshift, X.only_if,
                    X.chk, (uint8_t*)X.planes, X.slot};
  const unsigned gx = 4 * (unsigned)((X.rows + DR - 1) / DR);
  // planes that are seldom rewritten: few CTAs of many runs, since 65536 that only look at the word take 0.5 ms
  const dim3 grid(gx, X.only_if ? std::min<unsigned>(nrun, std::max(1u, 2432 / gx)) : nrun);
  const bool check = X.chk.large != nullptr;
  if (X.sym && (!X.kshift || check)) return OOC_ERR_INTERNAL;
  auto* kernel = X.kshift ? (check ? k_digits<true, true> : k_digits<true, false>)
                          : (check ? k_digits<false, true> : k_digits<false, false>);
  OOC_CUDA_TRY(launch_pdl(kernel, grid, 512, 0, s, a, status));
  return OOC_OK;
}

size_t digit_check_bytes(i64 rows, int K) {
  return (size_t)((rows + DR - 1) / DR) * DR * ((K + DIGIT_K - 1) / DIGIT_K) * sizeof(uint4);
}
size_t digit_cols_bytes(int K) { return (size_t)((K + DIGIT_K - 1) / DIGIT_K) * sizeof(uint4); }

int launch_digit_check(const DigitRuns& A, const DigitRuns& B, cudaStream_t s) {
  const int nrun = (A.K + DIGIT_K - 1) / DIGIT_K;
  if (A.rows <= 0 || B.rows <= 0 || nrun <= 0) return OOC_OK;
  if (!A.chk.large || !B.chk.large || A.chk.wide != B.chk.wide || A.K != B.K || nrun > 65535) return OOC_ERR_INTERNAL;
  const bool same = A.chk.large == B.chk.large;
  UnevenArgs a{};
  for (int z = 0; z < 2; z++) {
    const DigitRuns& X = z ? B : A;
    const size_t units = (size_t)((X.rows + DR - 1) / DR);
    const int last = (X.K - (nrun - 1) * DIGIT_K + DK - 1) / DK;
    a.large[z] = X.chk.large;
    a.cols[z] = X.chk.cols;
    a.exps[z] = (const int*)((const uint8_t*)X.planes + units * (nrun > 1 ? DIGIT_K / DK : last) * UNIT_STAGE);
    a.step[z] = X.slot / sizeof(int);
    a.last_exps[z] = (const int*)((const uint8_t*)X.planes + (size_t)(nrun - 1) * X.slot + units * last * UNIT_STAGE);
    a.rows[z] = (int)X.rows;
    a.pad[z] = (int)(units * DR);
  }
  a.nrun = nrun;
  a.K = A.K;
  a.wide = A.chk.wide;
  const unsigned gx = (unsigned)((std::max(A.rows, same ? A.rows : B.rows) + 127) / 128);
  OOC_CUDA_TRY(launch_pdl(k_uneven, dim3(gx, nrun, same ? 1 : 2), 128, 0, s, a));
  return OOC_OK;
}

// The runs of X as an operand whose first row is X.org.
static int operand_of(const DigitRuns& X, Operand* o, int* nst, bool general) {
  const int nrun = (X.K + DIGIT_K - 1) / DIGIT_K;
  if ((!general && nrun > DIGIT_RUNS) || X.rows > (1 << 30)) return OOC_ERR_INTERNAL;
  for (int q = 0; q < (general ? 1 : nrun); q++) {
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
  o->k0 = X.k0;
  o->sym = X.sym;
  o->ksign = X.ksign;
  o->kshift = X.kshift;
  o->slot = X.slot;
  return OOC_OK;
}

template <int MODE>
static int launch_blocks(const UpdateArgs& a, const TileMap& C, int T, int lo, int hi, i64 nblk, int* status,
                         cudaStream_t s, int reserve_sms) {
  if (nblk <= 0) return OOC_OK;
  int dev = 0, nsm = 0;
  OOC_CUDA_TRY(cudaGetDevice(&dev));
  OOC_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  OOC_CUDA_TRY(cudaFuncSetAttribute(k_digit_update<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, d_smem(MODE)));
  const i64 grid = std::max<i64>(1, std::min<i64>(nblk, std::max(1, nsm - std::max(0, reserve_sms))));
  OOC_CUDA_TRY(launch_pdl(k_digit_update<MODE>, dim3((unsigned)grid), D_THREADS, d_smem(MODE), s, a, C, T, lo, hi, nblk,
                          status));
  return OOC_OK;
}

int launch_digit_update(const DigitRuns& X, const TileMap& C, i64 c_lo, i64 c_hi, const int* status, cudaStream_t s,
                        int reserve_sms) {
  c_hi = std::min(c_hi, X.rows);
  if (X.rows <= 0 || X.K <= 0 || c_lo >= c_hi) return OOC_OK;
  if (!status || c_lo % DC != 0 || C.nb % DC != 0) return OOC_ERR_INTERNAL;
  UpdateArgs a{};
  int rc = operand_of(X, &a.a, a.nst, false);
  if (rc) return rc;
  a.b = a.a;
  a.nrun = (X.K + DIGIT_K - 1) / DIGIT_K;
  a.K = X.K;
  a.unless = X.chk.wide;
  const int T = (int)((X.rows + DC - 1) / DC), lo = (int)(c_lo / DC), hi = (int)((c_hi + DC - 1) / DC);
  return launch_blocks<UPDATE>(a, C, T, lo, hi, count_blocks2(T, lo, hi), const_cast<int*>(status), s, reserve_sms);
}

int launch_digit_gemm(const DigitRuns& A, const DigitRuns& B, double* C, i64 ldc, double alpha, double beta, int mask,
                      int* status, cudaStream_t s) {
  if (A.rows <= 0 || B.rows <= 0 || A.K <= 0) return OOC_OK;
  if (!status || A.K != B.K) return OOC_ERR_INTERNAL;
  UpdateArgs a{};
  int rc = operand_of(A, &a.a, a.nst, true);
  if (!rc) rc = operand_of(B, &a.b, a.nst, true);
  if (rc) return rc;
  a.nrun = (A.K + DIGIT_K - 1) / DIGIT_K;
  a.K = A.K;
  a.unless = A.chk.wide;
  a.alpha = alpha;
  a.beta = beta;
  a.mask = mask;
  const int T = (int)((B.rows + DC - 1) / DC);
  // (a triangle's blocks on the other side of the diagonal are computed and not stored)
  const TileMap map{C, ldc, 0, 1, 0};
  const i64 nblk = (A.rows + DR - 1) / DR * T;
  return B.rows <= NC ? launch_blocks<NARROW>(a, map, T, 0, 0, nblk, status, s, 0)
                      : launch_blocks<GENERAL>(a, map, T, 0, 0, nblk, status, s, 0);
}
