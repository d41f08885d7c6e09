// FP32 trailing updates on the tensor cores: digit products, as for
// FP64 (fp64_tc.cu, where the method is described), with four balanced base-256 digits.
//
// With |x(i, k)| < 2^e(i) over a run of at most 256 columns, x(i, k) ~ 2^(e(i) - 31) X with X of 32 bits:
// the 24 bits of any element within 2^-7 of the row's largest are kept whole, smaller ones are
// rounded at 2^-32 of the scale.  Digit products of orders 0..3 (10 of 16) are summed exactly (4
// pairs x 256 x 2^14 = 2^24); what is dropped stays below 2^-28 of 2^(e(i) + e(j)).  The four sums
// are put together in FP32, so a run costs about one rounding of its value where a chain of
// FP32 FMAs rounds at each of its terms.
//
// An element whose row or column holds an infinity or NaN takes the plain FP32 sum.
//
// Only the update: its operand's rows carry one scale each (|l(i, k)| <= sqrt(a(i, i))).  A column solve
// as a product with L_jj^{-1} is scaled along k as well, and a graded matrix lost its small
// elements there to one exponent per row; it stays on the FP32 pipe.

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "fp32_tc.cuh"
#include "tc_ptx.cuh"

namespace {

constexpr int FD = 4;                          // digits per element = product orders kept
constexpr int FR = 128;                        // rows per plane unit and block (square)
constexpr int FKS = 32;                        // K per stage
constexpr int FRUN = 8;                        // stages per run: K <= 256
constexpr int F_DIG = FR * FKS * 2;            // 8 KB: one digit of 128 rows x 32 columns
constexpr int F_UNIT = FD * F_DIG;             // 32 KB
constexpr int F_STAGE = 2 * F_UNIT;            // A and B
constexpr int F_STAGES = 3;
constexpr int F_EPI_WARPS = 8;                 // two per TMEM lane quadrant, 64 columns each
constexpr int F_THREADS = 64 + 32 * F_EPI_WARPS;
constexpr int F_SMEM = F_STAGES * F_STAGE + 1024 + 256;
constexpr int F_NONFINITE = 1 << 20;
static_assert(FD * FR == 512, "the four order sums fill the TMEM");

struct Op32 {
  const uint8_t* planes;
  const int* exps;  // [run][padded rows]
  const float* X;
  i64 ldx;
  int rows, pad;
  int nst, K;       // stages of 32 and columns in all
};

// CTA: 32 rows x one run; thread (row, stage of 32 columns).
__global__ void __launch_bounds__(256) k_digits32(const Op32 o, uint8_t* __restrict__ planes, int* __restrict__ exps,
                                                  const int* status) {
  // (one answer for the CTA: the next diagonal tile beside this kernel may set it)
  if (__syncthreads_or(status ? *(volatile const int*)status : 0)) return;
  __shared__ int smax[FRUN][32];
  const int rl = threadIdx.x & 31, cg = threadIdx.x >> 5;
  const int row = blockIdx.x * 32 + rl, run = blockIdx.y;
  const int st = run * FRUN + cg, k0 = st * FKS;  // the thread's stage and first column
  const bool live = row < o.rows;
  uint32_t v[FKS];
  int bmax = 0;
#pragma unroll
  for (int k = 0; k < FKS; k++) v[k] = (live && k0 + k < o.K) ? __float_as_uint(o.X[row + (i64)(k0 + k) * o.ldx]) : 0u;
#pragma unroll
  for (int k = 0; k < FKS; k++) bmax = max(bmax, (int)((v[k] >> 23) & 0xFF));
  smax[cg][rl] = bmax;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < FRUN; q++) bmax = max(bmax, smax[q][rl]);
  bool any = false;  // a row of zeros has scale 1 (any scale does), a subnormal one 2^-125
#pragma unroll
  for (int k = 0; k < FKS; k++) any = any || (v[k] & 0x7FFFFFFFu) != 0;
  // (a barrier, so every thread of the CTA takes it: rows of zeros, padding among them, share warps with others)
  const bool subnormal = __syncthreads_or(any && bmax == 0 ? 1 : 0);
  const int e = bmax == 0 && !subnormal ? 0 : max(bmax, 1) - 126;  // |x| < 2^e
  if (cg == 0) exps[(i64)run * o.pad + row] = bmax == 0xFF ? F_NONFINITE : e;
  const int swz = (row >> 1) & 3;
  {
    if (st >= o.nst) return;
    uint8_t* base = planes + ((i64)(row >> 7) * o.nst + st) * F_UNIT + (row & 127) * 64;
#pragma unroll
    for (int c = 0; c < 4; c++) {
      int x[8];
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const uint32_t b = v[8 * c + j];
        const int be = (int)((b >> 23) & 0xFF);
        uint32_t m = b & 0x7FFFFFu;
        if (be) m |= 0x800000u;
        const int sh = max(be, 1) - 119 - e;  // X = m 2^sh, sh <= 7
        if (sh >= 0) m <<= min(sh, 7);
        else m = sh < -25 ? 0u : (m + (1u << (-sh - 1))) >> (-sh);
        x[j] = (b >> 31) ? -(int)m : (int)m;
      }
#pragma unroll
      for (int s = FD - 1; s >= 0; s--) {
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          int d0 = x[j], d1 = x[j + 1];
          if (s > 0) {  // the sign-extended low byte; the carry goes into the rest
            d0 = (int)(signed char)(x[j] & 255);
            d1 = (int)(signed char)(x[j + 1] & 255);
            x[j] = (x[j] >> 8) + (d0 < 0);
            x[j + 1] = (x[j + 1] >> 8) + (d1 < 0);
          }
          w[j / 2] = (__float_as_uint((float)d0) >> 16) | (__float_as_uint((float)d1) & 0xFFFF0000u);
        }
        *reinterpret_cast<uint4*>(base + s * F_DIG + ((c ^ swz) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
}

constexpr uint32_t IDESC_F =
    (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(FR >> 3) << 17) | ((uint32_t)(FR >> 4) << 24);

// 2^E times v (E anywhere; the result rounds once).
__device__ __forceinline__ float scale2(float v, int E) {
  if (E >= -126 && E <= 127) return v * __int_as_float((E + 127) << 23);
  return scalbnf(v, E);
}
__device__ __noinline__ float plain_sum(const Op32& A, int run, int r, int c) {
  float v = 0.f;
  const int k1 = min(A.K, (run + 1) * FRUN * FKS);
  for (int k = run * FRUN * FKS; k < k1; k++) v = fmaf(A.X[r + (i64)k * A.ldx], A.X[c + (i64)k * A.ldx], v);
  return v;
}

// Blocks of 128 x 128, persistent: warp 0 loads (two 32 KB bulk copies per stage of K = 32), warp 1
// issues 10 MMAs (M = N = 128) per K = 16, warps 2..9 take the four sums out of TMEM and
// update C while the next block's MMAs run.
// A trailing matrix of 5,745 rows with K = 256 takes 21 us for its first 256 columns and 77 us for
// the rest (110 TFLOP/s of FP32 work), after 8 us of digits; k_syrk_f32 took 48 and 268.
__global__ void __launch_bounds__(F_THREADS, 1)
    k_digit32(const __grid_constant__ Op32 X, float* __restrict__ C, i64 ldc, int T, int bj_lo, int bj_hi, i64 nblk,
              int* status) {
  if (__syncthreads_or(*(volatile int*)status)) return;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + F_STAGES * F_STAGE);
  uint64_t* empty = full + F_STAGES;
  uint64_t* tfull = empty + F_STAGES;
  uint64_t* tempty = tfull + 1;
  uint64_t* done = tempty + 1;
  uint32_t* tmem_slot = (uint32_t*)(done + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
  volatile long long* n_issued = (volatile long long*)(tmem_slot + 2);
  volatile long long* n_consumed = n_issued + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < F_STAGES; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, F_EPI_WARPS);
    mbar_init(done, 1);
    *abort_flag = 0;
    *n_issued = 0;
    *n_consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
  const uint32_t tmem = *tmem_slot;
  if (warp == 0) {
    if (lane == 0) {
      long long c = 0;
      bool ok = true;
      for (i64 t = blockIdx.x; ok && t < nblk; t += gridDim.x) {
        int bi, bj;
        strip_block_decode(t, T, bj_lo, bj_hi, &bi, &bj);
        for (int kc = 0; kc < X.nst; kc++, c++) {
          const int s = (int)(c % F_STAGES);
          if (!mbar_wait(&empty[s], (uint32_t)((c / F_STAGES) & 1) ^ 1u, abort_flag)) {
            ok = false;
            break;
          }
          uint8_t* st = smem + s * F_STAGE;
          mbar_expect_tx(&full[s], F_STAGE);
          bulk_load(st, X.planes + ((i64)bi * X.nst + kc) * F_UNIT, F_UNIT, &full[s]);
          bulk_load(st + F_UNIT, X.planes + ((i64)bj * X.nst + kc) * F_UNIT, F_UNIT, &full[s]);
          *n_issued = c + 1;
        }
      }
      if (!ok) *abort_flag = 1;
    }
  } else if (warp == 1) {
    if (lane == 0) {
      long long c = 0;
      int tl = 0;  // runs of all blocks
      bool ok = true;
      for (i64 t = blockIdx.x; ok && t < nblk; t += gridDim.x) {
        for (int kc = 0; kc < X.nst; kc++, c++) {
          if (kc % FRUN == 0) {
            if (!mbar_wait(tempty, (uint32_t)(tl & 1) ^ 1u, abort_flag)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
          }
          const int s = (int)(c % F_STAGES);
          if (!mbar_wait(&full[s], (uint32_t)((c / F_STAGES) & 1), abort_flag)) { ok = false; break; }
          *n_consumed = c + 1;
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
          const uint32_t a0 = smem_u32(smem + s * F_STAGE), b0 = a0 + F_UNIT;
#pragma unroll
          for (int kk = 0; kk < FKS / 16; kk++) {
#pragma unroll
            for (int p = 0; p < FD; p++)
#pragma unroll
              for (int q = 0; p + q < FD; q++) {
                const uint32_t d = tmem + (uint32_t)((p + q) * FR);
                const uint64_t da = umma_desc_sw64(a0 + p * F_DIG + kk * 32), db = umma_desc_sw64(b0 + q * F_DIG + kk * 32);
                const uint32_t acc = (kk == 0 && p == 0 && kc % FRUN == 0) ? 0u : 1u;
                if (q == 0) umma_collect<0>(IDESC_F, d, da, db, acc);
                else if (p + q + 1 < FD) umma_collect<1>(IDESC_F, d, da, db, acc);
                else umma_collect<2>(IDESC_F, d, da, db, acc);
              }
          }
          umma_commit(&empty[s]);
          if (kc % FRUN == FRUN - 1 || kc == X.nst - 1) {
            umma_commit(tfull);
            tl++;
          }
        }
      }
      if (!ok) *abort_flag = 1;
    }
  } else {
    const int quad = warp & 3;
    const int half = ((warp - 2) >> 2) * 64;
    int tl = 0;
    bool ok = true;
    for (i64 t = blockIdx.x; ok && t < nblk; t += gridDim.x) {
      int bi, bj;
      strip_block_decode(t, T, bj_lo, bj_hi, &bi, &bj);
      const int row = bi * FR + quad * 32 + lane, col0 = bj * FR + half;
      const int nrun = (X.nst + FRUN - 1) / FRUN;
      float v[64];
#pragma unroll
      for (int q = 0; q < 64; q++) v[q] = 0.f;
      for (int run = 0; run < nrun; run++, tl++) {
        const int* exps = X.exps + (i64)run * X.pad;
        const int er = X.exps[(i64)run * X.pad + row];
        const bool got = mbar_wait(tfull, (uint32_t)(tl & 1), abort_flag);
        if (!__all_sync(0xffffffffu, got)) {
          if (lane == 0) *abort_flag = 1;
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
#pragma unroll
        for (int b = 0; b < 8; b++) {
          uint32_t g[FD][8];
#pragma unroll
          for (int o = 0; o < FD; o++)
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                         : "=r"(g[o][0]), "=r"(g[o][1]), "=r"(g[o][2]), "=r"(g[o][3]), "=r"(g[o][4]), "=r"(g[o][5]),
                           "=r"(g[o][6]), "=r"(g[o][7])
                         : "r"(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(o * FR + half + 8 * b)));
          asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::);
          const int4 ea = *reinterpret_cast<const int4*>(exps + col0 + 8 * b);
          const int4 eb = *reinterpret_cast<const int4*>(exps + col0 + 8 * b + 4);
          const int ec[8] = {ea.x, ea.y, ea.z, ea.w, eb.x, eb.y, eb.z, eb.w};
          float w[8];
          bool special = false;
#pragma unroll
          for (int j = 0; j < 8; j++) {
            // sum_g G_g 2^(-8 g) in units of 2^(e(i) + e(j) - 14)
            float f = fmaf(__uint_as_float(g[3][j]), 0x1.0p-8f, __uint_as_float(g[2][j]));
            f = fmaf(f, 0x1.0p-8f, __uint_as_float(g[1][j]));
            f = fmaf(f, 0x1.0p-8f, __uint_as_float(g[0][j]));
            const int E = er + ec[j] - 14;
            special = special || E < -126 || E > 127;
            w[j] = f * __int_as_float((E + 127) << 23);
            g[0][j] = __float_as_uint(f);
          }
          if (special) {  // the ends of the exponent range, and non-finite rows
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const int E = er + ec[j] - 14, col = col0 + 8 * b + j;
              if (E < F_NONFINITE / 2) w[j] = scale2(__uint_as_float(g[0][j]), E);
              else w[j] = row < X.rows && col < X.rows ? plain_sum(X, run, row, col) : 0.f;
            }
          }
#pragma unroll
          for (int j = 0; j < 8; j++) v[8 * b + j] = run == 0 ? w[j] : v[8 * b + j] + w[j];
        }
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty);
      }
      if (!ok) break;
      if (row < X.rows) {
        const int nc = min(64, row - col0 + 1);  // r >= c
        float* p = C + row + (i64)col0 * ldc;
#pragma unroll
        for (int h = 0; h < 4; h++) {
          float cv[16];
#pragma unroll
          for (int q = 0; q < 16; q++) cv[q] = 16 * h + q < nc ? p[(i64)(16 * h + q) * ldc] : 0.f;
#pragma unroll
          for (int q = 0; q < 16; q++)
            if (16 * h + q < nc) p[(i64)(16 * h + q) * ldc] = cv[q] - v[16 * h + q];
        }
      }
    }
  }

  // ---- teardown (as in fp64_tc.cu)
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) atomicCAS(status, 0, ERR_TIMEOUT_CODE);
    if (warp == 1 && lane == 0) {
      umma_commit(done);
      (void)mbar_wait(done, 0, nullptr);
    }
    if (warp == 0 && lane == 0) {
      for (long long c = *n_consumed; c < *n_issued; c++)
        (void)mbar_wait(&full[c % F_STAGES], (uint32_t)((c / F_STAGES) & 1), nullptr);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::);
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
  }
}

int stages_of(int K) { return (K + FKS - 1) / FKS; }
int runs_of(int K) { return (stages_of(K) + FRUN - 1) / FRUN; }

Op32 op_of(const Digit32& X) {
  Op32 o{};
  o.pad = (int)((X.rows + FR - 1) / FR * FR);
  o.planes = (const uint8_t*)X.planes;
  o.exps = (const int*)(o.planes + (size_t)(o.pad / FR) * stages_of(X.K) * F_UNIT);
  o.X = X.X;
  o.ldx = X.ldx;
  o.rows = (int)X.rows;
  o.nst = stages_of(X.K);
  o.K = X.K;
  return o;
}

}  // namespace

size_t digit32_bytes(i64 rows, int K) {
  const size_t pad = (size_t)((rows + FR - 1) / FR * FR);
  return pad / FR * (size_t)stages_of(K) * F_UNIT + pad * (size_t)runs_of(K) * sizeof(int);
}

int launch_digits32(const Digit32& X, const int* status, cudaStream_t s) {
  if (X.rows <= 0 || X.K <= 0) return OOC_OK;
  if (X.rows > (1 << 30)) return OOC_ERR_INTERNAL;
  const Op32 o = op_of(X);
  k_digits32<<<dim3(o.pad / 32, runs_of(X.K)), 256, 0, s>>>(o, (uint8_t*)X.planes, const_cast<int*>(o.exps), status);
  OOC_CUDA_TRY(cudaGetLastError());
  return OOC_OK;
}

int launch_digit32_update(const Digit32& X, float* C, i64 ldc, int bj_lo, int bj_hi, int* status, cudaStream_t s,
                          int reserve_sms) {
  if (X.rows <= 0 || X.K <= 0) return OOC_OK;
  const Op32 a = op_of(X);
  const int T = a.pad / FR, hi = bj_hi < 0 ? T : std::min(bj_hi, T);
  if (bj_lo >= hi) return OOC_OK;
  const i64 nblk = ooc_lower_blocks_before(hi, T) - ooc_lower_blocks_before(bj_lo, T);
  int dev = 0, nsm = 0;
  OOC_CUDA_TRY(cudaGetDevice(&dev));
  OOC_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const i64 grid = std::max<i64>(1, std::min<i64>(nblk, std::max(1, nsm - std::max(0, reserve_sms))));
  OOC_CUDA_TRY(cudaFuncSetAttribute(k_digit32, cudaFuncAttributeMaxDynamicSharedMemorySize, F_SMEM));
  k_digit32<<<(unsigned)grid, F_THREADS, F_SMEM, s>>>(a, C, ldc, T, bj_lo, hi, nblk, status);
  OOC_CUDA_TRY(cudaGetLastError());
  return OOC_OK;
}
