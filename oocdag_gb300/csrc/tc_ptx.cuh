// Blackwell building blocks shared by the tensor-core translation units (tcgen05 + TMA +
// mbarrier in inline PTX): bounded mbarrier waits, TMA copies and reductions, matrix
// descriptors, and the strip order in which the update kernels walk a lower triangle.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"

namespace {

constexpr int STRIP = 16;                         // block columns per scheduling strip
constexpr long long WAIT_LIMIT = 1LL << 22;       // polls before a wait is declared stuck
constexpr int ERR_TIMEOUT_CODE = -1000003;        // status value written on a stuck wait

// --------------------------------- PTX helpers -----------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
// Bounded parity wait: true when the phase with `parity` has completed; false when the
// poll limit runs out or another role raised the CTA's abort flag.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const volatile int* abort_flag) {
  const uint32_t a = smem_u32(bar);
  for (long long i = 0; i < WAIT_LIMIT; i++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if (abort_flag && *abort_flag) return false;
  }
  return false;
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n" ::"r"(
          smem_u32(dst)),
      "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
      : "memory");
}

// C (global, FP32) += box at smem `src`, added in L2 (TMA reduction); coordinates are
// (row, column) of the box's first element, rows innermost.
__device__ __forceinline__ void tma_reduce_add_2d(const CUtensorMap* map, const void* src, int c0, int c1) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.bulk_group [%0, {%2, %3}], [%1];\n" ::"l"(
                   (uint64_t)map),
               "r"(smem_u32(src)), "r"(c0), "r"(c1)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
// the bulk groups committed so far, all but the newest N, have finished reading shared memory
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}
__device__ __forceinline__ void named_bar_sync(uint32_t id, uint32_t count) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(count) : "memory");
}
// barrier over `count` threads that also returns the AND of their predicates
__device__ __forceinline__ bool named_bar_and(uint32_t id, uint32_t count, bool p) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred a, b;\n setp.ne.u32 a, %1, 0;\n bar.red.and.pred b, %2, %3, a;\n selp.u32 %0, 1, 0, b;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)p), "r"(id), "r"(count)
      : "memory");
  return r != 0;
}

// Shared-memory matrix descriptor: K-major operand in 128-byte-swizzled atoms of
// 8 rows x 128 bytes (stride between atoms 1024 bytes).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);          // start address
  d |= (uint64_t)(16 >> 4) << 16;                   // leading byte offset (unused for SW128 K-major)
  d |= (uint64_t)(1024 >> 4) << 32;                 // stride byte offset: 8 rows x 128 B
  d |= (uint64_t)1 << 46;                           // fixed 0b001
  d |= (uint64_t)2 << 61;                           // 128-byte swizzle
  return d;
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar))
               : "memory");
}
// Shared-memory matrix descriptor for a K-major BF16 tile with the 64-byte swizzle: rows
// of 64 bytes, 8-row atoms of 512 bytes one after another along M/N.
__device__ __forceinline__ uint64_t umma_desc_sw64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);          // start address
  d |= (uint64_t)(16 >> 4) << 16;                   // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(512 >> 4) << 32;                  // stride byte offset: 8 rows x 64 B
  d |= (uint64_t)1 << 46;                           // fixed 0b001
  d |= (uint64_t)4 << 61;                           // 64-byte swizzle
  return d;
}

// One product of BF16 operands (kind::f16, instruction descriptor `idesc`).
// USE: the A operand of the previous product is still in the collector buffer (0: read it and
// keep it, 1: take it from there, 2: take it and let it go; 3: the buffer is not used).
template <int USE>
__device__ __forceinline__ void umma_collect(uint32_t idesc, uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
#define OOC_DIGIT_MMA(COLLECTOR)                                                                       \
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"                                          \
               " tcgen05.mma.cta_group::1.kind::f16" COLLECTOR " [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d), \
               "l"(da), "l"(db), "r"(idesc), "r"(accumulate))
  if constexpr (USE == 0) OOC_DIGIT_MMA(".collector::a::fill");
  else if constexpr (USE == 1) OOC_DIGIT_MMA(".collector::a::use");
  else if constexpr (USE == 2) OOC_DIGIT_MMA(".collector::a::lastuse");
  else OOC_DIGIT_MMA("");
#undef OOC_DIGIT_MMA
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Block t of the lower-triangular block range [bj_lo, bj_hi) x rows (up to T), in strip
// order: strips of STRIP block columns, and inside a strip row by row (the first rows of
// a strip form its triangle).  Same set of blocks as ooc_lower_block_decode, other order.
__device__ __forceinline__ void strip_block_decode(i64 t, int T, int bj_lo, int bj_hi, int* bi, int* bj) {
  const int Tl = T - bj_lo, Wc = bj_hi - bj_lo;
  for (int J0 = 0; J0 < Wc; J0 += STRIP) {
    const i64 w = min(STRIP, Wc - J0);
    const i64 tri = w * (w + 1) / 2;
    const i64 cnt = tri + (i64)(Tl - J0 - w) * w;
    if (t < cnt) {
      int r, c;
      if (t < tri) {
        r = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);  // t < 136: exact enough, corrected below
        while ((i64)(r + 1) * (r + 2) / 2 <= t) r++;
        while ((i64)r * (r + 1) / 2 > t) r--;
        c = (int)(t - (i64)r * (r + 1) / 2);
      } else {
        const i64 u = t - tri;
        r = (int)(w + u / w);
        c = (int)(u % w);
      }
      *bi = bj_lo + J0 + r;
      *bj = bj_lo + J0 + c;
      return;
    }
    t -= cnt;
  }
  *bi = *bj = 0;  // not reached for t < number of blocks
}

// Block t of the block columns [bj_lo, bj_hi) x row blocks bi2 (twice as high as a block column
// is wide; T rows of the block columns' width) with 2 bi2 + 1 >= bj, in strips of STRIP block columns, row by row inside a strip.
__device__ __forceinline__ void strip2_decode(i64 t, int T, int bj_lo, int bj_hi, int* bi2, int* bj) {
  const int T2 = (T + 1) / 2;
  for (int J0 = bj_lo; J0 < bj_hi; J0 += STRIP) {
    const int w = min(STRIP, bj_hi - J0);
    const int r0 = J0 / 2;
    const int a = min(w, 2 * r0 + 2 - J0);
    const int Kt = (w - a + 1) / 2;  // rows with fewer than w blocks
    const int rows = T2 - r0;
    const int kt = min(Kt, rows);
    const i64 tri_full = (i64)Kt * a + (i64)Kt * (Kt - 1);
    const i64 cnt = (i64)kt * a + (i64)kt * (kt - 1) + (i64)max(0, rows - Kt) * w;
    if (t < cnt) {
      int k, c;
      if (t < tri_full) {  // k^2 + (a-1) k <= t
        k = (int)((-(float)(a - 1) + sqrtf((float)((a - 1) * (a - 1)) + 4.f * (float)t)) * 0.5f);
        while ((i64)(k + 1) * (k + 1) + (i64)(a - 1) * (k + 1) <= t) k++;
        while ((i64)k * k + (i64)(a - 1) * k > t) k--;
        c = (int)(t - ((i64)k * k + (i64)(a - 1) * k));
      } else {
        const i64 u = t - tri_full;
        k = (int)(Kt + u / w);
        c = (int)(u % w);
      }
      *bi2 = r0 + k;
      *bj = J0 + c;
      return;
    }
    t -= cnt;
  }
  *bi2 = *bj = 0;  // not reached for t < number of blocks
}

// Number of blocks strip2_decode walks for block columns [bj_lo, bj_hi).
inline i64 count_blocks2(int T, int bj_lo, int bj_hi) {
  const int T2 = (T + 1) / 2;
  i64 total = 0;
  for (int J0 = bj_lo; J0 < bj_hi; J0 += STRIP) {
    const int w = std::min(STRIP, bj_hi - J0);
    const int r0 = J0 / 2;
    const int a = std::min(w, 2 * r0 + 2 - J0);
    const int Kt = (w - a + 1) / 2;
    const int rows = T2 - r0;
    const int kt = std::min(Kt, rows);
    total += (i64)kt * a + (i64)kt * (kt - 1) + (i64)std::max(0, rows - Kt) * w;
  }
  return total;
}

}  // namespace
