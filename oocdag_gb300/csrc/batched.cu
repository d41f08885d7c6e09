// Batched factor + solve of many small SPD systems in ONE persistent launch.
//
// Thousands of uneven matrices (n in [16, 512]) are too small for the tile pipeline:
// each would be a handful of tiny launches.  Here every CTA of a persistent grid (one
// launch per size class) takes the next matrix from a queue sorted by decreasing size
// (largest first balances the tail), factors it with a blocked right-looking Cholesky
// inside the CTA, solves for its right-hand side, and moves on.  FP32 (factor_f32): the
// diagonal block factored by one warp in registers, the panel solved a row per thread in
// registers and kept transposed in shared memory, the trailing update by 32 x 32 blocks
// with a 4 x 8 register tile per lane, the forward substitution inside the factorization
// and the backward sweep on the vector in shared memory.  FP64 (factor_f64): the same steps with the
// trailing update by digit products on the tensor cores, the diagonal block by four warps.
// Per-matrix LAPACK info goes to an array; a failed matrix is skipped.  The panel width is
// chosen per size bucket by the autotuner (oocdag_gb300/autotune.py).
//
// The per-tile arithmetic restates the reference's task bodies at small n: the
// diagonal dpotrf (oocquark.cpp:87), the column dtrsm R/L/T/N (:130) and the
// dsyrk/dgemm trailing update (:176,222), followed by the dpotrs of its VERIFY block
// (oocdag.cpp:439).

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

#include "common.cuh"
#include "digits.cuh"
#include "fp64_panel.cuh"

namespace {

constexpr int BT = 256;        // threads per CTA
constexpr int NMAX = 512;      // largest matrix order supported
constexpr int NBUCKETS = 16;   // size buckets of 32: n in [32 q, 32 q + 31]

struct Item {
  void* a;    // the matrix (column-major, ld = n): A on entry, L on exit
  void* b;    // its right-hand side (overwritten by the solution)
  int n;
  int blk;    // panel width for this matrix
  int mode;   // 0: factor + solve, 1: solve with an L already in `a`
};

// sqrt(d) and its reciprocal, each within an ulp, from the approximate reciprocal root and one Newton step
// (a square root and a division are ~150 clocks of the chain, this 40); the functions themselves outside
// the range where d's square root and its square are normal.
__device__ __forceinline__ void root_f32(float d, float& sq, float& inv) {
  if (d > 0x1p-100f && d < 0x1p100f) {
    const float r = rsqrtf(d), s = d * r;
    sq = fmaf(fmaf(-s, s, d), 0.5f * r, s);
    inv = fmaf(fmaf(-sq, r, 1.f), r, r);
  } else {
    sq = sqrtf(d);
    inv = 1.f / sq;
  }
}

// v / d from ri = 1 / d rounded: one Newton step, as accurate as the division.
template <typename T>
__device__ __forceinline__ T div_by(T v, T d, T ri) {
  const T q = v * ri;
  return fma(fma(-q, d, v), ri, q);
}

// The kb x kb (kb <= 32) diagonal block at column k of the matrix, by one warp: lane r holds row r of
// D (column-major, pitch 65) in registers; the pivots pass by shuffles, column j to the other rows'
// updates through colb (two columns of 32 floats, 16-byte aligned), which the chain does not wait for.
// L_kk goes to D and the matrix, 1 / diag to rinv, and b_k := L_kk^{-1} b_k beside it (bs not null). A
// non-positive pivot is replaced by 1 so the steps stay finite; returns the first one (kb if
// none), and writes the block back only if it factored.  As loops over shared memory with a square root and a
// division per column it took 57k clocks a step, all the other warps waiting: this, whole-sector
// accesses in the trailing update and back_block's loads ahead took the kernel from 6.6 to 3.9 ms for 4000
// matrices of 16..512.
__device__ __forceinline__ int diag_f32(float* D, float* A, int n, int k, int kb, float* colb, float* rinv, float* bs,
                                        int lane) {
  float a[32];
#pragma unroll
  for (int c = 0; c < 32; c++) a[c] = (lane < kb && c <= lane) ? D[c * 65 + lane] : (c == lane ? 1.f : 0.f);
  float v = (bs && lane < kb) ? bs[k + lane] : 0.f, rv = 1.f;
  int bad = kb;
  float d = __shfl_sync(0xffffffffu, a[0], 0);
#pragma unroll
  for (int j = 0; j < 32; j++) {
    if (!(d > 0.f)) {
      bad = min(bad, j);
      d = 1.f;
    }
    float sq, inv;
    root_f32(d, sq, inv);
    const float lj = lane == j ? sq : a[j] * inv;  // L(lane, j) for lane >= j
    if (j + 1 < 32) d = __shfl_sync(0xffffffffu, fmaf(-lj, lj, a[j + 1 < 32 ? j + 1 : 0]), j + 1);
    const float y = __shfl_sync(0xffffffffu, div_by(v, sq, inv), j);
    v = lane == j ? y : lane > j ? fmaf(-lj, y, v) : v;
    if (lane == j) rv = inv;
    a[j] = lj;
    float* col = colb + (j & 1) * 32;
    col[lane] = lj;
    __syncwarp();
#pragma unroll
    for (int q = (j + 1) / 4; q < 8; q++) {  // (elements above the diagonal are never used)
      const float4 l = reinterpret_cast<const float4*>(col)[q];
      const float lc[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (4 * q + u > j) a[4 * q + u] = fmaf(-lj, lc[u], a[4 * q + u]);
    }
  }
  rinv[lane] = rv;
  if (bad == kb) {
#pragma unroll
    for (int c = 0; c < 32; c++)
      if (lane < kb && c <= lane) {
        D[c * 65 + lane] = a[c];
        A[(k + lane) + (i64)(k + c) * n] = a[c];
      }
    if (bs && lane < kb) bs[k + lane] = v;
  }
  return bad;
}

// FP32 factorization of one matrix by the CTA, in steps of BLK (16 or 32) columns:
//   1. the diagonal block is factored by one warp in registers (diag_f32), and the
//      reciprocals of its diagonal are kept; from the second step on this happens inside
//      the previous step's trailing update (warp 0 updates the block that holds it and
//      factors it while the other warps update the rest, then helps them);
//   2. every row below solves against L_kk^T, one thread per row with the row in registers,
//      right-looking (each column's FMAs independent of the others'); the result goes to
//      the matrix and, transposed, to PT (PT[c ldt + i] = L(k + kb + i, k + c)), zero-padded
//      to a multiple of 32 rows;
//   3. the trailing lower triangle is updated by 32 x 32 blocks, a warp a block, each lane a
//      4 x 8 register tile fed by shared loads of PT; the block's elements of the matrix are loaded before the products and stored after.
// The trailing matrix stays in global memory (up to 1 MB per matrix); every element of it is
// read and written once per step.
__device__ __forceinline__ void bt_block_ij(int b, int& I, int& J) {
  int i = (int)((sqrtf(8.f * (float)b + 1.f) - 1.f) * 0.5f);
  if ((i + 1) * (i + 2) / 2 <= b) i++;
  if (i * (i + 1) / 2 > b) i--;
  I = i;
  J = b - i * (i + 1) / 2;
}

template <int BLK>
__device__ int factor_f32(float* __restrict__ A, int n, float* D, float* PT, int ldt, float* bs, int* s_fail) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  float* rinv = D + 40 * 65;  // columns of D that a <= 32-wide block never uses
  float* colb = D + 44 * 65;  // (a multiple of 4)
  int* task = (int*)(D + 48 * 65);
  // a lane's elements of a 32 x 32 block: rows r0 + 8 i, so that a column's load or store is a whole
  // sector for eight lanes, columns c0 + j
  const int r0 = lane & 7, c0 = (lane >> 3) * 8;
  const int zero = n >> 30;  // n <= 512
  auto diag = [&](int k, int kb) {  // warp 0: the block already in D
    const int b = diag_f32(D, A, n, k, kb, colb, rinv, bs, lane);
    if (lane == 0) *s_fail = (b < kb) ? k + b + 1 : 0;
  };
  {
    const int kb = min(BLK, n);
    for (int idx = t; idx < kb * kb; idx += BT) {
      const int c = idx / kb, r = idx % kb;
      if (r >= c) D[c * 65 + r] = A[r + (i64)c * n];
    }
    __syncthreads();
    if (warp == 0) diag(0, kb);
    __syncthreads();
  }
  for (int k = 0; k < n; k += BLK) {
    const int kb = min(BLK, n - k);
    const int fail = *s_fail;
    if (fail) return fail;
    const int m = n - k - kb;
    if (m <= 0) break;
    const int m32 = (m + 31) & ~31;
    if (t == 0) *task = 1;
    for (int i = t; i < m32; i += BT) {
      float r[BLK];
      float* g = A + (k + kb + i);
      const bool live = i < m;
#pragma unroll
      for (int c = 0; c < BLK; c++) r[c] = (live && c < kb) ? g[(i64)(k + c) * n] : 0.f;
      float fw = 0.f;  // forward sweep: b_i -= L(i, k..) y_k (y_k sits in bs[k..])
      const float* yk = bs ? bs + k : rinv;
#pragma unroll
      for (int c = 0; c < BLK; c++) {
        r[c] *= rinv[c];
        // zero at run time: column c's loads of L_kk wait for r[c] (not all hoisted into registers)
        const int z = zero & __float_as_int(r[c]);
        const float* lc = D + c * 65 + z;
#pragma unroll
        for (int q = c + 1; q < BLK; q++) r[q] = fmaf(-r[c], lc[q], r[q]);
        const float v = (live && c < kb) ? r[c] : 0.f;
        PT[c * ldt + i] = v;
        if (live && c < kb) g[(i64)(k + c) * n] = v;
        if (c < kb) fw = fmaf(v, yk[c + z], fw);  // never reads past the vector
      }
      if (bs && live) bs[k + kb + i] -= fw;
    }
    __syncthreads();
    // Trailing update.  Warp 0 takes block (0, 0), which holds the next diagonal block: it
    // also leaves that block's kn x kn corner in D and factors it at once, while the other warps, and it
    // after that, take the other blocks in turn; the next step's row solve follows the barrier directly.
    const int nb32 = m32 >> 5, nblk = nb32 * (nb32 + 1) / 2;
    const int kn = min(BLK, m);
    float* C = A + (k + kb) + (i64)(k + kb) * n;
    auto next = [&]() {
      int x = 0;
      if (lane == 0) x = atomicAdd(task, 1);
      return __shfl_sync(0xffffffffu, x, 0);
    };
    for (int b = (warp == 0) ? 0 : next(); b < nblk; b = next()) {
      int I, J;
      bt_block_ij(b, I, J);
      const int rb = I * 32 + r0, cb = J * 32 + c0;
      float cv[4][8];
#pragma unroll
      for (int ii = 0; ii < 4; ii++)
#pragma unroll
        for (int jj = 0; jj < 8; jj++) {
          const int row = rb + 8 * ii, col = cb + jj;
          cv[ii][jj] = (row < m && col <= row) ? C[row + (i64)col * n] : 0.f;
        }
      float acc[4][8] = {};
#pragma unroll 8
      for (int q = 0; q < BLK; q++) {
        const float4 b0 = *reinterpret_cast<const float4*>(PT + q * ldt + cb);
        const float4 b1 = *reinterpret_cast<const float4*>(PT + q * ldt + cb + 4);
        const float* ar = PT + q * ldt + rb;
        const float av[4] = {ar[0], ar[8], ar[16], ar[24]};
        const float bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
        for (int ii = 0; ii < 4; ii++)
#pragma unroll
          for (int jj = 0; jj < 8; jj++) acc[ii][jj] = fmaf(av[ii], bv[jj], acc[ii][jj]);
      }
#pragma unroll
      for (int ii = 0; ii < 4; ii++)
#pragma unroll
        for (int jj = 0; jj < 8; jj++) {
          const int row = rb + 8 * ii, col = cb + jj;
          if (row < m && col <= row) {
            const float v = cv[ii][jj] - acc[ii][jj];
            C[row + (i64)col * n] = v;
            if (b == 0 && row < kn) D[col * 65 + row] = v;
          }
        }
      if (b == 0) {
        __syncwarp();
        diag(k + kb, kn);
      }
    }
    __syncthreads();
  }
  return 0;
}

// Backward sweep L^T x = y for the vector in shared memory (FP32 path; the forward sweep
// ran inside the factorization), blocks of 32 rows from the last.  Once x_K is known,
// warp 0 takes its share off the rows of block K-1 and solves that block at once (a
// 32 x 32 triangular system with shuffles), while the other warps take x_K's share off the
// rows above; one barrier per block.  Every row receives the same subtractions in the same
// order whichever warp performs them.
__device__ __forceinline__ void back_share(const float* __restrict__ L, int n, float* bs, int k, int kb, int i) {
  const float* li = L + k + (i64)i * n;  // L(k.., i): contiguous rows of column i
  float s0 = 0.f, s1 = 0.f;
#pragma unroll 8
  for (int j = 0; j + 1 < kb; j += 2) {
    s0 = fmaf(li[j], bs[k + j], s0);
    s1 = fmaf(li[j + 1], bs[k + j + 1], s1);
  }
  if (kb & 1) s0 = fmaf(li[kb - 1], bs[k + kb - 1], s0);
  bs[i] -= s0 + s1;
}

// (The block's 32 loads come first, then a chain of shuffles: with a load and a division in each step it took
// a sixth of the kernel.)
__device__ __forceinline__ void back_block(const float* __restrict__ L, int n, float* bs, int k, int lane) {
  const int kb = min(32, n - k);
  const float* l = L + k + (i64)(k + (lane < kb ? lane : 0)) * n;  // (L^T)(lane, j) = L(j, lane)
  float c[32];
#pragma unroll
  for (int j = 0; j < 32; j++) c[j] = (j < kb && lane <= j) ? l[j] : 0.f;
  float v = (lane < kb) ? bs[k + lane] : 0.f;
  const float d = (lane < kb) ? l[lane] : 1.f, ri = 1.f / d;
#pragma unroll
  for (int j = 31; j >= 0; j--) {
    const float x = __shfl_sync(0xffffffffu, div_by(v, d, ri), j);
    v = lane == j ? x : lane < j ? fmaf(-c[j], x, v) : v;
  }
  if (lane < kb) bs[k + lane] = v;
}

__device__ void solve_back_f32(const float* __restrict__ L, int n, float* bs) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int k = ((n - 1) / 32) * 32;
  if (warp == 0) back_block(L, n, bs, k, lane);
  __syncthreads();
  for (; k > 0; k -= 32) {  // x for rows k.. is final
    const int kb = min(32, n - k);
    if (warp == 0) {
      back_share(L, n, bs, k, kb, k - 32 + lane);
      __syncwarp();
      back_block(L, n, bs, k - 32, lane);
    } else {
      for (int i = t - 32; i < k - 32; i += BT - 32) back_share(L, n, bs, k, kb, i);
    }
    __syncthreads();
  }
}

// ---- FP64 ----------------------------------------------------------------------------
// One matrix by a CTA of NT threads, in steps of blk columns (8, 16 or 32; KS = K / 16 of a step's
// products).  The FP64 pipe does ~1.75 FMAs per clock per SM and was all of the time (57 % of its
// peak), so the n^3 / 6 of the trailing updates go to the tensor cores as digit products (the
// method: fp64_tc.cu):
//   1. four warps factor the diagonal block (two 16-column blocks of potrf_panel), from the second
//      step on inside the previous step's trailing update, while the other warps update the rest;
//   2. every row below solves against L_kk^T, a thread per row with the row in registers; it goes to
//      the matrix and, as seven BF16 digits with one exponent per row, to shared memory (448 bytes per
//      row of 32 columns; the 64-byte rows of a digit are swizzled for ldmatrix);
//   3. the trailing lower triangle takes the products by 16 x 8 blocks, a warp a block: 34 MMAs of
//      m16n8k16 per 16 columns into the eight order sums (32 registers), put together in integers and
//      taken off the matrix with one FP64 addition per element and step.
// mma.sync, not tcgen05: a step's operands are at most 480 rows by 32 columns, written by the CTA's own
// threads, and its results are wanted in registers at once; 16 x 8 blocks keep the triangle's
// waste small at these orders.
// 1200 matrices of 16..512: 5.3 ms against 26.7 ms with FP64 FMAs (7.4 with every class in steps of 32 columns and
// no class beside another's tail).
__device__ __forceinline__ void bar_group() { asm volatile("bar.sync 1, 128;\n" ::: "memory"); }  // warps 0..3
constexpr int DP = 33;          // column pitch of the diagonal block
constexpr int F64_GROUP = 4;    // 8-column blocks per task of the trailing update

struct Shared64 {
  double D[32 * DP];            // the diagonal block, identity beyond its order
  double rinv[32];              // the reciprocals of its diagonal
  double sq[16], rs[16];
  int nfin, fail, task, idx;
};

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldsm2(uint32_t (&r)[2], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Digit planes of a step's rows: row i's 16-byte chunk c (8 columns) of digit s at s plane + row_at(i, c).
template <int KS>
__device__ __forceinline__ int row_at(int i, int c) {
  return KS == 2 ? i * 64 + ((c ^ ((i >> 1) & 3)) << 4) : i * 32 + ((c ^ ((i >> 2) & 1)) << 4);
}

// Cholesky of the diagonal block in S.D by warps 0..3 (KS = 2: kb of 32 columns; KS = 1: kb of 16, in the
// lower right corner, where the panel step has eight threads a row); S.fail gets the first bad
// pivot's 1-based index.  Then L_kk (the columns before that pivot) to the matrix, and y_k = L_kk^{-1} b_k.
template <int KS>
__device__ __forceinline__ void diag_f64(Shared64& S, double* __restrict__ A, int n, int k, int kb, double* bs) {
  constexpr int O = KS == 1 ? PB : 0, W = 16 * KS;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int fail = 0, done = W;  // columns that factored
  for (int o = O; o < O + kb; o += PB) {
    int nf = o == 0 ? potrf_panel<4, 32, DP>(S.D, 0) : potrf_panel<8, 32, DP>(S.D, PB);
    if (t == 0) S.nfin = nf;
    bar_group();
    nf = S.nfin;
    if (lane < PB && warp < 2) {
      const double d = S.D[(o + lane) * DP + o + lane];
      if (warp == 0) S.sq[lane] = lane < nf ? sqrt(d) : 1.0;
      else S.rs[lane] = lane < nf ? rsqrt(d) : 1.0;
    }
    bar_group();
    for (int i = t; i < PB * 32; i += 128) {
      const int c = i >> 5, r = i & 31;
      double* e = S.D + (o + c) * DP + r;
      if (r == o + c && c < nf) *e = S.sq[c];
      else if (r > o + c) *e *= S.rs[c];
    }
    if (t < PB) S.rinv[o - O + t] = S.rs[t];
    bar_group();
    if (nf < PB) {
      done = o - O + nf;
      fail = k + done + 1;
      break;
    }
    if (o == 0 && kb > PB) {  // the lower right 16 x 16
      for (int i = t; i < PB * PB; i += 128) {
        const int c = PB + (i >> 4), r = PB + (i & 15);
        double v = S.D[c * DP + r];
#pragma unroll
        for (int q = 0; q < PB; q++) v = fma(-S.D[q * DP + r], S.D[q * DP + c], v);
        if (r >= c) S.D[c * DP + r] = v;
      }
      bar_group();
    }
  }
  if (t == 0) S.fail = fail;
  for (int i = t; i < W * 32; i += 128) {
    const int c = i >> 5, r = i & 31;
    if (r >= c && r < kb && c < done) A[(k + r) + (i64)(k + c) * n] = S.D[(O + c) * DP + O + r];
  }
  if (warp == 0 && bs && !fail) {  // (b_k is final: every earlier step has taken its share off)
    const int l = min(lane, W - 1);
    double v = lane < kb ? bs[k + lane] : 0.0;
    const double d = S.D[(O + l) * DP + O + l], ri = 1.0 / d;
#pragma unroll 8
    for (int j = 0; j < W; j++) {
      const double y = __shfl_sync(0xffffffffu, div_by(v, d, ri), j);
      v = lane == j ? y : lane > j && lane < W ? fma(-S.D[(O + j) * DP + O + l], y, v) : v;
    }
    if (lane < kb) bs[k + lane] = v;
  }
}

// The diagonal block at column k from the matrix into S.D, by warps 0..3.
template <int KS>
__device__ __forceinline__ void load_diag_f64(Shared64& S, const double* A, int n, int k, int kb) {
  constexpr int O = KS == 1 ? PB : 0, W = 16 * KS;
  for (int i = threadIdx.x; i < W * W; i += 128) {
    const int c = i / W, r = i % W;
    S.D[(O + c) * DP + O + r] = (r >= c && r < kb) ? A[(k + r) + (i64)(k + c) * n] : (r == c ? 1.0 : 0.0);
  }
  if (KS == 2 && threadIdx.x < 32) S.rinv[threadIdx.x] = 1.0;  // (columns that no panel step reaches)
}

// An element of the product where digits do not serve: a result out of the normal range, or a row with
// an infinity or NaN (the plain sum; X: the step's first column of the trailing rows).
__device__ __noinline__ double product_special(long long V, int es, const double* X, int n, int m, int kb, int r, int c) {
  if (es <= EXP_NONFINITE / 2) return scalbn((double)V, es - 54);
  if (r >= m || c >= m) return 0.0;
  double v = 0.0;
  for (int q = 0; q < kb; q++) v = fma(X[r + (i64)q * n], X[c + (i64)q * n], v);
  return v;
}

// The 16 x 8 block at strip I and column block J of the trailing triangle (m x m at C, column pitch n).
template <int KS>
__device__ __forceinline__ void update_block(double* __restrict__ C, const double* X, int n, int m, int kb, int I, int J,
                                             uint32_t planes, int plane, const int* exps, int lane) {
  const int r0 = 16 * I + (lane >> 2), c0 = 8 * J + 2 * (lane & 3);
  double cv[4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const int r = r0 + 8 * (e >> 1), c = c0 + (e & 1);
    cv[e] = (r < m && c <= r) ? C[r + (i64)c * n] : 0.0;
  }
  float acc[NG][4];
#pragma unroll
  for (int o = 0; o < NG; o++)
#pragma unroll
    for (int e = 0; e < 4; e++) acc[o][e] = 0.f;
  const int ra = 16 * I + (lane & 15), rb = 8 * J + (lane & 7);
#pragma unroll
  for (int kk = 0; kk < KS; kk++) {
    uint32_t b[ND][2];
    const uint32_t pb = planes + row_at<KS>(rb, 2 * kk + ((lane >> 3) & 1)), pa = planes + row_at<KS>(ra, 2 * kk + (lane >> 4));
#pragma unroll
    for (int q = 0; q < ND; q++) ldsm2(b[q], pb + q * plane);
#pragma unroll
    for (int p = 0; p < ND; p++) {
      uint32_t a[4];
      ldsm4(a, pa + p * plane);
#pragma unroll
      for (int q = 0; q < ND && p + q < NG; q++) mma_bf16(acc[p + q], a, b[q]);
    }
  }
  const int er[2] = {exps[r0], exps[r0 + 8]}, ec[2] = {exps[c0], exps[c0 + 1]};
  double w[4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    uint32_t g[NG];
#pragma unroll
    for (int o = 0; o < NG; o++) g[o] = __float_as_uint(acc[o][e]);
    const long long V = digit_sum<true>(g, 1);
    bool special = false;
    w[e] = digit_value(V, er[e >> 1] + ec[e & 1], special);
    if (special) w[e] = product_special(V, er[e >> 1] + ec[e & 1], X, n, m, kb, r0 + 8 * (e >> 1), c0 + (e & 1));
  }
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const int r = r0 + 8 * (e >> 1), c = c0 + (e & 1);
    if (r < m && c <= r) C[r + (i64)c * n] = cv[e] - w[e];
  }
}

template <int NT, int KS>
__device__ int factor_f64(double* __restrict__ A, int n, int blk, Shared64& S, double* bs, uint8_t* planes, int* exps) {
  constexpr int W = 16 * KS, O = KS == 1 ? PB : 0;  // (O: the diagonal block's place in S.D)
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int zero = n >> 30;  // n <= 512
  {
    if (t < 128) {
      load_diag_f64<KS>(S, A, n, 0, min(blk, n));
      bar_group();
      diag_f64<KS>(S, A, n, 0, min(blk, n), bs);
    }
    __syncthreads();
  }
  const uint32_t pl = (uint32_t)__cvta_generic_to_shared(planes);
  for (int k = 0; k < n; k += blk) {
    if (S.fail) return S.fail;
    const int kb = min(blk, n - k), m = n - k - kb;
    if (m <= 0) break;
    const int m16 = (m + 15) & ~15, plane = m16 * (32 * KS);
    double* X = A + (k + kb) + (i64)k * n;
    if (t == 0) S.task = 0;
    for (int i = t; i < m16; i += NT) {
      const bool live = i < m;
      double r[W];
#pragma unroll
      for (int c = 0; c < W; c++) r[c] = (live && c < kb) ? X[i + (i64)c * n] : 0.0;
      double fw = 0.0;  // b_i -= L(i, k..) y_k
      const double* yk = bs ? bs + k : S.rinv;
      int be = 0;
      bool any = false;
#pragma unroll
      for (int c = 0; c < W; c++) {
        r[c] *= S.rinv[c];
        // zero at run time: column c's loads of L_kk wait for r[c] (not all hoisted into registers)
        const int z = zero & __double2loint(r[c]);
        const double* lc = S.D + (O + c) * DP + O + z;
#pragma unroll
        for (int q = c + 1; q < W; q++) r[q] = fma(-r[c], lc[q], r[q]);
        if (live && c < kb) {
          X[i + (i64)c * n] = r[c];
          fw = fma(r[c], yk[c + z], fw);
        }
        const int hi = __double2hiint(r[c]) & 0x7FFFFFFF;
        be = max(be, hi >> 20);
        any = any || (hi | __double2loint(r[c])) != 0;
      }
      if (bs && live) bs[k + kb + i] -= fw;
      const int e = any ? max(be, 1) - 1022 : 0;  // |x| < 2^e
      exps[i] = be == 0x7FF ? EXP_NONFINITE : e;
#pragma unroll
      for (int c = 0; c < W / 8; c++) {
        unsigned long long x[8];
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = digit_fixed((unsigned long long)__double_as_longlong(r[8 * c + j]), -e);
        put_digits<0>(x, planes + row_at<KS>(i, c), plane);
      }
    }
    __syncthreads();
    // Strips of 16 rows.  Warps 0..3 take strips 0 and 1 (they hold the next diagonal block) and factor it at
    // once; the others, and these four after it, take groups of up to four blocks of the later
    // strips: strips 2 j and 2 j + 1 have j + 1 groups each.
    double* C = A + (k + kb) + (i64)(k + kb) * n;
    const int ns = m16 / 16;
    if (warp < 4) {
      for (int b = warp; b < 6; b += 4) {
        const int I = b >= 2, J = b - 2 * I;
        if (I < ns) update_block<KS>(C, X, n, m, kb, I, J, pl, plane, exps, lane);
      }
      bar_group();
      const int kn = min(blk, m);
      load_diag_f64<KS>(S, A, n, k + kb, kn);
      bar_group();
      diag_f64<KS>(S, A, n, k + kb, kn, bs);
    }
    const int np = ns / 2, ntask = ns < 3 ? 0 : np * np + np - 2 + ((ns & 1) ? np + 1 : 0);
    for (;;) {
      int x = 0;
      if (lane == 0) x = atomicAdd(&S.task, 1);
      x = __shfl_sync(0xffffffffu, x, 0);
      if (x >= ntask) break;
      int j = (int)((sqrtf(4.f * (float)x + 9.f) - 1.f) * 0.5f);  // j^2 + j - 2 <= x
      if ((j + 1) * (j + 1) + (j + 1) - 2 <= x) j++;
      if (j * j + j - 2 > x) j--;
      const int rem = x - (j * j + j - 2), I = 2 * j + (rem > j), g = rem > j ? rem - j - 1 : rem;
      for (int J = F64_GROUP * g; J < min(F64_GROUP * (g + 1), 2 * (I + 1)); J++)
        update_block<KS>(C, X, n, m, kb, I, J, pl, plane, exps, lane);
    }
    __syncthreads();
  }
  return 0;
}

// Sweeps on the vector in shared memory, blocks of 32 rows: warp 0 solves the diagonal block with
// shuffles and reciprocals, then every thread takes the block's share off its rows.
template <int NT>
__device__ void solve_forward_f64(const double* __restrict__ L, int n, double* bs) {
  const int t = threadIdx.x, lane = t & 31;
  for (int k = 0; k < n; k += 32) {
    const int kb = min(32, n - k);
    if (t < 32) {
      double v = lane < kb ? bs[k + lane] : 0.0;
      const double d = lane < kb ? L[(k + lane) + (i64)(k + lane) * n] : 1.0, ri = 1.0 / d;
      const double* l = L + (k + lane) + (i64)k * n;
#pragma unroll 8
      for (int j = 0; j < 32; j++) {
        const double c = (lane > j && lane < kb) ? l[(i64)j * n] : 0.0;
        const double y = __shfl_sync(0xffffffffu, div_by(v, d, ri), j);
        v = lane == j ? y : fma(-c, y, v);
      }
      if (lane < kb) bs[k + lane] = v;
    }
    __syncthreads();
    for (int i = k + kb + t; i < n; i += NT) {
      double s0 = 0.0, s1 = 0.0;
      const double* l = L + i + (i64)k * n;
#pragma unroll 8
      for (int j = 0; j < 32; j += 2) {  // (rows below: the block is full)
        s0 = fma(l[(i64)j * n], bs[k + j], s0);
        s1 = fma(l[(i64)(j + 1) * n], bs[k + j + 1], s1);
      }
      bs[i] -= s0 + s1;
    }
    __syncthreads();
  }
}
template <int NT>
__device__ void solve_back_f64(const double* __restrict__ L, int n, double* bs) {
  const int t = threadIdx.x, lane = t & 31;
  for (int k = (n - 1) / 32 * 32; k >= 0; k -= 32) {
    const int kb = min(32, n - k);
    if (t < 32) {
      double v = lane < kb ? bs[k + lane] : 0.0;
      const double* l = L + k + (i64)(k + (lane < kb ? lane : 0)) * n;  // (L^T)(lane, j) = L(j, lane)
      const double d = lane < kb ? l[lane] : 1.0, ri = 1.0 / d;
#pragma unroll 8
      for (int j = 31; j >= 0; j--) {
        const double c = (j < kb && lane < j) ? l[j] : 0.0;
        const double x = __shfl_sync(0xffffffffu, div_by(v, d, ri), j);
        v = lane == j ? x : fma(-c, x, v);
      }
      if (lane < kb) bs[k + lane] = v;
    }
    __syncthreads();
    for (int i = t; i < k; i += NT) {
      const double* l = L + k + (i64)i * n;
      double s0 = 0.0, s1 = 0.0;
#pragma unroll 8
      for (int j = 0; j + 1 < kb; j += 2) {
        s0 = fma(l[j], bs[k + j], s0);
        s1 = fma(l[j + 1], bs[k + j + 1], s1);
      }
      if (kb & 1) s0 = fma(l[kb - 1], bs[k + kb - 1], s0);
      bs[i] -= s0 + s1;
    }
    __syncthreads();
  }
}

// Step width where the caller gives none: 16 columns need half the FP64 work of 32 in the panel's solve and
// half the shared memory, 32 fewer passes over the matrix.  Kernel ms for 16 and 32: n in 16..64 (2000 matrices) 0.31,
// 0.34; 64..128 (1000) 0.45, 0.54; 128..256 (1000) 1.75, 1.88; 256..384 (608) 2.67 (two CTAs per SM), 3.33;
// 400..512 (608) 7.78, 6.54 (one CTA either way above 448).
inline int default_blk_f64(int n) { return n <= 448 ? 16 : 32; }
constexpr size_t F64_TWO = 113 * 1024;  // shared memory that lets two CTAs share an SM

// Shared memory of a launch whose matrices have orders <= nmax: bytes of digits for rows below a
// step, their exponents, the right-hand side, Shared64.
__host__ __device__ inline size_t digit_bytes_f64(int n, int blk) {
  const int m = n > blk ? (n - blk + 15) / 16 * 16 : 0;
  return (size_t)m * ND * (blk <= 16 ? 32 : 64);
}
inline size_t smem_f64(size_t digits, int nmax) { return digits + (size_t)((nmax + 31) / 32 * 32) * 12 + sizeof(Shared64); }

// The size classes' launches do not depend on one another: each lets the next one's CTAs take the places that
// its own leave (a class's tail beside the next class), and ends after the one before it.
__device__ __forceinline__ void class_begin() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void class_end() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// A persistent CTA takes the next matrix until there are none.  128 threads and 4 CTAs per SM up to n = 128,
// 256 and 2 where the digits leave room for two CTAs, else 512 and 1: one matrix's FP64 panel solve and chains run
// beside another's products.
template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT) k_batched_f64(const Item* __restrict__ items, int count, int* info,
                                                             int* counter, int do_solve, int nmax, int digits) {
  extern __shared__ __align__(128) uint8_t smem64_raw[];
  double* bs = (double*)(smem64_raw + digits);
  int* exps = (int*)(bs + nmax);
  Shared64& S = *(Shared64*)(exps + nmax);
  class_begin();
  for (;;) {
    if (threadIdx.x == 0) S.idx = atomicAdd(counter, 1);
    __syncthreads();
    const int idx = S.idx;
    if (idx >= count) break;
    const Item it = items[idx];
    double *a = (double*)it.a, *b = (double*)it.b;
    if (do_solve)
      for (int i = threadIdx.x; i < it.n; i += NT) bs[i] = b[i];
    __syncthreads();
    int f = 0;
    if (it.mode == 0)
      f = it.blk <= 16 ? factor_f64<NT, 1>(a, it.n, it.blk, S, do_solve ? bs : nullptr, smem64_raw, exps)
                       : factor_f64<NT, 2>(a, it.n, it.blk, S, do_solve ? bs : nullptr, smem64_raw, exps);
    else if (do_solve)
      solve_forward_f64<NT>(a, it.n, bs);
    if (threadIdx.x == 0) info[idx] = f;
    if (f == 0 && do_solve) {
      solve_back_f64<NT>(a, it.n, bs);
      for (int i = threadIdx.x; i < it.n; i += NT) b[i] = bs[i];
    }
    __syncthreads();
  }
  class_end();
}

// Two resident CTAs per SM requested from the register allocator (the shared memory, sized per size
// class, lets two CTAs share an SM up to n = 256).
__global__ void __launch_bounds__(BT, 2) k_batched_f32(const Item* __restrict__ items, int count, int* info, int* counter,
                                                       int do_solve, int ldt) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  float* D = (float*)smem_raw;
  float* P = D + 64 * 65;
  __shared__ int s_idx, s_fail;
  class_begin();
  for (;;) {
    if (threadIdx.x == 0) s_idx = atomicAdd(counter, 1);
    __syncthreads();
    const int idx = s_idx;
    __syncthreads();
    if (idx >= count) break;
    const Item it = items[idx];
    float* a = (float*)it.a;
    int f = 0;
    // 16- or 32-wide steps (the autotuner's choice); the right-hand side in shared memory: the
    // forward sweep runs inside the factorization, the backward sweep after it
    float* bs = do_solve ? P + 32 * ldt : nullptr;
    if (bs) {
      for (int i = threadIdx.x; i < it.n; i += BT) bs[i] = ((const float*)it.b)[i];
      __syncthreads();
    }
    if (it.blk <= 16) f = factor_f32<16>(a, it.n, D, P, ldt, bs, &s_fail);
    else f = factor_f32<32>(a, it.n, D, P, ldt, bs, &s_fail);
    if (bs && f == 0) {
      solve_back_f32(a, it.n, bs);
      for (int i = threadIdx.x; i < it.n; i += BT) ((float*)it.b)[i] = bs[i];
    }
    if (threadIdx.x == 0) info[idx] = f;
    __syncthreads();
  }
  class_end();
}

// Scatter per-matrix info from sorted order back to the caller's order.
__global__ void k_scatter_info(const int* sorted_info, const int* order, int count, int* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) out[order[i]] = sorted_info[i];
}

// Shared memory of an FP32 launch whose matrices have orders <= nmax: the panel transposed (32 rows
// of ldt floats, ldt = nmax rounded up to 32, plus 4), the right-hand side (ldt floats), D.
inline int ldt_for(int nmax) { return (nmax + 31) / 32 * 32 + 4; }
inline size_t smem_f32(int nmax) { return (size_t)(64 * 65 + 33 * ldt_for(nmax)) * sizeof(float); }

// One size class on the stream: items [0, count) on the device, orders <= nmax.  `first`: the launch
// tables before it in the stream are its inputs, so it waits for them.
template <typename K, typename... Args>
int launch_class(K kernel, int threads, size_t smem, int nsm, int ctas_per_sm, int count, bool first, cudaStream_t s,
                 Args... args) {
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
    cudaGetLastError();
    return OOC_ERR_UNSUPPORTED;
  }
  int occ = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem);
  const int per = std::max(1, std::min(ctas_per_sm > 0 ? ctas_per_sm : occ, std::max(occ, 1)));
  const unsigned grid = (unsigned)std::max(1, std::min(count, nsm * per));
  if (first) kernel<<<grid, threads, smem, s>>>(args...);
  else OOC_CUDA_TRY(launch_pdl(kernel, dim3(grid), threads, smem, s, args...));
  return OOC_OK;
}

template <typename T>
int run_items(cudaStream_t s, int dev, std::vector<Item>& items_in, int* info_host, const int* blk_table,
              int ctas_per_sm, int do_solve, double* seconds, int (*wait)(void*, cudaStream_t), void* wait_arg,
              GrowBuf* ws);

template <typename T>
int run_batched(ooc_handle* h, int count, const int* n, const int64_t* a_off, const int64_t* b_off, T* A, T* B,
                int* info_host, const int* blk_table, int ctas_per_sm, int do_solve, double* seconds) {
  std::vector<Item> items(count);
  for (int i = 0; i < count; i++) items[i] = Item{(void*)(A + a_off[i]), (void*)(B + b_off[i]), n[i], 0, 0};
  return run_items<T>(ooc_compute_stream(h), ooc_device(h), items, info_host, blk_table, ctas_per_sm, do_solve, seconds,
                      [](void* hh, cudaStream_t st) { return ooc_wait_stream((ooc_handle*)hh, st); }, (void*)h,
                      ooc_handle_batch_ws(h));
}

// Sorts the items by decreasing order, picks each one's panel width from the table, and
// runs them in persistent launches on `s`, one per size class; info_host receives LAPACK
// info per item in the caller's order.
template <typename T>
int run_items(cudaStream_t s, int dev, std::vector<Item>& items_in, int* info_host, const int* blk_table,
              int ctas_per_sm, int do_solve, double* seconds, int (*wait)(void*, cudaStream_t), void* wait_arg,
              GrowBuf* ws) {
  const int count = (int)items_in.size();
  std::vector<int> order(count);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return items_in[x].n > items_in[y].n; });
  std::vector<Item> items(count);
  for (int i = 0; i < count; i++) {
    const int j = order[i];
    const int bucket = std::min(NBUCKETS - 1, items_in[j].n / 32);
    int blk = blk_table ? blk_table[bucket] : (sizeof(T) == 8 ? default_blk_f64(items_in[j].n) : 64);
    blk = std::max(1, std::min(blk, 32));
    blk = sizeof(T) == 4 ? (blk <= 16 ? 16 : 32) : (blk <= 8 ? 8 : blk <= 16 ? 16 : 32);  // the compiled widths
    items[i] = items_in[j];
    items[i].blk = blk;
  }
  // Size classes (orders in (0,64], (64,128], (128,256], (256,384], (384,512], FP64 448 for 384; the items
  // are sorted by decreasing order, so a class is a contiguous range): one persistent
  // launch each, its shared memory sized for the class's largest order and panel width,
  // so that the small classes fit several CTAs per SM.
  const int bounds[] = {512, sizeof(T) == 8 ? 448 : 384, 256, 128, 64};
  std::vector<std::pair<int, int>> classes;  // [first, one past the last) in sorted order
  {
    int i = 0;
    for (int ci = 0; ci < 5 && i < count; ci++) {
      const int lo = ci + 1 < 5 ? bounds[ci + 1] : 0;
      int j = i;
      while (j < count && items[j].n > lo) j++;
      if (j > i) classes.emplace_back(i, j);
      i = j;
    }
  }
  const int ncls = (int)classes.size();
  // the launch tables, in the caller's workspace (kept across calls): items, then four
  // int arrays (info, order, scattered info, one counter per class), each 256-byte aligned
  auto up = [](size_t b) { return (b + 255) / 256 * 256; };
  const size_t b_items = up(sizeof(Item) * (size_t)count), b_int = up(sizeof(int) * (size_t)count);
  int rc = ws->ensure(b_items + 3 * b_int + 256);
  Item* d_items = nullptr;
  int *d_info = nullptr, *d_order = nullptr, *d_out = nullptr, *d_counter = nullptr;
  if (!rc) {
    char* base = (char*)ws->p;
    d_items = (Item*)base;
    d_info = (int*)(base + b_items);
    d_order = (int*)(base + b_items + b_int);
    d_out = (int*)(base + b_items + 2 * b_int);
    d_counter = (int*)(base + b_items + 3 * b_int);
  }
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (!rc) {
    cudaMemcpyAsync(d_items, items.data(), sizeof(Item) * count, cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(d_order, order.data(), sizeof(int) * count, cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(d_counter, 0, sizeof(int) * 8, s);
    int nsm = 0;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    for (int ci = 0; ci < ncls && !rc; ci++) {
      const int i0 = classes[ci].first, cnt = classes[ci].second - i0;
      int cmax = 1;
      size_t digits = 0;
      for (int i = i0; i < i0 + cnt; i++) {
        cmax = std::max(cmax, items[i].n);
        if (sizeof(T) == 8) digits = std::max(digits, digit_bytes_f64(items[i].n, items[i].blk));
      }
      auto go = [&](auto kernel, int threads, size_t smem, auto... more) {
        return launch_class(kernel, threads, smem, nsm, ctas_per_sm, cnt, ci == 0, s, (const Item*)d_items + i0, cnt, d_info + i0,
                            d_counter + ci, do_solve, more...);
      };
      if constexpr (sizeof(T) == 4) {
        rc = go(k_batched_f32, BT, smem_f32(cmax), ldt_for(cmax));
      } else {
        const int nmax = (cmax + 31) / 32 * 32;
        const size_t sm = smem_f64(digits, cmax);
        rc = cmax <= 128     ? go(k_batched_f64<128>, 128, sm, nmax, (int)digits)
             : sm <= F64_TWO ? go(k_batched_f64<256>, 256, sm, nmax, (int)digits)
                             : go(k_batched_f64<512>, 512, sm, nmax, (int)digits);
      }
    }
    cudaEventRecord(e1, s);
    if (!rc) k_scatter_info<<<(count + 255) / 256, 256, 0, s>>>(d_info, d_order, count, d_out);
    cudaError_t e = cudaGetLastError();
    if (!rc && e != cudaSuccess) { ooc_set_last_error(e, "batched factor and solve", __FILE__, __LINE__); rc = OOC_ERR_CUDA; }
  }
  if (!rc) {
    cudaMemcpyAsync(info_host, d_out, sizeof(int) * count, cudaMemcpyDeviceToHost, s);
    rc = wait(wait_arg, s);
  }
  if (!rc && seconds) {
    float ms = 0;
    cudaEventElapsedTime(&ms, e0, e1);
    *seconds = ms * 1e-3;
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  return rc;
}

template <typename T>
int check_args(int count, const int* n, const int64_t* a_off, const int64_t* b_off, const T* A, const T* B,
               int* info) {
  if (count < 0) return -3;
  if (count > 0 && (!n || !a_off || !b_off)) return -4;
  if (count > 0 && (!A || !B)) return -7;
  if (!info && count > 0) return -9;
  for (int i = 0; i < count; i++)
    if (n[i] < 1 || n[i] > NMAX) return -4;
  return OOC_OK;
}

}  // namespace

// Server hook: FP64 items given by absolute device pointers (mode 0 factor+solve, 1 solve).
// `ws`: the caller's workspace for the launch tables (kept across calls).
int ooc_batched_run_ptrs(cudaStream_t s, int dev, int count, double* const* a, double* const* b, const int* n,
                         const int* mode, int* info_host, const int* blk_table, GrowBuf* ws) {
  std::vector<Item> items(count);
  for (int i = 0; i < count; i++) items[i] = Item{(void*)a[i], (void*)b[i], n[i], 0, mode[i]};
  return run_items<double>(s, dev, items, info_host, blk_table, 0, 1, nullptr,
                           [](void*, cudaStream_t st) -> int {
                             cudaError_t e = cudaStreamSynchronize(st);
                             return e == cudaSuccess ? OOC_OK : OOC_ERR_CUDA;
                           },
                           nullptr, ws);
}

extern "C" int ooc_batched_dposv(ooc_handle* h, int count, const int* n, const int64_t* a_off, const int64_t* b_off,
                                 double* A, double* B, int* info, const int* blk_table, int ctas_per_sm,
                                 double* seconds) {
  if (!h) return -1;
  int rc = check_args<double>(count, n, a_off, b_off, A, B, info);
  if (rc) return rc;
  if (count == 0) return OOC_OK;
  cudaSetDevice(ooc_device(h));
  return run_batched<double>(h, count, n, a_off, b_off, A, B, info, blk_table, ctas_per_sm, 1, seconds);
}

extern "C" int ooc_batched_sposv(ooc_handle* h, int count, const int* n, const int64_t* a_off, const int64_t* b_off,
                                 float* A, float* B, int* info, const int* blk_table, int ctas_per_sm,
                                 double* seconds) {
  if (!h) return -1;
  int rc = check_args<float>(count, n, a_off, b_off, A, B, info);
  if (rc) return rc;
  if (count == 0) return OOC_OK;
  cudaSetDevice(ooc_device(h));
  return run_batched<float>(h, count, n, a_off, b_off, A, B, info, blk_table, ctas_per_sm, 1, seconds);
}
