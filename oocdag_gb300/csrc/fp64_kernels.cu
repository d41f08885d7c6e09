// FP64 tile kernels for the out-of-core Cholesky on GB300 (sm_103a).
//
// GB300 executes FP64 at about 1/1800 of its dense BF16 tensor rate: the measured
// FP64 DMMA rate is ~1.05 TFLOP/s per GPU (about two FP64 FMAs per clock per SM).  At
// that rate every FP64 tile operation is bound by the FP64 pipe, not by HBM or shared
// memory.  The large contractions therefore go to the BF16 tensor cores as digit products
// (fp64_tc.cu); here are the chain's kernels and the contraction for what digits do not take
// (tile widths that 64 does not divide, small tile calls, no room for the planes):
//   * the contraction (gemm / syrk, oocquark.cpp:130,176,222 use cuBLAS there) runs on
//     FP64 tensor-core MMAs (mma.sync m8n8k4 f64) with 64x64 output blocks per CTA,
//     16-deep K slabs double-buffered in shared memory by cp.async;
//   * the diagonal-tile factor (host dpotrf_ at oocquark.cpp:87 in the reference) and
//     the column solve (cublasDtrsm at oocquark.cpp:130) are blocked into 64-wide steps
//     so that almost all of their flops go through the same contraction kernel, with
//     only the 64x64 diagonal pieces done in shared memory.
// Every kernel reads the device status word first and returns at once when an earlier
// step has reported a non-positive-definite minor.

#include <cuda_runtime.h>
#include <math.h>

#include "common.cuh"
#include "fp64_panel.cuh"

namespace {

constexpr int BM = 64;
constexpr int BN = 64;
constexpr int BK = 16;
constexpr int PAD = 4;               // row length BM+PAD makes fragment loads conflict-free
constexpr int GEMM_THREADS = 128;    // 4 warps in a 2 x 2 arrangement, 32 x 32 each

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int src_bytes) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void dmma884(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// Loads rows [r0, r0+BMX) x columns [k0, k0+16) of the column-major operand M (rows
// valid below `rows`, columns below `kmax`) into S[k][r] (row length BMX + PAD).
template <bool VEC, int BMX = BM, int BKX = BK>
__device__ __forceinline__ void load_slab(double* S, const double* M, i64 ld, int r0, int rows,
                                          int k0, int kmax) {
  constexpr int L = BMX + PAD;
  const int t = threadIdx.x;
  if (VEC) {
#pragma unroll
    for (int it = 0; it < (BMX * BKX / 2) / GEMM_THREADS; it++) {
      int idx = t + it * GEMM_THREADS;
      int kc = idx / (BMX / 2);
      int r = (idx % (BMX / 2)) * 2;
      int gr = r0 + r, gk = k0 + kc;
      int nvalid = 0;
      if (gk < kmax) nvalid = min(max(rows - gr, 0), 2);
      const double* src = (nvalid > 0) ? (M + gr + (i64)gk * ld) : M;
      cp_async16(S + kc * L + r, src, nvalid * 8);
    }
  } else {
    for (int idx = t; idx < BMX * BKX; idx += GEMM_THREADS) {
      int kc = idx / BMX;
      int r = idx % BMX;
      int gr = r0 + r, gk = k0 + kc;
      S[kc * L + r] = (gr < rows && gk < kmax) ? M[gr + (i64)gk * ld] : 0.0;
    }
  }
}

// C[m0:m0+BMX, n0:n0+BMX] += alpha * A[m0:, 0:k] * B[n0:, 0:k]^T, restricted to the lower
// triangle (row >= column) when `lower` is set.  Four warps in a 2 x 2 arrangement, each
// (BMX/2) x (BMX/2) as (BMX/16)^2 DMMA tiles.  BMX = 32 gives four times as many CTAs for
// the same output (for launches too small to fill the GPU with 64 x 64 blocks); every
// output element takes the same DMMA steps in the same order either way.
template <bool VEC, int BMX = BM>
__device__ __forceinline__ void gemm_block(const double* __restrict__ A, i64 lda,
                                           const double* __restrict__ B, i64 ldb,
                                           double* __restrict__ C, i64 ldc, int m, int n, int k,
                                           int m0, int n0, int lower, double alpha) {
  constexpr int L = BMX + PAD;
  constexpr int BKX = BMX == 16 ? 64 : BK;  // a 16 x 16 block takes K <= 64 in one slab: one round trip
  constexpr int TI = BMX / 16;  // DMMA tiles per warp dimension
  constexpr int WT = BMX / 2;   // warp tile
  __shared__ __align__(16) double As[2][BKX * L];
  __shared__ __align__(16) double Bs[2][BKX * L];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int wm = warp & 1, wn = warp >> 1;
  const int g = lane >> 2, tig = lane & 3;

  double acc[TI][TI][2];
#pragma unroll
  for (int i = 0; i < TI; i++)
#pragma unroll
    for (int j = 0; j < TI; j++) acc[i][j][0] = acc[i][j][1] = 0.0;

  const int nslab = (k + BKX - 1) / BKX;
  if (nslab > 0) {
    load_slab<VEC, BMX, BKX>(As[0], A, lda, m0, m, 0, k);
    load_slab<VEC, BMX, BKX>(Bs[0], B, ldb, n0, n, 0, k);
    if (VEC) cp_async_commit();
  }
  for (int s = 0; s < nslab; s++) {
    const int cur = s & 1;
    if (s + 1 < nslab) {
      load_slab<VEC, BMX, BKX>(As[cur ^ 1], A, lda, m0, m, (s + 1) * BKX, k);
      load_slab<VEC, BMX, BKX>(Bs[cur ^ 1], B, ldb, n0, n, (s + 1) * BKX, k);
      if (VEC) { cp_async_commit(); cp_async_wait<1>(); }
    } else {
      if (VEC) cp_async_wait<0>();
    }
    __syncthreads();
    const double* as = As[cur];
    const double* bs = Bs[cur];
#pragma unroll 4
    for (int kk = 0; kk < BKX; kk += 4) {
      double a[TI], b[TI];
#pragma unroll
      for (int i = 0; i < TI; i++) a[i] = as[(kk + tig) * L + wm * WT + i * 8 + g];
#pragma unroll
      for (int j = 0; j < TI; j++) b[j] = bs[(kk + tig) * L + wn * WT + j * 8 + g];
#pragma unroll
      for (int i = 0; i < TI; i++)
#pragma unroll
        for (int j = 0; j < TI; j++) dmma884(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
    __syncthreads();
  }

  // Epilogue, one 8-row group at a time: its loads of C first, then its stores (a load
  // after a store to a possibly aliasing address would wait for memory each time).
#pragma unroll
  for (int i = 0; i < TI; i++) {
    const int r = m0 + wm * WT + i * 8 + g;
    double cv[TI][2];
#pragma unroll
    for (int j = 0; j < TI; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int c = n0 + wn * WT + j * 8 + 2 * tig + h;
        const bool ok = r < m && c < n && !(lower && c > r);
        cv[j][h] = ok ? C[r + (i64)c * ldc] : 0.0;
      }
#pragma unroll
    for (int j = 0; j < TI; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int c = n0 + wn * WT + j * 8 + 2 * tig + h;
        if (r < m && c < n && !(lower && c > r)) C[r + (i64)c * ldc] = fma(alpha, acc[i][j][h], cv[j][h]);
      }
  }
}

// ---------------------------------------------------------------------------------
// Panel update: every tile pair (i >= j) of a trapezoid, one launch per X column.
// grid.x = 64x64 blocks within a tile, grid.y = tile pair.
// ---------------------------------------------------------------------------------
template <bool VEC>
__global__ void __launch_bounds__(GEMM_THREADS)
k_panel_update(TileCol X, TileMap Cm, int Ht, int Kt, i64 H, i64 Kcols, int K, const int* status) {
  if (status && *(volatile const int*)status) return;
  int p = blockIdx.y;
  int j = 0;
  while (j < Kt && p >= Ht - j) { p -= Ht - j; j++; }
  if (j >= Kt) return;
  const int i = j + p;
  const int nb = Cm.nb;
  const int LM = (int)min((i64)nb, H - (i64)i * nb);
  const int LN = (int)min((i64)nb, Kcols - (i64)j * nb);
  const int mblocks = (nb + BM - 1) / BM;
  const int m0 = (blockIdx.x % mblocks) * BM;
  const int n0 = (blockIdx.x / mblocks) * BN;
  if (m0 >= LM || n0 >= LN) return;
  const int lower = (i == j);
  if (lower && n0 > m0 + BM - 1) return;
  const double* Xi = X.base + (i64)i * X.stride;
  const double* Xj = X.base + (i64)j * X.stride;
  double* Cij = tile_ptr(Cm, i, j);
  gemm_block<VEC>(Xi, X.ld, Xj, X.ld, Cij, Cm.ld, LM, LN, K, m0, n0, lower, -1.0);
}

// ---------------------------------------------------------------------------------
// Batched generic NT gemm: C_z += alpha A_z B_z^T, z = blockIdx.y; the last batch entry
// may have a different row count (m_last).
// ---------------------------------------------------------------------------------
struct GemmBatch {
  const double* A; i64 lda, sA;
  const double* B; i64 ldb, sB;
  double* C; i64 ldc, sC;
  int m, m_last, n, k, lower, batch;
  double alpha;
  int tri_b;  // B lower triangular (B(j, kk) = 0 for kk > j): skip the zero K range
};

template <bool VEC, int BMX = BM>
__global__ void __launch_bounds__(GEMM_THREADS) k_gemm_batched(GemmBatch gb, const int* status) {
  pdl_wait();
  if (status && *(volatile const int*)status) return;
  const int z = blockIdx.y;
  const int m = (z == gb.batch - 1) ? gb.m_last : gb.m;
  const int mblocks = (max(gb.m, gb.m_last) + BMX - 1) / BMX;
  const int m0 = (blockIdx.x % mblocks) * BMX;
  const int n0 = (blockIdx.x / mblocks) * BMX;
  if (m0 >= m || n0 >= gb.n) return;
  if (gb.lower && n0 > m0 + BMX - 1) return;
  const int kmax = gb.tri_b ? min(gb.k, n0 + BMX) : gb.k;
  gemm_block<VEC, BMX>(gb.A + (i64)z * gb.sA, gb.lda, gb.B + (i64)z * gb.sB, gb.ldb,
                       gb.C + (i64)z * gb.sC, gb.ldc, m, gb.n, kmax, m0, n0, gb.lower, gb.alpha);
}

// ---------------------------------------------------------------------------------
// Lower Cholesky of an n x n block (n <= 64) in shared memory, by four warps in column
// blocks of 16.  A warp-wide FP64 instruction occupies its SM sub-partition for 64 clocks
// whatever its active lanes, and an SM issues one per 19 clocks, so both the number of FP64
// instructions and the dependent chain per column count:
//   * inside a block the columns stay unscaled (a(r,j), not l(r,j)): thread (row r, half h)
//     holds every second column of its row in registers, and column j's step is
//     u = a(r,j) / d, a(r,c) -= u a(c,j), with the quotient from an FP32 reciprocal seed
//     refined by one cubic Newton step (e = 1 - d r0, a r0 (1 + e + e^2): error e^3 <
//     2^-66), four dependent FP64 instructions where a square root and a division took
//     twenty; one barrier per column;
//   * the columns to the right take the block as one rank-16 update on the FP64 MMA, from the
//     unscaled columns and the quotients;
//   * the 64 square roots and their reciprocals are taken side by side at the end.
// Measured on a 64 x 64 block: 90 us with a square root and a division per column on the
// barrier-to-barrier path, 50 us with the roots and a scaling pass per 16 columns, 46 us now.
// LAPACK convention: a pivot that is not > 0 (or is NaN) stops the factorization and reports
// info = col0 + j + 1; the columns before it are written back.
// ---------------------------------------------------------------------------------
constexpr int SB = 64;
constexpr int PT_THREADS = 128;
constexpr int SP = SB + 1;           // column pitch in shared memory

__global__ void __launch_bounds__(PT_THREADS) k_potrf_small(double* A, i64 ld, int n, i64 col0, int* status) {
  pdl_wait();
  if (*(volatile int*)status) return;
  __shared__ double S[SB * SP];       // S[c * SP + r], unscaled until the end
  __shared__ double U[PB * SP];       // a block's columns over their pivots
  __shared__ double sq[SB], rs[SB];
  __shared__ int s_nfin;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  {  // 64 rows x 2 column groups; beyond n the identity
    const int r = t & (SB - 1), cg = t >> 6;
#pragma unroll 16
    for (int i = 0; i < SB / 2; i++) {
      const int c = cg + 2 * i;
      S[c * SP + r] = (r < n && c < n) ? (r >= c ? A[r + (i64)c * ld] : 0.0) : (r == c ? 1.0 : 0.0);
    }
  }
  __syncthreads();
  const int g = lane >> 2, tig = lane & 3;
  int done = SB;  // columns that factored
  for (int k = 0; k < n; k += PB) {
    int nfin = k < 32 ? potrf_panel<2, SB, SP>(S, k, U) : k < 48 ? potrf_panel<4, SB, SP>(S, k, U) : potrf_panel<8, SB, SP>(S, k, U);
    if (t == 0) s_nfin = nfin;
    __syncthreads();
    nfin = s_nfin;
    if (nfin < PB) {
      done = k + nfin;
      if (t == 0) atomicCAS(status, 0, (int)(col0 + done + 1));
      break;
    }
    // rank-16 update of the lower triangle to the right, an 8 x 8 MMA tile per warp and turn
    const int o = k + PB, nt = (SB - o) / 8;
    for (int b = warp; b < nt * (nt + 1) / 2; b += PT_THREADS / 32) {
      int I = (int)((sqrtf(8.f * (float)b + 1.f) - 1.f) * 0.5f);
      if ((I + 1) * (I + 2) / 2 <= b) I++;
      if (I * (I + 1) / 2 > b) I--;
      const int J = b - I * (I + 1) / 2;
      const int row = o + 8 * I + g, col = o + 8 * J;
      double c0 = S[(col + 2 * tig) * SP + row], c1 = S[(col + 2 * tig + 1) * SP + row];
#pragma unroll
      for (int q = 0; q < PB; q += 4)
        dmma884(c0, c1, -U[(q + tig) * SP + row], S[(k + q + tig) * SP + col + g]);
      S[(col + 2 * tig) * SP + row] = c0;
      S[(col + 2 * tig + 1) * SP + row] = c1;
    }
    __syncthreads();
  }
  {  // every square root and its reciprocal, side by side, scale the columns on their way out
    const int c = t & (SB - 1);
    const double d = c < done ? S[c * SP + c] : 1.0;
    if (t < SB) sq[c] = sqrt(d);
    else rs[c] = rsqrt(d);
  }
  __syncthreads();
  {
    const int rr = t & (SB - 1), cg = t >> 6;
#pragma unroll 16
    for (int i = 0; i < SB / 2; i++) {
      const int c = cg + 2 * i;
      if (rr < n && c <= rr) A[rr + (i64)c * ld] = rr == c && c < done ? sq[c] : S[c * SP + rr] * rs[c];
    }
  }
}

// ---------------------------------------------------------------------------------
// B := B L^-T for a block of up to 64 columns: L is n x n lower (n <= 64), B rows are
// independent.  R rows per CTA of 128 threads, 128 / R lanes per row, each holding every
// (128/R)-th column in registers.  FP64 issues from each SM sub-partition at about one FMA
// per two clocks, so a row group must spread over the sub-partitions, and a launch with few
// rows over as many SMs as there are: R = 4 solves its rows in 12.5 us,
// R = 32 in 31 us (31 us for any row count with 32 rows a CTA only).  Right-looking: once x_c is final (computed by its owner lane and passed to the
// row's other lanes by a shuffle), every later column takes its FMA with it, in increasing c,
// as a substitution does; the same operations whatever R.  L sits in shared memory, padded
// to 64 with the identity, and is read by broadcast; x_c = v * (1 / L(c,c)).
// Row i of the m rows sits at B + ((org + i) / nb) * sB + (org + i) % nb (a column of tiles of
// nb rows).  z = blockIdx.y walks a batch of independent systems: L + z sL, B + z sZ, the last
// of which has n_last columns.
// ---------------------------------------------------------------------------------
constexpr int TS_THREADS = 128;

struct TrsmArgs {
  const double* L;
  i64 ldl, sL;
  double* B;
  i64 ldb, sB, sZ;
  int nb;
  i64 org;
  int m, n, n_last;
  int identity;  // B starts as the identity and is not read
};

template <int R>
__global__ void __launch_bounds__(TS_THREADS) k_trsm_small(const TrsmArgs a, const int* status) {
  constexpr int LPR = TS_THREADS / R;  // lanes per row
  constexpr int TC = SB / LPR;         // columns per lane
  pdl_wait();
  if (status && *(volatile const int*)status) return;
  __shared__ __align__(16) double Ls[SB * SB];  // Ls[c * SB + r] = L(r, c)
  __shared__ double Rinv[SB];
  const int t = threadIdx.x, lane = t & 31;
  const int s = t & (LPR - 1);   // this lane holds columns s, s + LPR, ...
  const int z = blockIdx.y;
  const int n = (z == (int)gridDim.y - 1) ? a.n_last : a.n;
  const int r0 = blockIdx.x * R;
  if (r0 >= a.m || n <= 0) return;
  const double* L = a.L + (i64)z * a.sL;
  const int row = r0 + t / LPR;
  const int nl = (row < a.m) ? n : 0;  // columns this row loads and stores
  const i64 gr = a.org + (row < a.m ? row : 0);
  double* p = a.B + (i64)z * a.sZ + (gr / a.nb) * a.sB + gr % a.nb;
  double x[TC];
#pragma unroll
  for (int j = 0; j < TC; j++) {
    const int q = LPR * j + s;
    x[j] = a.identity ? (q == row && q < nl ? 1.0 : 0.0) : (q < nl) ? p[(i64)q * a.ldb] : 0.0;
  }
  {  // L column by column, threads down the rows (two columns per pass), 16 loads in flight
    const int r = t & (SB - 1), cg = t / SB;
#pragma unroll 16
    for (int c = cg; c < SB; c += TS_THREADS / SB) {
      double v = (r == c) ? 1.0 : 0.0;
      if (r < n && c < n && r >= c) v = L[r + (i64)c * a.ldl];
      Ls[c * SB + r] = v;
    }
  }
  __syncthreads();
  if (t < SB) Rinv[t] = 1.0 / Ls[t * SB + t];
  __syncthreads();
  const int base = lane & ~(LPR - 1);
#pragma unroll
  for (int i = 0; i < TC; i++) {
#pragma unroll (R == 4 ? 8 : LPR)
    for (int sc = 0; sc < LPR; sc++) {  // column c = LPR i + sc, held by lane sc of the row
      const double* lc = Ls + (LPR * i + sc) * SB + s;
      const double xc = __shfl_sync(0xffffffffu, x[i] * Rinv[LPR * i + sc], base | sc);  // the owner's x_c
      if (s == sc) x[i] = xc;
      if (s > sc) x[i] = fma(-xc, lc[LPR * i], x[i]);
#pragma unroll
      for (int j = i + 1; j < TC; j++) x[j] = fma(-xc, lc[LPR * j], x[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < TC; j++) {
    const int q = LPR * j + s;
    if (q < nl) p[(i64)q * a.ldb] = x[j];
  }
}

// ---------------------------------------------------------------------------------
// C(r, c) -= X(r) X(c)^T for the rows r >= c of a tile column and `w` <= 64 of its columns: the
// step between the two 64-column halves of a 128-column run.  Row i (counted from org, the
// run's second half) is addressed as in k_trsm_small; 16 divides nb and org.
// ---------------------------------------------------------------------------------
template <bool VEC, int BMX>
__global__ void __launch_bounds__(GEMM_THREADS)
k_half_update(const double* X, double* C, i64 ld, i64 stride, int nb, i64 org, int m, int w, int K, const int* status) {
  pdl_wait();
  if (status && *(volatile const int*)status) return;
  const int cblocks = (w + BMX - 1) / BMX;
  const int rb = blockIdx.x / cblocks, cb = blockIdx.x % cblocks;
  if (cb > rb) return;
  const i64 gr = org + (i64)rb * BMX, gc = org + (i64)cb * BMX;
  const i64 ro = (gr / nb) * stride + gr % nb, co = (gc / nb) * stride + gc % nb;
  gemm_block<VEC, BMX>(X + ro, ld, X + co, ld, C + ro + (i64)cb * BMX * ld, ld, min(BMX, m - rb * BMX),
                       min(BMX, w - cb * BMX), K, 0, 0, cb == rb, -1.0);
}

inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

}  // namespace

// =================================================================================
// Launchers
// =================================================================================

int launch_panel_update(const TileCol& X, const TileMap& C, int Ht, int Kt, i64 H, i64 Kcols, int K,
                        const int* status, cudaStream_t s) {
  if (Ht <= 0 || Kt <= 0 || K <= 0) return OOC_OK;
  i64 npairs = (i64)Kt * Ht - ((i64)Kt * (Kt - 1)) / 2;
  if (npairs > 65535) return OOC_ERR_INTERNAL;  // a panel never has that many tile pairs
  const int mblocks = (C.nb + BM - 1) / BM;
  const int nblocks = (C.nb + BN - 1) / BN;
  dim3 grid(mblocks * nblocks, (unsigned)npairs);
  bool vec = aligned16(X.base) && aligned16(C.base) && (X.ld % 2 == 0) && (C.ld % 2 == 0) &&
             (X.stride % 2 == 0);
  if (vec) k_panel_update<true><<<grid, GEMM_THREADS, 0, s>>>(X, C, Ht, Kt, H, Kcols, K, status);
  else k_panel_update<false><<<grid, GEMM_THREADS, 0, s>>>(X, C, Ht, Kt, H, Kcols, K, status);
  OOC_CUDA_TRY(cudaGetLastError());
  return OOC_OK;
}

static int sm_count() {
  static int nsm = [] {
    int d = 0, v = 0;
    cudaGetDevice(&d);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d);
    return v > 0 ? v : 1;
  }();
  return nsm;
}

static int launch_gemm_batched(const GemmBatch& gb, const int* status, cudaStream_t s) {
  if (gb.batch <= 0 || gb.n <= 0 || (gb.m <= 0 && gb.m_last <= 0)) return OOC_OK;
  if (gb.batch > 65535) return OOC_ERR_INTERNAL;
  const int mb = (max(gb.m, gb.m_last) + BM - 1) / BM;
  const int nbk = (gb.n + BN - 1) / BN;
  dim3 grid(mb * nbk, gb.batch);
  bool vec = aligned16(gb.A) && aligned16(gb.B) && aligned16(gb.C) && gb.lda % 2 == 0 &&
             gb.ldb % 2 == 0 && gb.sA % 2 == 0 && gb.sB % 2 == 0;
  if (gb.k <= 0) return OOC_OK;
  // An SM does ~1.75 FP64 FMAs per clock, so a 64 x 64 x 64 block alone takes ~75 us, a 32 x 32
  // one ~20 and a 16 x 16 one ~5: the blocks are as small as it takes to fill the GPU (up
  // to four 16 x 16 blocks per SM, which then take about as long as one 32 x 32 block).
  const i64 b64 = (i64)mb * nbk * gb.batch;
  cudaError_t e;
  if (8 * b64 < 2LL * sm_count()) {
    const int mb16 = (max(gb.m, gb.m_last) + 15) / 16, nb16 = (gb.n + 15) / 16;
    dim3 g16(mb16 * nb16, gb.batch);
    if (vec) e = launch_pdl(k_gemm_batched<true, 16>, g16, GEMM_THREADS, 0, s, gb, status);
    else e = launch_pdl(k_gemm_batched<false, 16>, g16, GEMM_THREADS, 0, s, gb, status);
  } else if (b64 < 2LL * sm_count()) {
    const int mb32 = (max(gb.m, gb.m_last) + 31) / 32, nb32 = (gb.n + 31) / 32;
    dim3 g32(mb32 * nb32, gb.batch);
    if (vec) e = launch_pdl(k_gemm_batched<true, 32>, g32, GEMM_THREADS, 0, s, gb, status);
    else e = launch_pdl(k_gemm_batched<false, 32>, g32, GEMM_THREADS, 0, s, gb, status);
  } else if (vec) {
    e = launch_pdl(k_gemm_batched<true, BM>, grid, GEMM_THREADS, 0, s, gb, status);
  } else {
    e = launch_pdl(k_gemm_batched<false, BM>, grid, GEMM_THREADS, 0, s, gb, status);
  }
  OOC_CUDA_TRY(e);
  return OOC_OK;
}

int launch_gemm_nt(const double* A, i64 lda, const double* B, i64 ldb, double* C, i64 ldc, int m, int n,
                   int k, int lower, double alpha, const int* status, cudaStream_t s) {
  GemmBatch gb{A, lda, 0, B, ldb, 0, C, ldc, 0, m, m, n, k, lower, 1, alpha, 0};
  return launch_gemm_batched(gb, status, s);
}

int launch_gemm_nt_trib(const double* A, i64 lda, const double* B, i64 ldb, double* C, i64 ldc, int m, int n, int k,
                        double alpha, const int* status, cudaStream_t s) {
  GemmBatch gb{A, lda, 0, B, ldb, 0, C, ldc, 0, m, m, n, k, 0, 1, alpha, 1};
  return launch_gemm_batched(gb, status, s);
}

// Rows per CTA: as few as fill the GPU (4 rows a CTA up to one wave, then 8, 16, 32).
static int launch_trsm(const TrsmArgs& a, int batch, const int* status, cudaStream_t s) {
  if (batch <= 0 || a.m <= 0 || (a.n <= 0 && a.n_last <= 0)) return OOC_OK;
  if (a.n > SB || a.n_last > SB || batch > 65535) return OOC_ERR_INTERNAL;
  const i64 rows = (i64)a.m * batch;
  cudaError_t e;
  if (rows <= 4LL * sm_count()) e = launch_pdl(k_trsm_small<4>, dim3((a.m + 3) / 4, batch), TS_THREADS, 0, s, a, status);
  else if (rows <= 8LL * sm_count()) e = launch_pdl(k_trsm_small<8>, dim3((a.m + 7) / 8, batch), TS_THREADS, 0, s, a, status);
  else if (rows <= 16LL * sm_count()) e = launch_pdl(k_trsm_small<16>, dim3((a.m + 15) / 16, batch), TS_THREADS, 0, s, a, status);
  else e = launch_pdl(k_trsm_small<32>, dim3((a.m + 31) / 32, batch), TS_THREADS, 0, s, a, status);
  OOC_CUDA_TRY(e);
  return OOC_OK;
}

static int launch_trsm_small(const double* L, i64 ldl, double* B, i64 ldb, i64 sB, int m, int m_last,
                             int batch, int n, const int* status, cudaStream_t s) {
  if (batch <= 0 || n <= 0) return OOC_OK;
  return launch_trsm(TrsmArgs{L, ldl, 0, B, ldb, sB, 0, m > 0 ? m : 1, 0, (batch - 1) * m + m_last, n, n, 0}, 1, status, s);
}

int launch_trsm_rows(const double* L, i64 ldl, double* B, i64 ldb, i64 stride, int nb, i64 org, i64 m, int n,
                     const int* status, cudaStream_t s) {
  if (m <= 0 || n <= 0) return OOC_OK;
  if (m > (1 << 30)) return OOC_ERR_INTERNAL;
  return launch_trsm(TrsmArgs{L, ldl, 0, B, ldb, stride, 0, nb, org, (int)m, n, n, 0}, 1, status, s);
}

int launch_diag_inverses(const double* L, i64 ldl, i64 n, double* Dinv, cudaStream_t s) {
  if (n > 0 && n < SB)
    return launch_trsm(TrsmArgs{L, ldl, 0, Dinv, n, 0, 0, SB, 0, (int)n, (int)n, (int)n, 1}, 1, nullptr, s);
  const i64 nblk = (n + SB - 1) / SB;
  for (i64 z = 0; z < nblk; z += 65535) {
    const int batch = (int)min(nblk - z, (i64)65535);
    const int last = z + batch == nblk ? (int)(n - (nblk - 1) * SB) : SB;
    int rc = launch_trsm(TrsmArgs{L + z * SB * (ldl + 1), ldl, SB * (ldl + 1), Dinv + z * SB * SB, SB, 0, SB * SB, SB, 0, SB, SB,
                                  last, 1}, batch, nullptr, s);
    if (rc) return rc;
  }
  return OOC_OK;
}

int launch_potrf_block(double* A, i64 ld, int n, i64 col0, int* status, cudaStream_t s) {
  if (n <= 0) return OOC_OK;
  if (n > SB) return OOC_ERR_INTERNAL;
  OOC_CUDA_TRY(launch_pdl(k_potrf_small, dim3(1), PT_THREADS, 0, s, A, ld, n, col0, status));
  return OOC_OK;
}

// 16 x 16 blocks up to about two per SM, then 32 x 32.
int launch_half_update(const double* X, double* C, i64 ld, i64 stride, int nb, i64 org, i64 m, int w, int K,
                       const int* status, cudaStream_t s) {
  if (m <= 0 || w <= 0 || K <= 0) return OOC_OK;
  if (w > SB || m > (1 << 30) || nb % 32 || org % 32) return OOC_ERR_INTERNAL;
  const bool vec = aligned16(X) && aligned16(C) && ld % 2 == 0 && stride % 2 == 0;
  const bool small = ((m + 15) / 16) * ((w + 15) / 16) <= 2LL * sm_count();
  const int bx = small ? 16 : 32;
  const unsigned grid = (unsigned)(((m + bx - 1) / bx) * ((w + bx - 1) / bx));
  cudaError_t e;
  if (small) {
    if (vec) e = launch_pdl(k_half_update<true, 16>, dim3(grid), GEMM_THREADS, 0, s, X, C, ld, stride, nb, org, (int)m, w, K, status);
    else e = launch_pdl(k_half_update<false, 16>, dim3(grid), GEMM_THREADS, 0, s, X, C, ld, stride, nb, org, (int)m, w, K, status);
  } else {
    if (vec) e = launch_pdl(k_half_update<true, 32>, dim3(grid), GEMM_THREADS, 0, s, X, C, ld, stride, nb, org, (int)m, w, K, status);
    else e = launch_pdl(k_half_update<false, 32>, dim3(grid), GEMM_THREADS, 0, s, X, C, ld, stride, nb, org, (int)m, w, K, status);
  }
  OOC_CUDA_TRY(e);
  return OOC_OK;
}

int launch_potrf_tile(double* A, i64 ld, int n, i64 col0, int* status, cudaStream_t s) {
  for (int k = 0; k < n; k += SB) {
    const int kb = min(SB, n - k);
    double* Akk = A + k + (i64)k * ld;
    int rc = launch_potrf_block(Akk, ld, kb, col0 + k, status, s);
    if (rc) return rc;
    const int rest = n - k - kb;
    if (rest > 0) {
      double* Bp = A + (k + kb) + (i64)k * ld;  // rows below the block, columns k..k+kb
      rc = launch_trsm_small(Akk, ld, Bp, ld, 0, rest, rest, 1, kb, status, s);
      if (rc) return rc;
      double* Ct = A + (k + kb) + (i64)(k + kb) * ld;
      rc = launch_gemm_nt(Bp, ld, Bp, ld, Ct, ld, rest, rest, kb, 1, -1.0, status, s);
      if (rc) return rc;
    }
  }
  return OOC_OK;
}

int launch_trsm_col(const double* L, i64 ldl, const TileCol& B, int ntiles, int nb, int m_last, int n,
                    const int* status, cudaStream_t s) {
  if (ntiles <= 0) return OOC_OK;
  double* Bb = const_cast<double*>(B.base);
  for (int k = 0; k < n; k += SB) {
    const int kb = min(SB, n - k);
    const double* Lkk = L + k + (i64)k * ldl;
    int rc = launch_trsm_small(Lkk, ldl, Bb + (i64)k * B.ld, B.ld, B.stride, nb, m_last, ntiles, kb,
                               status, s);
    if (rc) return rc;
    const int rest = n - k - kb;
    if (rest > 0) {
      // B[:, k+kb:n] -= B[:, k:k+kb] L[k+kb:n, k:k+kb]^T for every tile of the column.
      GemmBatch gb{Bb + (i64)k * B.ld, B.ld, B.stride,
                   L + (k + kb) + (i64)k * ldl, ldl, 0,
                   Bb + (i64)(k + kb) * B.ld, B.ld, B.stride,
                   nb, m_last, rest, kb, 0, ntiles, -1.0, 0};
      rc = launch_gemm_batched(gb, status, s);
      if (rc) return rc;
    }
  }
  return OOC_OK;
}
