// Triangular solves L L^T X = B with a factor on the device: both sweeps in one launch.
//
// A sweep in panels (inverse product, then panel product, two launches per panel) is bound
// by launches and by the few CTAs a panel fills: 11 us per 256 rows where the factor's bytes
// take 0.7.  Here the rows are cut into blocks of BS and the CTAs take (sweep, block) tasks from
// a ticket counter in dependence order, so a CTA only ever waits for tasks that others have
// already started (no assumption on how many CTAs are resident).  Task (forward, i):
//     y_i = L_ii^{-1} (b_i - sum_{j < i} L_ij y_j),     L_ij loaded before y_j is waited for,
// and the same with L^T from the last block for the backward sweep.  A finished block goes to
// the others as packets: 64-bit words of 32 data bits and a 32-bit tag (the launch's epoch), so
// the arrival of the data is its own flag and one L2 round trip passes it on.
// Bound by that chain: 2.2 us per 128 rows in FP32 (0.69 ms for both sweeps at n = 20000, where
// the launches per panel took 1.7 ms), 3.1 us per 64 rows in FP64, two thirds of it the FP64 pipe of one SM
// (0.58 ms for both sweeps at n = 6000, 0.67 by launches per panel of 512 columns and 0.73 with L^T's
// sums by shuffles, an addition chain per block and the words of a number polled one after the other); the
// factor streams from HBM beside it.  Several right-hand sides in FP64 are bound by the FP64 pipe: 16 at
// n = 30000 take 37 ms (40.7 by launches per panel).
// Sums are block by block in a fixed order, so results do not depend on scheduling.
//
// Every wait is bounded: one that runs out raises the buffer's error word, which ends the
// other CTAs' waits too.

#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "trsolve.cuh"

namespace {

constexpr int TS_RMAX = 8;                 // right-hand sides per task
constexpr unsigned TS_POLLS = 1u << 22;    // polls before a wait is declared stuck
constexpr size_t TS_CTL = 256;             // ticket, error word

template <typename T>
struct Cfg;
template <>
struct Cfg<float> { static constexpr int BS = 128, WORDS = 1; };
template <>
struct Cfg<double> { static constexpr int BS = 64, WORDS = 2; };

__device__ __forceinline__ unsigned long long ld_packet(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];\n" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_packet(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;\n" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long pack(uint32_t bits, unsigned tag) {
  return ((unsigned long long)tag << 32) | bits;
}
__device__ __forceinline__ void send(unsigned long long* x, i64 at, float v, unsigned tag) {
  st_packet(x + at, pack(__float_as_uint(v), tag));
}
// The two words of a double go and come together (each has its tag, so they may still arrive apart).
__device__ __forceinline__ void send(unsigned long long* x, i64 at, double v, unsigned tag) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};\n" ::"l"(x + 2 * at), "l"(pack((uint32_t)__double2loint(v), tag)),
               "l"(pack((uint32_t)__double2hiint(v), tag))
               : "memory");
}
// One word, waiting (bounded) for its tag; 0 when the wait ends without it.
__device__ __forceinline__ uint32_t take(const unsigned long long* p, unsigned tag, int* ctl) {
  for (unsigned i = 0; i < TS_POLLS; i++) {
    const unsigned long long v = ld_packet(p);
    if ((unsigned)(v >> 32) == tag) return (uint32_t)v;
    if ((i & 63) == 63 && *(volatile int*)(ctl + 1)) return 0;
  }
  atomicExch(ctl + 1, 1);
  return 0;
}
__device__ __forceinline__ float receive(const unsigned long long* x, i64 at, unsigned tag, int* ctl, float) {
  return __uint_as_float(take(x + at, tag, ctl));
}
__device__ __forceinline__ double receive(const unsigned long long* x, i64 at, unsigned tag, int* ctl, double) {
  for (unsigned i = 0; i < TS_POLLS; i++) {
    unsigned long long lo, hi;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n" : "=l"(lo), "=l"(hi) : "l"(x + 2 * at) : "memory");
    if ((unsigned)(lo >> 32) == tag && (unsigned)(hi >> 32) == tag) return __hiloint2double((int)(uint32_t)hi, (int)(uint32_t)lo);
    if ((i & 63) == 63 && *(volatile int*)(ctl + 1)) return 0.0;
  }
  atomicExch(ctl + 1, 1);
  return 0.0;
}

// Rows of block b: start, count, and its diagonal inverse (ld).
template <typename T>
__device__ __forceinline__ void block_of(const TriSolve<T>& a, int b, i64* s, int* m, const T** U, int* ldu) {
  constexpr int BS = Cfg<T>::BS;
  const int hc = a.tail0 >= a.n ? (int)((a.n + a.nb - 1) / a.nb) : (int)(a.tail0 / a.nb);
  const int pp = (a.nb + BS - 1) / BS, pp2 = (a.nb2 + BS - 1) / BS;
  i64 J0, off;
  int q, W;
  if (b < hc * pp) {
    const int p = b / pp;
    q = b - p * pp;
    J0 = (i64)p * a.nb;
    off = (i64)p * a.nb * a.nb;
    W = a.nb;
  } else {
    const int u = b - hc * pp, p = u / pp2;
    q = u - p * pp2;
    J0 = a.tail0 + (i64)p * a.nb2;
    off = (i64)hc * a.nb * a.nb + (i64)p * a.nb2 * a.nb2;
    W = a.nb2;
  }
  *ldu = W;
  *U = a.Dinv + off + (i64)q * BS * (W + 1);
  *s = J0 + (i64)q * BS;
  *m = (int)min((i64)min(BS, W - q * BS), a.n - *s);
}

// v[0..V) summed over the warp's lanes; afterwards lane l holds the sums of indices
// first(l) .. first(l) + V/32 - 1 (V < 32: of one index, the same in 32/V lanes).
template <int V, typename T>
__device__ __forceinline__ int warp_transpose_sum(T (&v)[V], int lane) {
  int idx = 0;
#pragma unroll
  for (int st = 0; st < 5; st++) {
    const int off = 16 >> st;
    const int cnt = V >> st;  // values still held
    if (cnt > 1) {
      const bool hi = (lane & off) != 0;
#pragma unroll
      for (int j = 0; j < V / 2; j++)
        if (j < cnt / 2) {
          const T send = hi ? v[j] : v[j + cnt / 2];
          const T keep = hi ? v[j + cnt / 2] : v[j];
          v[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
      if (hi) idx += cnt / 2;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    }
  }
  return idx;
}

template <typename T, int R>
__global__ void __launch_bounds__(Cfg<T>::BS * 4)
    k_trsolve(const __grid_constant__ TriSolve<T> a, int nblk, int ngrp, unsigned long long* __restrict__ xch, int* ctl,
              unsigned tag) {
  constexpr int BS = Cfg<T>::BS, NT = BS * 4, KS = BS / 4, NW = NT / 32, CPW = BS / NW, RPL = BS / 32;
  static_assert(CPW == 8, "eight columns per warp");
  extern __shared__ __align__(16) unsigned char sm_raw[];
  T* D = reinterpret_cast<T*>(sm_raw);   // the block's inverse, D[k + i * (BS + 1)] = U(k, i)
  T* xs = D + (R == 1 ? 0 : BS * (BS + 1));  // arriving block, xs[buf][k * R + q]
  T* red = xs + 2 * BS * R;              // partial sums, red[(slice * BS + row) * R + q]
  T* ys = red + 4 * BS * R;              // ys[row * R + q]
  __shared__ int s_ticket;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int row = t % BS, slice = t / BS;
  const int nsw = a.sweeps == 3 ? 2 : 1;
  const int total = nsw * nblk * ngrp;
  const i64 dir_words = (i64)a.n * a.r * Cfg<T>::WORDS;
  for (;;) {
    __syncthreads();
    if (t == 0) s_ticket = *(volatile int*)(ctl + 1) ? total : atomicAdd(ctl, 1);  // (a wait ran out: stop)
    __syncthreads();
    const int tk = s_ticket;
    if (tk >= total) {
      // the last CTA to stop leaves the counter at zero for the next launch
      if (t == 0 && atomicAdd(ctl + 2, 1) == (int)gridDim.x - 1) {
        ctl[0] = 0;
        ctl[2] = 0;
      }
      return;
    }
    const int grp = tk % ngrp, u = tk / ngrp;
    const bool fwd = a.sweeps != 2 && u < nblk;
    const int i = fwd ? u : (nsw * nblk - 1 - u);
    const int q0 = grp * R, rn = min(R, a.r - q0);  // this task's right-hand sides
    i64 si;
    int mi, ldu;
    const T* U;
    block_of(a, i, &si, &mi, &U, &ldu);
    // The block's inverse, used only after the sums below (its loads overlap them): one
    // right-hand side keeps the thread's elements in registers, more share them.
    constexpr bool DREG = R == 1;
    T dr[DREG ? KS : 1];
    if constexpr (DREG) {
#pragma unroll
      for (int k = 0; k < KS; k++) {
        const int kk = slice * KS + k;
        dr[k] = T(0);
        if (row < mi && kk < mi && (fwd ? kk <= row : kk >= row)) dr[k] = fwd ? U[kk + (i64)row * ldu] : U[row + (i64)kk * ldu];
      }
    } else {
#pragma unroll 8
      for (int idx = t; idx < BS * BS; idx += NT) {
        const int k = idx % BS, c = idx / BS;
        D[k + c * (BS + 1)] = (k <= c && c < mi) ? U[k + (i64)c * ldu] : T(0);
      }
    }
    unsigned long long* out = xch + (fwd || nsw == 1 ? 0 : dir_words);
    auto fetch = [&](int j, int buf) {  // block j of this sweep's solution into xs[buf]
      i64 sj;
      int mj, l2;
      const T* u2;
      block_of(a, j, &sj, &mj, &u2, &l2);
      for (int idx = t; idx < BS * R; idx += NT) {
        const int k = idx % BS, q = idx / BS;
        T v = T(0);
        if (k < mj && q < rn) v = receive(out, (i64)(q0 + q) * a.n + sj + k, tag, ctl, T(0));
        xs[buf * BS * R + k * R + q] = v;
      }
    };
    // b (forward) or y (backward) of the thread's element(s), off the chain
    constexpr int PE = (BS * R + NT - 1) / NT;
    T rhs[PE];
#pragma unroll
    for (int z = 0; z < PE; z++) {
      const int idx = t + z * NT, rr = idx % BS, q = idx / BS;
      rhs[z] = T(0);
      if (q < rn && rr < mi) {
        if (fwd || nsw == 1) rhs[z] = a.B[si + rr + (i64)(q0 + q) * a.ldb];
        else rhs[z] = receive(xch, (i64)(q0 + q) * a.n + si + rr, tag, ctl, T(0));
      }
    }
    int buf = 0;
    if (fwd) {
      T acc[R];
#pragma unroll
      for (int q = 0; q < R; q++) acc[q] = T(0);
      const T* Lr = a.L + si + (row < mi ? row : 0);
      for (int j = 0; j < i; j++, buf ^= 1) {
        i64 sj;
        int mj, l2;
        const T* u2;
        block_of(a, j, &sj, &mj, &u2, &l2);
        T l[KS];
#pragma unroll
        for (int k = 0; k < KS; k++) {
          const int c = slice * KS + k;
          l[k] = (row < mi && c < mj) ? Lr[(sj + c) * a.ldl] : T(0);
        }
        fetch(j, buf);
        __syncthreads();
        const T* x = xs + buf * BS * R + slice * KS * R;
        constexpr int PS = R == 1 ? 4 : 1;  // partial sums per right-hand side (a chain of KS FMAs otherwise)
        T p[PS][R];
#pragma unroll
        for (int z = 0; z < PS; z++)
#pragma unroll
          for (int q = 0; q < R; q++) p[z][q] = T(0);
#pragma unroll
        for (int k = 0; k < KS; k++)
#pragma unroll
          for (int q = 0; q < R; q++) p[k % PS][q] = fma(l[k], x[k * R + q], p[k % PS][q]);
#pragma unroll
        for (int q = 0; q < R; q++) acc[q] += PS == 4 ? (p[0][q] + p[1 % PS][q]) + (p[2 % PS][q] + p[3 % PS][q]) : p[0][q];
      }
#pragma unroll
      for (int q = 0; q < R; q++) red[t * R + q] = acc[q];
      __syncthreads();
#pragma unroll
      for (int z = 0; z < PE; z++) {
        const int idx = t + z * NT, rr = idx % BS, q = idx / BS;
        if (q < R) {
          T v = rhs[z];
          if (rr < mi && q < rn)
            v -= (red[rr * R + q] + red[(BS + rr) * R + q]) + (red[(2 * BS + rr) * R + q] + red[(3 * BS + rr) * R + q]);
          ys[rr * R + q] = v;
        }
      }
      __syncthreads();
    } else {
      T v[CPW * R];
#pragma unroll
      for (int z = 0; z < CPW * R; z++) v[z] = T(0);
      for (int j = nblk - 1; j > i; j--, buf ^= 1) {
        i64 sj;
        int mj, l2;
        const T* u2;
        block_of(a, j, &sj, &mj, &u2, &l2);
        T l[CPW * RPL];
#pragma unroll
        for (int c = 0; c < CPW; c++)
#pragma unroll
          for (int p = 0; p < RPL; p++) {
            const int k = lane + 32 * p, cc = warp * CPW + c;
            l[c * RPL + p] = (k < mj && cc < mi) ? a.L[sj + k + (si + cc) * a.ldl] : T(0);
          }
        fetch(j, buf);
        __syncthreads();
        const T* x = xs + buf * BS * R;
        T w[R];
#pragma unroll
        for (int c = 0; c < CPW; c++) {
#pragma unroll
          for (int q = 0; q < R; q++) w[q] = T(0);
#pragma unroll
          for (int p = 0; p < RPL; p++)
#pragma unroll
            for (int q = 0; q < R; q++) w[q] = fma(l[c * RPL + p], x[(lane + 32 * p) * R + q], w[q]);
#pragma unroll
          for (int q = 0; q < R; q++) v[c * R + q] += w[q];
        }
      }
      const int first = warp_transpose_sum<CPW * R>(v, lane);
      constexpr int KEEP = CPW * R >= 32 ? CPW * R / 32 : 1;
      if (CPW * R >= 32 || (lane & (32 / (CPW * R) - 1)) == 0) {
#pragma unroll
        for (int z = 0; z < KEEP; z++) red[(warp * CPW) * R + first + z] = v[z];
      }
      __syncthreads();
#pragma unroll
      for (int z = 0; z < PE; z++) {
        const int idx = t + z * NT, rr = idx % BS, q = idx / BS;
        if (q < R) ys[rr * R + q] = rr < mi && q < rn ? rhs[z] - red[rr * R + q] : T(0);
      }
      __syncthreads();
    }
    // The block's inverse: forward x(row) = sum_{k <= row} U(k, row) y(k), backward x(row) =
    // sum_{k >= row} U(row, k) y(k); thread (row, slice of k), warps outside the triangle idle.
    T p[R];
#pragma unroll
    for (int q = 0; q < R; q++) p[q] = T(0);
    const int wr = row & ~31, k0 = slice * KS;  // the warp's first row, the slice's first k
    if (fwd ? k0 <= wr + 31 : k0 + KS > wr) {
#pragma unroll
      for (int k = 0; k < KS; k++) {
        const T d = DREG ? dr[DREG ? k : 0] : fwd ? D[k0 + k + row * (BS + 1)] : D[row + (k0 + k) * (BS + 1)];
#pragma unroll
        for (int q = 0; q < R; q++) p[q] = fma(d, ys[(k0 + k) * R + q], p[q]);
      }
    }
    // (red was last read before the barrier above)
#pragma unroll
    for (int q = 0; q < R; q++) red[t * R + q] = p[q];
    __syncthreads();
#pragma unroll
    for (int z = 0; z < PE; z++) {
      const int idx = t + z * NT, rr = idx % BS, q = idx / BS;
      if (rr < mi && q < rn) {
        const T x =
            (red[rr * R + q] + red[(BS + rr) * R + q]) + (red[(2 * BS + rr) * R + q] + red[(3 * BS + rr) * R + q]);
        send(out, (i64)(q0 + q) * a.n + si + rr, x, tag);
        if (!fwd || nsw == 1) a.B[si + rr + (i64)(q0 + q) * a.ldb] = x;
      }
    }
  }
}

// FP64, one right-hand side per task.  A block step is 64 x 64 products with L and with the inverse on one SM's
// FP64 pipe (1.75 FMAs per clock, a warp-wide instruction every 64 clocks of a sub-partition), so the chain has nothing
// in it but the FMAs of the last block and of the inverse, and eight additions: the other blocks' sums are put
// together while the last block is waited for, L^T's elements go through shared memory to the thread (row of the
// result, slice of 16 columns) that sums them, the next block's loads are in flight meanwhile, and a half of the
// inverse's triangle is cut so that each sub-partition has 24 of its FMAs.
__global__ void __launch_bounds__(256, 2)
    k_trsolve_f64(const __grid_constant__ TriSolve<double> a, int nblk, unsigned long long* __restrict__ xch, int* ctl,
                  unsigned tag) {
  constexpr int BS = 64, KS = 16, LD = BS + 1;
  constexpr int FOLD = 4;  // blocks summed before they join the row's sum
  __shared__ double Lt[BS * LD];  // L^T of a block, Lt[column * LD + row]
  __shared__ double xs[2][BS], red[4 * BS], ys[BS];
  __shared__ int s_ticket;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int half = warp >> 2, slice = warp & 3, row = lane + 32 * half;
  const int nsw = a.sweeps == 3 ? 2 : 1;
  const int total = nsw * nblk * a.r;
  const i64 dir_words = 2 * (i64)a.n * a.r;
  for (;;) {
    __syncthreads();
    if (t == 0) s_ticket = *(volatile int*)(ctl + 1) ? total : atomicAdd(ctl, 1);  // (a wait ran out: stop)
    __syncthreads();
    const int tk = s_ticket;
    if (tk >= total) {
      // the last CTA to stop leaves the counter at zero for the next launch
      if (t == 0 && atomicAdd(ctl + 2, 1) == (int)gridDim.x - 1) {
        ctl[0] = 0;
        ctl[2] = 0;
      }
      return;
    }
    const int q = tk % a.r, u = tk / a.r;  // (right-hand sides side by side: L comes from L2 for all but one)
    const bool fwd = a.sweeps != 2 && u < nblk;
    const int i = fwd ? u : (nsw * nblk - 1 - u);
    i64 si;
    int mi, ldu;
    const double* U;
    block_of(a, i, &si, &mi, &U, &ldu);
    unsigned long long* out = xch + (fwd || nsw == 1 ? 0 : dir_words);
    double* Bq = a.B + (i64)q * a.ldb;
    // the thread's elements of the inverse: forward columns k <= row of U^T, backward k >= row of U
    const bool whole = fwd == (half == 1);  // 16 columns, else 8 of the 32 that the triangle leaves
    const int kd = whole ? KS * slice : (fwd ? 8 * slice : 32 + 8 * slice);
    double dr[KS];
#pragma unroll
    for (int k = 0; k < KS; k++) {
      const int kk = kd + k;
      dr[k] = 0.0;
      if ((k < 8 || whole) && row < mi && kk < mi && (fwd ? kk <= row : kk >= row))
        dr[k] = fwd ? U[kk + (i64)row * ldu] : U[row + (i64)kk * ldu];
    }
    // block j of L as it lies in memory: forward the thread's own elements, backward rows lane and lane + 32 of
    // eight columns
    double nx[KS];
    auto load = [&](int j) {
      i64 sj;
      int mj, l2;
      const double* u2;
      block_of(a, j, &sj, &mj, &u2, &l2);
      if (fwd) {
        const double* p = a.L + si + (row < mi ? row : 0) + (sj + KS * slice) * a.ldl;
#pragma unroll
        for (int k = 0; k < KS; k++) nx[k] = row < mi && KS * slice + k < mj ? p[k * a.ldl] : 0.0;
      } else {
        const double* p = a.L + sj + (si + 8 * warp) * a.ldl;
#pragma unroll
        for (int k = 0; k < KS; k++) {
          const int c = k >> 1, r = lane + 32 * (k & 1);
          nx[k] = r < mj && 8 * warp + c < mi ? p[r + c * a.ldl] : 0.0;
        }
      }
    };
    const int steps = fwd ? i : nblk - 1 - i;
    if (steps > 0) load(fwd ? 0 : nblk - 1);
    // b (forward) or y (backward), off the chain; it meets the sums once, at the end, so that they are rounded to
    // their own size
    double rhs = 0.0, acc = 0.0, p = 0.0;
    if (t < mi) rhs = fwd || nsw == 1 ? Bq[si + t] : receive(xch, (i64)q * a.n + si + t, tag, ctl, 0.0);
    for (int st = 0; st < steps; st++) {
      const int j = fwd ? st : nblk - 1 - st;
      double l[KS];
      if (fwd) {
#pragma unroll
        for (int k = 0; k < KS; k++) l[k] = nx[k];
      } else {
        // (the last block's elements were read before the barrier that followed)
#pragma unroll
        for (int k = 0; k < KS; k++) Lt[(8 * warp + (k >> 1)) * LD + lane + 32 * (k & 1)] = nx[k];
        __syncthreads();
#pragma unroll
        for (int k = 0; k < KS; k++) l[k] = Lt[row * LD + KS * slice + k];
      }
      if ((st & (FOLD - 1)) == 0 || st + 1 == steps) {
        acc += p;
        p = 0.0;
      }
      if (st + 1 < steps) load(fwd ? j + 1 : j - 1);
      if (t < BS) {
        i64 sj;
        int mj, l2;
        const double* u2;
        block_of(a, j, &sj, &mj, &u2, &l2);
        xs[st & 1][t] = t < mj ? receive(out, (i64)q * a.n + sj + t, tag, ctl, 0.0) : 0.0;
      }
      __syncthreads();
      const double* x = xs[st & 1] + KS * slice;
#pragma unroll
      for (int k = 0; k < KS; k++) p = fma(l[k], x[k], p);
    }
    red[slice * BS + row] = acc + p;
    __syncthreads();
    if (t < BS) ys[t] = t < mi ? rhs - ((red[t] + red[BS + t]) + (red[2 * BS + t] + red[3 * BS + t])) : 0.0;
    __syncthreads();
    p = 0.0;
#pragma unroll
    for (int k = 0; k < 8; k++) p = fma(dr[k], ys[kd + k], p);
    if (whole) {
#pragma unroll
      for (int k = 8; k < KS; k++) p = fma(dr[k], ys[kd + k], p);
    }
    // (red was last read before the barrier above)
    red[slice * BS + row] = p;
    __syncthreads();
    if (t < mi) {
      const double x = (red[t] + red[BS + t]) + (red[2 * BS + t] + red[3 * BS + t]);
      send(out, (i64)q * a.n + si + t, x, tag);
      if (!fwd || nsw == 1) Bq[si + t] = x;
    }
  }
}

template <typename T, int R>
int launch_r(const TriSolve<T>& a, int nblk, int ngrp, void* exchange, unsigned epoch, cudaStream_t s) {
  constexpr int BS = Cfg<T>::BS;
  const size_t smem = (size_t)((R == 1 ? 0 : BS * (BS + 1)) + 2 * BS * R + 4 * BS * R + BS * R) * sizeof(T);
  OOC_CUDA_TRY(cudaFuncSetAttribute(k_trsolve<T, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int dev = 0, nsm = 0;
  OOC_CUDA_TRY(cudaGetDevice(&dev));
  OOC_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  const int tasks = nblk * ngrp;  // tasks of one sweep
  k_trsolve<T, R><<<std::max(1, std::min(tasks, nsm)), BS * 4, smem, s>>>(
      a, nblk, ngrp, (unsigned long long*)((char*)exchange + TS_CTL), (int*)exchange, epoch);
  OOC_CUDA_TRY(cudaGetLastError());
  return OOC_OK;
}

}  // namespace

size_t trsolve_bytes(i64 n, int r, int elem_size, int sweeps) {
  return TS_CTL + (size_t)sweeps * (size_t)n * (size_t)r * (elem_size == 4 ? 8 : 16);
}

template <typename T>
int launch_trsolve(const TriSolve<T>& a, void* exchange, unsigned epoch, cudaStream_t s) {
  constexpr int BS = Cfg<T>::BS;
  if (a.n <= 0 || a.r <= 0) return OOC_OK;
  if (a.nb <= 0 || a.sweeps < 1 || a.sweeps > 3 || epoch == 0) return OOC_ERR_INTERNAL;
  TriSolve<T> b = a;
  if (b.tail0 >= b.n || b.nb2 <= 0) {
    b.tail0 = b.n;
    b.nb2 = b.nb;
  }
  const i64 hc = b.tail0 >= b.n ? (b.n + b.nb - 1) / b.nb : b.tail0 / b.nb;
  const i64 pp = (b.nb + BS - 1) / BS, pp2 = (b.nb2 + BS - 1) / BS;
  i64 nblk;  // whole panels, then the pieces of the last one
  if (b.tail0 >= b.n) {
    nblk = (hc - 1) * pp + (b.n - (hc - 1) * b.nb + BS - 1) / BS;
  } else {
    const i64 tc = (b.n - b.tail0 + b.nb2 - 1) / b.nb2;
    nblk = hc * pp + (tc - 1) * pp2 + (b.n - b.tail0 - (tc - 1) * b.nb2 + BS - 1) / BS;
  }
  // FP64: one right-hand side per task.  A block step is FP64 work of one SM (64 x 64 products
  // with L and with the inverse, 2.4 us at 1.75 FMAs per clock for each right-hand side), so
  // the right-hand sides go side by side on different SMs; L comes from L2 for all but one.
  // FP32: R per task.  Fewer make a block step of the chain shorter, more make the groups, which all read
  // L, fewer: the smallest R whose tasks still fit the SMs, 4 while they are at most four to an SM.  us
  // for R = 1, 2, 4, 8:  n = 2048  r = 8 117 119 134 195,  r = 16 144 121 133 207
  //                      n = 6000  r = 4 266 245 283 445,  r = 16 592 401 321 496
  //                      n = 16384 r = 2 789 636 714 1226, r = 16 3611 2118 1380 1471
  //                      n = 30000 r = 8 6238 3542 2381 2676, r = 16 11591 6503 4005 3703
  const int r = b.r;
  if (nblk * r * 2 > 0x3fffffff) return OOC_ERR_INTERNAL;
  int dev = 0, nsm = 0;
  OOC_CUDA_TRY(cudaGetDevice(&dev));
  OOC_CUDA_TRY(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  if constexpr (sizeof(T) == 8) {
    // two CTAs per SM, one's products beside the other's round trips
    k_trsolve_f64<<<(unsigned)std::min<i64>(nblk * r, 2 * nsm), 256, 0, s>>>(
        b, (int)nblk, (unsigned long long*)((char*)exchange + TS_CTL), (int*)exchange, epoch);
    OOC_CUDA_TRY(cudaGetLastError());
    return OOC_OK;
  } else {
    auto groups = [&](int R) { return (r + R - 1) / R; };
    if (r == 1 || nblk * r <= nsm) return launch_r<T, 1>(b, (int)nblk, r, exchange, epoch, s);
    if (r == 2 || 4 * nblk * groups(2) <= 5 * nsm) return launch_r<T, 2>(b, (int)nblk, groups(2), exchange, epoch, s);
    if (r <= 4 || nblk * groups(4) <= 4 * nsm) return launch_r<T, 4>(b, (int)nblk, groups(4), exchange, epoch, s);
    return launch_r<T, TS_RMAX>(b, (int)nblk, groups(TS_RMAX), exchange, epoch, s);
  }
}
template int launch_trsolve<float>(const TriSolve<float>&, void*, unsigned, cudaStream_t);
template int launch_trsolve<double>(const TriSolve<double>&, void*, unsigned, cudaStream_t);
