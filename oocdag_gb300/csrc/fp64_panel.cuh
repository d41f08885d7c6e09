// A block of 16 columns of an FP64 Cholesky factorization in shared memory (the method and what
// bounds it: k_potrf_small in fp64_kernels.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace {

constexpr int PB = 16;  // columns per block

// r0 ~ 1 / d to 23 bits, from the FP32 reciprocal of the mantissa, for a d well inside the
// exponent range (recip_ok).
__device__ __forceinline__ bool recip_ok(double d) {
  return (unsigned)((__double2hiint(d) >> 20) - 23) <= 2000u;  // 2^-1000 <= d < 2^1001
}
__device__ __forceinline__ double recip_seed(double d) {
  const int hi = __double2hiint(d), lo = __double2loint(d);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(0x3F800000u | ((uint32_t)(hi & 0xFFFFF) << 3) | ((uint32_t)lo >> 29))));
  const uint32_t rb = __float_as_uint(r);  // in [1/2, 1]
  const int e = (int)(rb >> 23) - 127 - ((hi >> 20) - 1023) + 1023;
  return __hiloint2double((e << 20) | (int)((rb & 0x7FFFFFu) >> 3), (int)(rb << 29));
}
__device__ __noinline__ double slow_div(double a, double d) { return a / d; }
__device__ __forceinline__ bool positive(double d) {  // d > 0 (false for NaN), off the FP64 pipe
  return (unsigned long long)__double_as_longlong(d) - 1ull < 0x7FF0000000000000ull;
}

// One column block: columns k .. k+15 of the rows from k on of an SB x SB block in shared memory
// (S[c SP + r]), LPR threads per row (threads t <
// (SB - k) LPR; the others return at once).  More threads per row where rows are few: an
// instruction costs a warp 64 clocks whatever its lanes.  Returns the columns that factored.
// U, where given (PB columns of pitch SP), gets a(r, j) / d(j): the other factor of an update by the
// unscaled columns.
template <int LPR, int SB, int SP>
__device__ __forceinline__ int potrf_panel(double* S, int k, double* U = nullptr) {
  constexpr int XC = PB / LPR;  // columns per thread: k + LPR i + h
  const int t = threadIdx.x;
  const int r = k + t / LPR, h = t % LPR, nthr = (SB - k) * LPR;
  if (r >= SB) return PB;
  double x[XC];
#pragma unroll
  for (int i = 0; i < XC; i++) x[i] = S[(k + LPR * i + h) * SP + r];
  int nfin = PB;
#pragma unroll
  for (int j = 0; j < PB; j++) {
    asm volatile("bar.sync 1, %0;\n" ::"r"(nthr) : "memory");  // column j is in shared memory
    const double* cb = S + (k + j) * SP;
    const double d = cb[k + j];
    if (nfin == PB) {
      if (!positive(d)) {
        nfin = j;
      } else {
        double u = cb[r];
        if (recip_ok(d)) {
          const double r0 = recip_seed(d), e = fma(-d, r0, 1.0), w = u * r0;
          u = fma(w, fma(e, e, e), w);
        } else {
          u = slow_div(u, d);
        }
        if (U && h == 0) U[j * SP + r] = u;
        if (j + 1 < PB) {  // the next column first: it is stored before the row's other FMAs
          const int i1 = (j + 1) / LPR, h1 = (j + 1) % LPR;
          if (h >= h1) x[i1] = fma(-u, cb[k + LPR * i1 + h], x[i1]);
          if (h == h1) S[(k + j + 1) * SP + r] = x[i1];
#pragma unroll
          for (int i = i1 + 1; i < XC; i++) x[i] = fma(-u, cb[k + LPR * i + h], x[i]);
        }
      }
    }
  }
  return nfin;
}

}  // namespace
