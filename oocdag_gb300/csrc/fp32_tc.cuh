// FP32 products on the tensor cores by digit products (fp32_tc.cu).
#pragma once

#include "common.cuh"

// A column panel of `rows` rows and K columns (ld ldx), its digits at planes (digit32_bytes(rows, K)
// bytes).
struct Digit32 {
  const float* X;
  i64 ldx;
  i64 rows;
  int K;
  void* planes;
};
size_t digit32_bytes(i64 rows, int K);
int launch_digits32(const Digit32& X, const int* status, cudaStream_t s);

// C(r, c) -= X(r) X(c)^T for r >= c and c in the 128-wide block columns [bj_lo, bj_hi) (bj_hi < 0: all).
int launch_digit32_update(const Digit32& X, float* C, i64 ldc, int bj_lo, int bj_hi, int* status, cudaStream_t s,
                          int reserve_sms);
