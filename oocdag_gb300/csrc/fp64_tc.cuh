// FP64 updates on the tensor cores by digit products (fp64_tc.cu).
#pragma once

#include <cstdint>

#include "common.cuh"

constexpr int DIGIT_K = 128;    // columns of X per run (one exponent per row and run)
constexpr int DIGIT_RUNS = 4;   // most runs an update sums before it rounds into C

// Notes of an operand whose values are not known to suit digits (fp64_tc.cu): which elements of a row are large
// (digit_check_bytes(rows, K)), which columns are not all zero (digit_cols_bytes(K), zeroed before launch_digits), and the word that
// launch_digit_check raises (to 1, never lowers) where the rows are too uneven for a product to be as
// accurate as an FP64 sum; an update with such an operand then does nothing.
struct DigitCheck {
  uint32_t* large = nullptr;
  uint32_t* cols = nullptr;
  int* wide = nullptr;
  int least = 1 << 20;  // launch_digits itself raises it at an element below 2^-least of its row's scale in a run
};

// Runs of at most DIGIT_K columns of a column of tiles: element (r, k), r = org .. org + rows - 1,
// k < K, of run q sits at X + (r / nb) * stride + r % nb + (q DIGIT_K + k) * ldx (stride = nb for a plain
// column-major panel); its digits at planes + q * slot.
struct DigitRuns {
  const double* X;
  i64 ldx, stride;
  int nb;
  i64 org, rows;
  int K;                 // columns in all; every run but the last has DIGIT_K
  void* planes;
  size_t slot;           // bytes between the runs' planes, >= digit_plane_bytes of each
  i64 org_of[DIGIT_RUNS];  // row each run's planes start at (org, or a multiple of 128 rows above it)
  // Operands of launch_digit_gemm only.  kshift: element (r, k) enters as x 2^(ksign kshift[k]) (the
  // other operand with the opposite sign).  sym: X is a symmetric matrix given by its lower
  // triangle, rows 0.. and columns k0.. of it (org 0, ld ldx; stride and nb unused).
  const int* kshift = nullptr;
  int ksign = 0;
  int sym = 0;
  i64 k0 = 0;
  const int* only_if = nullptr;  // planes are rewritten only where this word is not 0 (with kshift)
  DigitCheck chk;  // (launch_digit_update's operands as well)
};

// Bytes of the digit planes and row exponents of `rows` rows of K columns.
size_t digit_plane_bytes(i64 rows, int K);

// The planes of every run of X for rows org.. (sets org_of; any number of runs for
// launch_digit_gemm, at most DIGIT_RUNS for launch_digit_update).
int launch_digits(DigitRuns& X, const int* status, cudaStream_t s);

size_t digit_check_bytes(i64 rows, int K);
size_t digit_cols_bytes(int K);
// After launch_digits of both operands of a product (the same one twice for a symmetric product), org 0.
int launch_digit_check(const DigitRuns& A, const DigitRuns& B, cudaStream_t s);

// C(org + r, org + c) -= sum over the runs of X(r) X(c)^T, for r < rows, c in [c_lo, c_hi), r >= c, after
// launch_digits: one rounding into C per call.  64 divides C.nb, org and c_lo; columns are
// updated in whole groups of 64, so c_hi is a multiple of 64 or the last row.  X is read
// where a row holds an infinity or NaN.
int launch_digit_update(const DigitRuns& X, const TileMap& C, i64 c_lo, i64 c_hi, const int* status, cudaStream_t s,
                        int reserve_sms = 0);

// C (A.rows x B.rows, ld ldc) = beta C + alpha (sum over the runs of A B^T) after launch_digits of both,
// A.K == B.K, both with org 0 and any number of runs: all of C (mask 0), its lower (1) or its upper (2) triangle.  A zero
// beta leaves C unread.
int launch_digit_gemm(const DigitRuns& A, const DigitRuns& B, double* C, i64 ldc, double alpha, double beta, int mask,
                      int* status, cudaStream_t s);
