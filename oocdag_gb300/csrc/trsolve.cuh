// Triangular solves with a stored factor and the inverses of its diagonal tiles, one launch
// for all right-hand sides and both sweeps (trsolve.cu).
#pragma once

#include "common.cuh"

// Lower factor L (n x n, ld ldl) in panels: nb-wide up to column tail0, then nb2-wide (tail0 >= n:
// uniform nb).  Panel p's Dinv tile holds L_pp^{-T} (upper, ld = the panel's nominal width),
// the tiles stored one after another; any narrower diagonal sub-block of such a tile is the
// inverse of the same sub-block of L.
template <typename T>
struct TriSolve {
  i64 n;
  const T* L;
  i64 ldl;
  const T* Dinv;
  i64 tail0;
  int nb, nb2;
  T* B;      // n x r, overwritten
  i64 ldb;
  int r;
  int sweeps;  // 1: L y = b, 2: L^T x = b, 3: both
};

// Exchange buffer of a solve (n, r) whose launches make both sweeps or one each: zeroed once when allocated; epoch is a number > 0 that no
// earlier launch on the buffer since then has used.
size_t trsolve_bytes(i64 n, int r, int elem_size, int sweeps = 2);
template <typename T>
int launch_trsolve(const TriSolve<T>& a, void* exchange, unsigned epoch, cudaStream_t s);
// The buffer's error word (an int, 0 while every wait has ended), for the host to read after
// the launch is done.
inline const int* trsolve_error(const void* exchange) { return (const int*)exchange + 1; }
