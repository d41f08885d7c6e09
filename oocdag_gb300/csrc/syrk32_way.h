// How the FP32 trailing updates of one panel are made, and what room they get in a budget.  The
// choice is made when the panel is prepared and kept for its later block-column ranges: what the
// work buffer holds afterwards depends on it.
#pragma once

#include <cstddef>
#include <cstdint>

enum class Syrk32Way {
  kNone,    // nothing prepared
  kDirect,  // FP32 pipe on the panel itself
  kCopied,  // FP32 pipe on an aligned copy in the buffer
  kDigits   // tensor cores, the panel's digit planes in the buffer
};

// `work` is grown for the way taken.  Without room for the planes the FP32 pipe does it; 0, or the
// buffer's error where the copy that it needs finds no room either.
template <typename Buf>
int syrk32_choose(Buf& work, bool digits_serve, size_t digit_bytes, bool aligned, size_t copy_bytes, Syrk32Way* way) {
  if (digits_serve && work.ensure(digit_bytes) == 0) {
    *way = Syrk32Way::kDigits;
    return 0;
  }
  *way = aligned ? Syrk32Way::kDirect : Syrk32Way::kCopied;
  const int rc = aligned ? 0 : work.ensure(copy_bytes);
  if (rc) *way = Syrk32Way::kNone;
  return rc;
}

// Bytes of the largest preparation in a factorization of order n with tiles of nb columns in panels of w <= nb:
// bytes(rows, columns) for the updates inside the first tile by its first panel, and right of it by all of it.
template <typename Bytes>
size_t syrk32_largest(int64_t n, int nb, int w, Bytes bytes) {
  size_t b = 0;
  if (w < nb && n > w) b = bytes(n - w, w);
  if (n > nb) {
    const size_t whole = bytes(n - nb, nb);
    b = whole > b ? whole : b;
  }
  return b;
}

// Panel width of an out-of-core FP32 factorization (0: not even nb columns fit): the widest multiple of nb with 3 n W
// floats within the budget.  *planes: an update's digit planes (plane_bytes(rows, columns), at most `chunk`
// columns at a time) fit beside them.  Up to a quarter of the width is given for them: the update by
// tensor cores takes a third of the FP32 pipe's time, but a narrower panel reads the earlier columns more often.
template <typename PlaneBytes>
int64_t spotrf_ooc_width(int64_t n, int nb, size_t budget, PlaneBytes plane_bytes, int chunk, bool* planes) {
  const size_t per_column = (size_t)3 * n * sizeof(float);
  const int64_t widest = (int64_t)(budget / per_column) / nb * nb;
  *planes = false;
  for (int64_t W = widest; W >= nb && 4 * W >= 3 * widest; W -= nb)
    if (per_column * W + plane_bytes(n, (int)(W < chunk ? W : chunk)) <= budget) {
      *planes = true;
      return W;
    }
  return widest < nb ? 0 : widest;
}
