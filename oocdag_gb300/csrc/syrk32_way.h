// How the FP32 trailing updates of one panel are made, chosen when the panel is prepared and
// kept for its later block-column ranges: what the work buffer holds afterwards depends on it.
#pragma once

#include <cstddef>

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
