// Workspace of a solve with a stored factor (ooc_dpotrs_L) in a caller's budget.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

// Order of the diagonal blocks whose inverses such a solve keeps, side by side (ld min(64, n)).
constexpr int DPOTRS_BLOCK = 64;
inline size_t dpotrs_inverse_bytes(int64_t n) { return (size_t)n * (size_t)std::min<int64_t>(n, DPOTRS_BLOCK) * 8; }

// Byte offsets into the workspace: exchange words, inverses, B's device copy, two panels.
struct DpotrsPlan {
  bool ok = false;     // the budget (0: none) holds a solve panel by panel
  bool whole = false;  // a factor on the device in one launch
  int group = 0;       // right-hand sides per launch, panel by panel
  size_t least = 0;    // the smallest budget
  size_t inverses = 0, b = 0, panels = 0, panel = 0, need = 0;
};

// exchange(n, r, sweeps): bytes of the exchange buffer of r right-hand sides.  A budget is enough from two panels, an
// nb x nb inverse and 128 nb bytes of right-hand sides on: the panels' inverses and the exchange words
// of eight right-hand sides and one sweep never take more, and 16 go together where there is room.
template <typename Exchange>
DpotrsPlan dpotrs_plan(int64_t n, int nb, int nrhs, bool l_dev, bool b_dev, size_t budget, Exchange exchange) {
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  const size_t b_B = b_dev ? 0 : up((size_t)n * nrhs * 8), b_pan = l_dev ? 0 : up((size_t)n * nb * 8);
  DpotrsPlan p;
  p.least = 256 + up((size_t)nb * nb * 8) + up((size_t)nb * 128) + b_B + 2 * b_pan;
  p.ok = budget == 0 || p.least <= budget;
  if (!p.ok) return p;
  auto lay_out = [&](bool whole, int group) {
    p.whole = whole;
    p.group = group;
    p.panel = b_pan;
    p.inverses = up(whole ? exchange(n, group, 2) : exchange((int64_t)nb, group, 1));
    p.b = p.inverses + up(dpotrs_inverse_bytes(whole ? n : nb));
    p.panels = p.b + b_B;
    p.need = p.panels + 2 * b_pan;
    return budget == 0 || p.need <= budget;
  };
  if (l_dev && lay_out(true, nrhs)) return p;
  if (!lay_out(false, nrhs)) lay_out(false, std::min(nrhs, 8));
  return p;
}
