// FP64 numbers as seven balanced base-256 digits (the method: fp64_tc.cu): from an element to its
// BF16 digits, and from the sums of the products of one order back to FP64.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace {

constexpr int ND = 7;                         // digits per element
constexpr int NG = 8;                         // product orders kept
constexpr int EXP_NONFINITE = 1 << 28;        // row exponent of a row with an infinity or NaN

// The digits of the element with bits b in a row of exponent e as one integer: 128 added at each,
// so that they are its bytes less 128 (the top one 0..256).  shift: -e, and what the element's exponent
// is moved by.  An element below 2^-56 of the row's scale rounds to 0.
__device__ __forceinline__ unsigned long long digit_fixed(unsigned long long b, int shift) {
  const int be = (int)((b >> 52) & 0x7FF);
  unsigned long long m = b & 0xFFFFFFFFFFFFFull;
  if (be) m |= 1ull << 52;
  const int sh = max(be, 1) - 1020 + shift;  // X = m 2^sh < 2^55: sh <= 2 but for subnormal elements
  if (sh >= 0) m <<= min(sh, 63);
  else m = sh < -55 ? 0ull : (m + (1ull << (-sh - 1))) >> (-sh);
  return ((b >> 63) ? 0ull - m : m) + 0x0080808080808080ull;
}
// The byte of w that `sel` picks, less 128, as a float: 2^23 + byte is an FP32 number.
template <int SEL>
__device__ __forceinline__ uint32_t digit_float(uint32_t w) {
  return __float_as_uint(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540 | SEL)) - 8388736.f);
}
// The same digit of x0 and x1 as two BF16 (an integer of magnitude <= 128 is exact in it: the upper
// half of its FP32 encoding).  Digit 0 is the top one, 0..256 before the 128 are taken off.
template <int S>
__device__ __forceinline__ uint32_t digit_pair(unsigned long long x0, unsigned long long x1) {
  uint32_t f0, f1;
  if constexpr (S == 0) {
    f0 = __float_as_uint(__uint_as_float((uint32_t)(x0 >> 48) | 0x4B000000u) - 8388736.f);
    f1 = __float_as_uint(__uint_as_float((uint32_t)(x1 >> 48) | 0x4B000000u) - 8388736.f);
  } else {
    constexpr int B = ND - 1 - S;
    f0 = digit_float<(B & 3)>((uint32_t)(B < 4 ? x0 : x0 >> 32));
    f1 = digit_float<(B & 3)>((uint32_t)(B < 4 ? x1 : x1 >> 32));
  }
  return __byte_perm(f0, f1, 0x7632);
}
// Digits S.. of eight elements, `plane` bytes from one digit to the next.
template <int S>
__device__ __forceinline__ void put_digits(const unsigned long long (&x)[8], uint8_t* p, int plane) {
  *reinterpret_cast<uint4*>(p + S * plane) = make_uint4(digit_pair<S>(x[0], x[1]), digit_pair<S>(x[2], x[3]),
                                                        digit_pair<S>(x[4], x[5]), digit_pair<S>(x[6], x[7]));
  if constexpr (S + 1 < ND) put_digits<S + 1>(x, p, plane);
}

// The eight order sums of one element put together: sum_g G_g 2^(8 (5 - g)) as a 64-bit integer
// (|G_0| <= 2^21, so it stays below 2^62).  Orders 5..7 are added in FP32 first, to within one
// unit of order 5, 2^-54 of 2^(e(i) + e(j)): an FP64 chain over the K products errs by several
// times that.
// SMALL: every |G_g| < 2^22 (K <= 32).  An FP32 addition of 1.5 2^23 leaves such an integer in the low
// bits, where a conversion instruction issues at a quarter of the rate.
template <bool SMALL = false>
__device__ __forceinline__ long long digit_sum(const uint32_t* g, int stride) {
  auto f = [&](int o) { return __uint_as_float(g[o * stride]); };
  auto small_int = [](float x) { return __float_as_int(x + 12582912.f) - 0x4B400000; };
  auto whole = [&](float x) { return SMALL ? small_int(x) : __float2int_rn(x); };
  const int t = whole(fmaf(f(7), 0x1.0p-16f, fmaf(f(6), 0x1.0p-8f, f(5))));
  const int a1 = small_int(f(0)) * 256 + small_int(f(1));  // (2^21 and 2^22 whatever K) < 2^30
  const int a2 = whole(f(2)) * 256 + whole(f(3));          // < 2^31
  return ((long long)a1 << 32) + ((long long)a2 * 65536 + ((long long)whole(f(4)) * 256 + t));
}
// V 2^(es - 54) rounded to FP64 (es = e(i) + e(j)), on the integer pipe and without branches:
// `special` is raised where the result needs digit_value_special.
__device__ __forceinline__ double digit_value(long long V, int es, bool& special) {
  const unsigned long long sg = (unsigned long long)(V >> 63);
  const unsigned long long a = ((unsigned long long)V ^ sg) - sg;
  const int lz = __clzll((long long)a);
  const int be = es + 1023 + 9 - lz;  // V = 1.x 2^(63 - lz)
  special = special || (a != 0 && (unsigned)(be - 1) > 2044u) || es > EXP_NONFINITE / 2;
  const unsigned long long M = a << (lz & 63);
  const unsigned long long r = (M >> 11) + ((M >> 10) & 1u) + ((unsigned long long)(uint32_t)((be - 1) << 20) << 32);
  return a == 0 ? 0.0 : __longlong_as_double((long long)(r | (sg << 63)));
}

}  // namespace
