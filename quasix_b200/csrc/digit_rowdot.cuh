// Integer arithmetic of the digit kernel's row-dot epilogue (k_digits.cu):
// acc += the part of X y above 2^64, in units of 2^64, from 32-bit words.
// Plain C++ apart from the two intrinsics, so that it can be run on the host.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define QX_HD __host__ __device__ __forceinline__
#else
#define QX_HD inline
#endif

namespace qx {
namespace rowdot {

#ifdef __CUDA_ARCH__
QX_HD int clz32(uint32_t x) { return __clz((int)x); }
QX_HD int mulhi32(int a, int b) { return __mulhi(a, b); }
#else
QX_HD int clz32(uint32_t x) { return x ? __builtin_clz(x) : 32; }
QX_HD int mulhi32(int a, int b) { return (int)(((int64_t)a * b) >> 32); }
#endif

// The integers of b times 2^XSHIFT: |X| < 2^60.
constexpr int XSHIFT = 5;

// v = 2^32 hi + lo, lo signed.  hi takes a carry when bit 31 of v is set: |v|
// < 2^63 - 2^31, or it would wrap.
struct Words {
  int lo, hi;
};
QX_HD Words words(int64_t v) {
  Words w;
  w.lo = (int)(uint32_t)v;
  w.hi = (int)((uint32_t)(int32_t)(v >> 32) - (uint32_t)(w.lo >> 31));
  return w;
}

// The bits of |s| >> 32 (ones' complement), for the OR over a row.
QX_HD uint32_t top_bits(int64_t s) {
  const int h = (int)(s >> 32);
  return (uint32_t)(h ^ (h >> 31));
}

// Shift by which a row's sums (|s| < 2^62) take 62 bits: one bit is left for the
// carry into the high word.  (With 63 bits a sum within 2^31 of 2^63 came out
// with the wrong sign.)
QX_HD int norm_shift(uint32_t top) { return clz32(top) - 2; }

// |X| < 2^60 and |y| < 2^62, so that the sum of 16 terms stays below 2^62 + 2^35.
QX_HD int64_t term(int xlo, int xhi, int64_t y) {
  const Words w = words(y);
  return (int64_t)xhi * w.hi + mulhi32(xhi, w.lo) + mulhi32(xlo, w.hi);
}

}  // namespace rowdot
}  // namespace qx
