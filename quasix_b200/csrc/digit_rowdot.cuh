// Integer arithmetic of the digit kernel's row-dot epilogue (k_digits.cu):
// sums of products of a 56-bit and a 63-bit integer from 32-bit words.
// Plain C++ apart from one intrinsic, so that it can be run on the host.
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
QX_HD int clz64(uint64_t x) { return __clzll((int64_t)x); }
#else
QX_HD int clz64(uint64_t x) { return x ? __builtin_clzll(x) : 64; }
#endif

// X = 2^28 hi + lo, |X| < 0.996 2^55: |lo| <= 2^27, |hi| < 0.997 2^27.
constexpr int XBITS = 28;
struct Words {
  int lo, hi;
};
QX_HD Words x_words(int64_t v) {
  Words w;
  w.lo = (int)((uint32_t)v << (32 - XBITS)) >> (32 - XBITS);
  w.hi = (int)((v - w.lo) >> XBITS);
  return w;
}

// y = 2^32 hi + lo, lo signed.  hi takes a carry when bit 31 of y is set: |y|
// < 2^63 - 2^31, or it would wrap.
QX_HD Words y_words(int64_t v) {
  Words w;
  w.lo = (int)(uint32_t)v;
  w.hi = (int)((uint32_t)(int32_t)(v >> 32) - (uint32_t)(w.lo >> 31));
  return w;
}

// The sums of a row stand in units of their columns' scales; dn (0 .. 63) is how
// far a column's scale lies below the largest of the 64.  The row is
// normalised in the units of that largest scale; where no column lies further
// below than NEAR, by the sums as they are (dn 0), which costs NEAR bits at most.
constexpr int NEAR = 3;

// The bits of |s| in these units (ones' complement), for the OR over a row.
QX_HD uint64_t top_bits(int64_t s, int dn) {
  const int64_t h = s >> dn;
  return (uint64_t)(h ^ (h >> 63));
}

// Shift by which a row's sums (|s| < 2^62) take 62 bits: one bit is left for the
// carry into the high word.  (With 63 bits a sum within 2^31 of 2^63 came out
// with the wrong sign.)
QX_HD int norm_shift(uint64_t top) { return clz64(top) - 2; }

// The sum shifted up by z in these units.  (With the shift taken from the sums
// as they are, a column of small scale and large sum left the others, and itself
// after its own shift down, that many bits fewer.)
QX_HD int64_t aligned(int64_t s, int z, int dn) {
  const int up = z - dn;
  return up >= 0 ? (int64_t)((uint64_t)s << up) : s >> -up;
}

// The sum of TERMS products X y, |y| <= 2^62, in units of 2^60, without the
// product of the low words: |hi hi| <= 2^57, |hi lo| <= 2^58, |lo hi| <= 2^57,
// and TERMS of each stay below 2^63.  The middle sums join as a whole, rounded
// to nearest: floors of each product added up to an error of one sign, 32 units
// per 16 terms at most.
constexpr int TERMS = 16, UNIT = 60;
struct Sum {
  int64_t hh = 0, hl = 0, lh = 0;
  QX_HD void add(int xlo, int xhi, int64_t y) {
    const Words w = y_words(y);
    hh += (int64_t)xhi * w.hi;
    hl += (int64_t)xhi * w.lo;
    lh += (int64_t)xlo * w.hi;
  }
  template <int B>
  QX_HD static int64_t rounded(int64_t m) {
    return (m >> B) + ((m >> (B - 1)) & 1);
  }
  QX_HD int64_t result() const { return hh + rounded<32>(hl) + rounded<XBITS>(lh); }
};

}  // namespace rowdot
}  // namespace qx
