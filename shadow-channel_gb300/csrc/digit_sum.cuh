// The integer arithmetic of the digit GEMMs' sums (tc_common.cuh), plain code
// for the host as well, so that a test without a GPU runs it.
//
// A sum of the kept levels is exact: an integer in units of level 6, up to 71
// bits, held as t 2^kFoldShift + r with a 64-bit t and 0 <= r < 2^kFoldShift.
// What a chunk leaves in r enters the next chunk's level 6 accumulator, and the
// sum is rounded to FP64 once.  Against sums with r rounded off chunk by chunk,
// which added an error of their own, this costs an instruction a fold and ten a
// rounding: 192 instances at 32x65x32 reconstruction 1.116 -> 1.132 ms, inverse
// 2.83 -> 2.86, products 2.74 -> 2.73, solve 1.54 -> 1.58; 16 of 64x65x64
// inverse 2.12 -> 2.19.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define CHN_HD __host__ __device__ __forceinline__
#else
#define CHN_HD inline
#endif

namespace chn {

static constexpr int kDig = 7;      // base-256 digits per operand

// Level accumulators start at 1.5 * 2^23 instead of 0: while a level sum
// stays within +-2^22 the FP32 accumulator is 1.5 * 2^23 + sum exactly and
// its bit pattern is kAccBits + sum, so the integer comes out without a
// float-to-integer conversion.
static constexpr uint32_t kAccBits = 0x4B400000u;
// t's unit: 2^kFoldShift of level 6's
static constexpr int kFoldShift = 8;
static constexpr uint32_t kFoldMask = (1u << kFoldShift) - 1;
// half of t's unit: the first r of a sum that is kept as t alone, rounded
static constexpr uint32_t kFoldHalf = 1u << (kFoldShift - 1);
// level sums' bound: the exact range less what r adds to level 6
static constexpr long long kLevelMax = (1LL << 22) - (1LL << kFoldShift);

constexpr uint32_t kPairBits = kAccBits + (kAccBits << 8);  // of two combined start values (mod 2^32)
constexpr unsigned long long kFoldBias =
    (unsigned long long)(kPairBits >> kFoldShift) + ((unsigned long long)kPairBits << (16 - kFoldShift)) +
    ((unsigned long long)kPairBits << (32 - kFoldShift)) + ((unsigned long long)kAccBits << (48 - kFoldShift));

// Adds a chunk's level sums to t and leaves the rest in r: b the bit patterns
// of the accumulators of levels 0..6, level 6 started at kAccBits + r.
// Adjacent levels combine in 32 bits (|l + 256 l'| < 2^31).
CHN_HD void fold_bits(const uint32_t (&b)[kDig], long long& t, uint32_t& r) {
  const uint32_t u56 = b[6] + (b[5] << 8), u34 = b[4] + (b[3] << 8), u12 = b[2] + (b[1] << 8);
  unsigned long long s = u56 >> kFoldShift;
  s += (unsigned long long)u34 * (1u << (16 - kFoldShift));
  s += (unsigned long long)u12 * (1u << (32 - kFoldShift));
  s += (unsigned long long)b[0] << (48 - kFoldShift);
  t += (long long)(s - kFoldBias);
  r = u56 & kFoldMask;  // (the start values' low bits are zero)
}

// the same of seven integer level sums (the tcgen05 kernel)
CHN_HD void fold_ints(const int (&v)[kDig], long long& t, uint32_t& r) {
  const int p56 = v[6] + v[5] * 256 + (int)r, p34 = v[4] + v[3] * 256, p12 = v[2] + v[1] * 256;
  t += (long long)(p56 >> kFoldShift) + (long long)p34 * (1LL << (16 - kFoldShift)) +
       (long long)p12 * (1LL << (32 - kFoldShift)) + (long long)v[0] * (1LL << (48 - kFoldShift));
  r = (uint32_t)p56 & kFoldMask;
}

// a + b and a - b of two sums (r < 2^(kFoldShift + 1) then)
CHN_HD void sum_plus(long long ta, uint32_t ra, long long tb, uint32_t rb, long long& t, uint32_t& r) {
  t = ta + tb;
  r = ra + rb;
}
CHN_HD void sum_minus(long long ta, uint32_t ra, long long tb, uint32_t rb, long long& t, uint32_t& r) {
  t = ta + ~tb;  // less one, which r returns
  r = ra - rb + (1u << kFoldShift);
}
// a sum as t alone (of sums that began at kFoldHalf: rounded)
CHN_HD long long sum_whole(long long t, uint32_t r) { return t + (r >> kFoldShift); }

// The sum as one 64-bit integer whose conversion to FP64 rounds it correctly:
// (t 2^kFoldShift + r) = x 2^(kFoldShift - up), exactly while |t| < 2^54; from
// there on an FP64 value ends two bits or more above t's last, and a last bit
// that is set stands for what lies below.
CHN_HD long long sum_word(long long t, uint32_t r, int& up) {
  const bool small = (uint32_t)((int)(t >> 32) + 0x00400000) < 0x00800000u;
  up = small ? kFoldShift : 0;
  return small ? (long long)((unsigned long long)t << kFoldShift) + r : sum_whole(t, r) | 1;
}

}  // namespace chn
