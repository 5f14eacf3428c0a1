// The integer arithmetic of the digit GEMMs' sums (tc_common.cuh), plain code
// for the host as well, so that a test without a GPU runs it.
//
// A sum of the kept levels is exact: an integer in units of level 6, up to 71
// bits, held as t 2^fs + r with a 64-bit t and 0 <= r < 2^fs.
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
// t's unit is 2^fs of level 6's.  The sums that a transform keeps between its
// stages are t alone and want the finer one, fs = 8, whose t holds rows of a table
// whose entries, scaled to 56 bits, sum to at most kRowSum 2^56 in magnitude; fs =
// 10 takes longer rows (kLongRowSum: Rp from Ny = 133 on, DFTs past 84 points at
// the earliest) and gives away two bits at 2^-62 of the operands' scale.
template <int N>
struct FixedFold {
  CHN_HD constexpr int shift() const { return N; }
};
using Fold = FixedFold<8>;
using LongFold = FixedFold<10>;
static constexpr double kRowSum = 126.5, kLongRowSum = 506.0;
// level sums' bound: the exact range less what r adds to level 6
static constexpr long long kLevelMax = (1LL << 22) - (1LL << 10);

constexpr uint32_t kPairBits = kAccBits + (kAccBits << 8);  // of two combined start values (mod 2^32)
// what the start values add to a fold
CHN_HD constexpr unsigned long long fold_bias(int fs) {
  return (unsigned long long)(kPairBits >> fs) + ((unsigned long long)kPairBits << (16 - fs)) +
         ((unsigned long long)kPairBits << (32 - fs)) + ((unsigned long long)kAccBits << (48 - fs));
}
// half of t's unit: the first r of a sum that is kept as t alone, rounded
template <class F>
CHN_HD uint32_t fold_half(F f) {
  return 1u << (f.shift() - 1);
}

// Adds a chunk's level sums to t and leaves the rest in r: b the bit patterns
// of the accumulators of levels 0..6, level 6 started at kAccBits + r.
// Adjacent levels combine in 32 bits (|l + 256 l'| < 2^31).
template <class F>
CHN_HD void fold_bits(F f, const uint32_t (&b)[kDig], long long& t, uint32_t& r) {
  const int fs = f.shift();
  const uint32_t u56 = b[6] + (b[5] << 8), u34 = b[4] + (b[3] << 8), u12 = b[2] + (b[1] << 8);
  unsigned long long s = u56 >> fs;
  s += (unsigned long long)u34 * (1u << (16 - fs));
  s += (unsigned long long)u12 * (1u << (32 - fs));
  s += (unsigned long long)b[0] << (48 - fs);
  t += (long long)(s - fold_bias(fs));
  r = u56 & ((1u << fs) - 1);  // (the start values' low bits are zero)
}

// the same of seven integer level sums (the tcgen05 kernel)
template <class F>
CHN_HD void fold_ints(F f, const int (&v)[kDig], long long& t, uint32_t& r) {
  const int fs = f.shift();
  const int p56 = v[6] + v[5] * 256 + (int)r, p34 = v[4] + v[3] * 256, p12 = v[2] + v[1] * 256;
  t += (long long)(p56 >> fs) + (long long)p34 * (1LL << (16 - fs)) + (long long)p12 * (1LL << (32 - fs)) +
       (long long)v[0] * (1LL << (48 - fs));
  r = (uint32_t)p56 & ((1u << fs) - 1);
}

// a + b and a - b of two sums (r < 2^(fs + 1) then)
CHN_HD void sum_plus(long long ta, uint32_t ra, long long tb, uint32_t rb, long long& t, uint32_t& r) {
  t = ta + tb;
  r = ra + rb;
}
template <class F>
CHN_HD void sum_minus(F f, long long ta, uint32_t ra, long long tb, uint32_t rb, long long& t, uint32_t& r) {
  t = ta + ~tb;  // less one, which r returns
  r = ra - rb + (1u << f.shift());
}
// a sum as t alone (of sums that began at fold_half: rounded)
template <class F>
CHN_HD long long sum_whole(F f, long long t, uint32_t r) {
  return t + (r >> f.shift());
}

// bits of |t|: |t| < 2^n (0 for t = 0)
CHN_HD int sum_bits(long long t) {
  const unsigned long long a = (unsigned long long)(t < 0 ? -t : t);
#ifdef __CUDA_ARCH__
  return 64 - __clzll((long long)a);
#else
  return a ? 64 - __builtin_clzll(a) : 0;
#endif
}

// exponent field of t 2^e, a sum of columns with the largest field ce: at least
// 1 for what is not zero; 0x7FF (a column that comes out NaN) past FP64's range and where ce is
CHN_HD int sum_field(long long t, int e, int ce) {
  if (ce == 0x7FF) return 0x7FF;
  const int f = sum_bits(t) + e + 1022;
  return t == 0 ? 0 : (f < 1 ? 1 : (f > 0x7FF ? 0x7FF : f));
}

// The sum as one 64-bit integer whose conversion to FP64 rounds it correctly:
// (t 2^fs + r) = x 2^(fs - up), exactly (fs 10: cut to four units of level 6)
// while |t| < 2^54; from there on an FP64 value ends two bits or more above t's
// last, and a last bit that is set stands for what lies below.
template <class F>
CHN_HD long long sum_word(F f, long long t, uint32_t r, int& up) {
  constexpr int kUp = 8;
  const bool small = (uint32_t)((int)(t >> 32) + 0x00400000) < 0x00800000u;
  up = small ? kUp : 0;
  return small ? (long long)((unsigned long long)t << kUp) + (r >> (f.shift() - kUp)) : sum_whole(f, t, r) | 1;
}

}  // namespace chn
