// Exact FP64 contractions on the 16-bit tensor cores (shared by the
// reconstruction, recon_tc.cu, and the quadratures of the implicit solve,
// recon_solve.cu).
//
// An operand row or column is scaled by a power of two into an integer of 56
// significant bits and written as seven balanced base-256 digits (the top
// digit in [-256, 256], the others in [-128, 127]), each exact in fp16 (and
// in the bf16 of the tcgen05 kernel).  Digit products of level l = i + k
// accumulate in FP32 through mma.sync m16n8k16, exactly, in chunks of at most
// two or three k-tiles.  Levels l < 7 are kept (the rest lie below 2^-56 of the
// operands' scale), folded exactly (digit_sum.cuh) and rounded once to FP64.
//
// What bounds these tiles is the work around the products: the digits, the
// folds and the roundings.  Start values that make a level's integer readable
// from the accumulator's bit pattern, levels combined in pairs in 32 bits, one
// 64-bit sum and a byte instead of two 64-bit sums and a rounding without a
// normalising shift take a fold and rounding from about 45 instructions to 40
// (30 without the rest, whose price digit_sum.cuh gives),
// the packed fp16 digits those of a pair of values from 39 to 17.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <cstring>
#include <type_traits>
#include <vector>

#include "chn_common.cuh"
#include "digit_sum.cuh"

namespace chn {

inline uint16_t bf16_bits_of_int(int d) {
  const float f = (float)d;  // |d| <= 256: exact in bf16, low 16 bits zero
  uint32_t u;
  std::memcpy(&u, &f, 4);
  return (uint16_t)(u >> 16);
}

// seven balanced base-256 digits of x (|x| < 2^56), most significant first
inline void digits56(long long x, int* d) {
  for (int i = kDig - 1; i >= 1; --i) {
    const long long lo = ((x + 128) & 255) - 128;
    d[i] = (int)lo;
    x = (x - lo) >> 8;
  }
  d[0] = (int)x;
}

// fp16 bit pattern of an integer |d| <= 2048 held as a bf16 bit pattern (the
// host tables): both formats hold every digit exactly
inline uint16_t half_bits_of_bf16_digit(uint16_t b) {
  const uint32_t u = (uint32_t)b << 16;
  float f;
  std::memcpy(&f, &u, 4);
  const __half_raw r = __half_raw(__float2half_rn(f));
  return r.x;
}

// k-tiles per accumulation chunk: append_digit_table finds the most for which
// every level sum stays within +-2^22 whatever the data (a digit of a table
// averages 64 of 128 at most, so two k-tiles have a margin of two; three do
// for most tables)
static constexpr int kChunkKT = 2;     // the Legendre tables (FP64 kernels where a table allows fewer)
static constexpr int kMaxChunkKT = 3;  // the transforms': Grid::tcch

__device__ __forceinline__ void mma_f16_16816(float* d, const uint4& a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// the same with a fresh accumulator c in every element
__device__ __forceinline__ void mma_f16_16816_from(float* d, const uint4& a, uint32_t b0, uint32_t b1, float c) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "f"(c));
}

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}

__device__ __forceinline__ void ldsm_x2(uint32_t addr, uint32_t& r0, uint32_t& r1) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(addr));
}

// biased exponent field of v
__device__ __forceinline__ int exp_field(double v) { return (__double2hiint(v) >> 20) & 0x7FF; }

// the exponent of a column whose largest biased exponent field is ce
// (|v| < 2^col_exp); a column that held an infinity or a NaN (its digits
// carry no meaning) gets one that round_sum turns into NaN
static constexpr int kNanExp = 1 << 20;
__device__ __forceinline__ int col_exp(int ce) { return ce == 0x7FF ? kNanExp : ce - 1022; }

// The (0, 0) line's two real systems (u and w) run as Re and Im of one column of
// a contraction.  They are independent, w often far below u, so each has an
// exponent of its own (eim where `mean`).
__device__ __forceinline__ void column_exponents(const cpx& v, bool mean, int& e, int& eim) {
  const int im = exp_field(v.im);
  e = max(e, max(exp_field(v.re), mean ? 0 : im));
  if (mean) eim = max(eim, im);
}

// v * 2^(56 - ex) as an integer, rounded half away from zero, from the bit
// pattern (integer ops only); ex bounds the column: |v| < 2^ex
__device__ __forceinline__ long long scaled56(double v, int ex) {
  const int hi = __double2hiint(v);
  const int ef = (hi >> 20) & 0x7FF;
  const unsigned long long m =
      (((unsigned long long)((hi & 0xFFFFF) | 0x100000) << 32) | (unsigned)__double2loint(v)) << 4;
  long long x = (long long)(((m >> min(max(ex + 1022 - ef, 0), 63)) + 1) >> 1);
  if (ef == 0) x = 0;  // zero (denormals are below every scale in use)
  return hi < 0 ? -x : x;
}

// a folded sum t (below) scaled by 2^-s, rounded half up
__device__ __forceinline__ long long scaled_sum(long long t, int s) {
  if (s > 0) return ((t >> min(s - 1, 62)) + 1) >> 1;
  return t << min(-s, 63);
}

// the sum (t, r) (digit_sum.cuh) * 2^e, e that of t's unit, rounded once: one
// FP64 conversion, the power of two added to the exponent field.  Zeros,
// results outside the normal range and NaN columns (e >= kNanExp / 2) take the
// multiplications below; bad is set for results that are not finite.
template <class F>
__device__ __forceinline__ double round_sum(F f, long long t, uint32_t r, int e, bool& bad) {
  int up;
  const double v = (double)sum_word(f, t, r, up);
  e -= up;
  const int hi = __double2hiint(v);
  const int ef = hi & 0x7FF00000;
  if (ef != 0 && (unsigned)((ef >> 20) + e - 1) < 2046u) return __hiloint2double(hi + (e << 20), __double2loint(v));
  if (e >= kNanExp / 2) {
    bad = true;
    return __longlong_as_double(0x7FF8000000000000LL);
  }
  const int h = e >> 1;
  const double f0 = __hiloint2double((min(max(h, -1022), 1023) + 1023) << 20, 0);
  const double f1 = __hiloint2double((min(max(e - h, -1022), 1023) + 1023) << 20, 0);
  const double y = v * f0 * f1;
  bad |= exp_field(y) == 0x7FF;
  return y;
}

template <class F>
__device__ __forceinline__ double round_sum(F f, long long t, uint32_t r, int e) {
  bool bad = false;
  return round_sum(f, t, r, e, bad);
}

// the four rests of a tile that wait while the warp runs its next one, PACK: as
// bytes of one register, or (LongFold) halves of two
template <bool PACK, class F>
struct Rests {
  static constexpr int kPer = PACK ? (std::is_same<F, Fold>::value ? 4 : 2) : 1;
  uint32_t v[4 / kPer];
  __device__ __forceinline__ explicit Rests(const uint32_t (&R)[4]) {
    if constexpr (kPer == 4) {
      v[0] = __byte_perm(__byte_perm(R[0], R[1], 0x0040), __byte_perm(R[2], R[3], 0x0040), 0x5410);
    } else if constexpr (kPer == 2) {
      v[0] = __byte_perm(R[0], R[1], 0x5410);
      v[1] = __byte_perm(R[2], R[3], 0x5410);
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r) v[r] = R[r];
    }
  }
  __device__ __forceinline__ uint32_t operator[](int r) const {
    if constexpr (kPer == 4) return __byte_perm(v[0], 0, 0x4440 + r);
    else if constexpr (kPer == 2) return __byte_perm(v[r >> 1], 0, r & 1 ? 0x4432 : 0x4410);
    else return v[r];
  }
};

// of the sum and of the difference of two sums
template <class F>
__device__ __forceinline__ double round_plus(F f, long long ta, uint32_t ra, long long tb, uint32_t rb, int e, bool& bad) {
  long long t;
  uint32_t r;
  sum_plus(ta, ra, tb, rb, t, r);
  return round_sum(f, t, r, e, bad);
}
template <class F>
__device__ __forceinline__ double round_minus(F f, long long ta, uint32_t ra, long long tb, uint32_t rb, int e, bool& bad) {
  long long t;
  uint32_t r;
  sum_minus(f, ta, ra, tb, rb, t, r);
  return round_sum(f, t, r, e, bad);
}

// x is neither infinite nor NaN (integer test on the exponent field)
__device__ __forceinline__ bool finite_bits(double x) { return exp_field(x) != 0x7FF; }

// Balanced digits without a carry chain: with B = sum_{i<6} 128 * 256^i,
// x + B = sum_{q>=1} (d_q + 128) 256^(6-q) + d_0 256^6, so every lower digit
// is an unsigned byte of x + B less 128 and the top digit (in [-256, 256])
// its arithmetic shift by 48.  The digits come out as floats without an
// integer-to-float conversion.  FP32 (the tcgen05 kernel's bf16 digits): for
// 0 <= u < 2^23 the bit pattern 0x4B000000 | u is the float 2^23 + u, so a
// byte b placed under that exponent (one byte permute) less 2^23 + 128 is
// b - 128, exactly (one FP32 add); the top digit goes the same way through
// u = d_0 + 256.  Every digit has at most 8 significant bits, so the float's
// upper half is its exact bf16.
__device__ __forceinline__ void balanced_digits_f32(long long x, float (&f)[kDig]) {
  const long long xb = x + 0x808080808080LL;
  const unsigned lo = (unsigned)xb, hi = (unsigned)(xb >> 32);
  constexpr float kOff = 8388736.0f;  // 2^23 + 128
  // __byte_perm selector 0x765k: byte 0 from byte k of the word, bytes 1-3 from 0x4B000000
  f[6] = __uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7650)) - kOff;
  f[5] = __uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7651)) - kOff;
  f[4] = __uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7652)) - kOff;
  f[3] = __uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7653)) - kOff;
  f[2] = __uint_as_float(__byte_perm(hi, 0x4B000000u, 0x7650)) - kOff;
  f[1] = __uint_as_float(__byte_perm(hi, 0x4B000000u, 0x7651)) - kOff;
  f[0] = __uint_as_float((unsigned)(((int)hi >> 16) + (0x4B000000 + 256))) - 8388864.0f;  // 2^23 + 256
}

// the balanced digits of two values (re, im) as bf16 packed per digit into
// one 32-bit word (re in the low half): out[q * stride] for q = 0..6
__device__ __forceinline__ void digits_pair_bf16(long long xr, long long xi, uint32_t* out, size_t stride) {
  float fr[kDig], fi[kDig];
  balanced_digits_f32(xr, fr);
  balanced_digits_f32(xi, fi);
#pragma unroll
  for (int q = 0; q < kDig; ++q)  // the upper halves of the two floats
    out[(size_t)q * stride] = __byte_perm(__float_as_uint(fr[q]), __float_as_uint(fi[q]), 0x7632);
}

// The same as fp16, two values a word and two digits a permute (17 permutes
// and packed adds for a pair where the bf16 form takes 39): a byte b under
// the exponent of 1024 (0x6400 | b) is 1024 + b, less 1152 it is b - 128; the
// top digit enters the 64-bit sum under 0x6500 (1024 + 256 + d_0).
// WIDE: |x| up to 2^57 (the sum or difference of two 56-bit integers), the top
// digit in [-512, 512] under 0x6600 (1536 + d_0).
template <bool WIDE = false>
__device__ __forceinline__ void digits_pair(long long x0, long long x1, uint32_t* out, size_t stride) {
  constexpr long long kB = WIDE ? 0x6600808080808080LL : 0x6500808080808080LL;
  const long long a = x0 + kB, b = x1 + kB;
  const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32), bl = (uint32_t)b, bh = (uint32_t)(b >> 32);
  constexpr uint32_t kE = 0x64646464u;
  const uint32_t p65 = __byte_perm(al, bl, 0x5140), p43 = __byte_perm(al, bl, 0x7362), p21 = __byte_perm(ah, bh, 0x5140);
  const uint32_t w[kDig] = {__byte_perm(ah, bh, 0x7632), __byte_perm(p21, kE, 0x4342), __byte_perm(p21, kE, 0x4140),
                            __byte_perm(p43, kE, 0x4342), __byte_perm(p43, kE, 0x4140), __byte_perm(p65, kE, 0x4342),
                            __byte_perm(p65, kE, 0x4140)};
#pragma unroll
  for (int q = 0; q < kDig; ++q) {
    const uint32_t off = q == 0 ? (WIDE ? 0xE600E600u : 0xE500E500u) : 0xE480E480u;  // -1536 or -1280, -1152
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;\n" : "=r"(r) : "r"(w[q]), "r"(off));
    out[(size_t)q * stride] = r;
  }
}

// the level sums of one mma accumulator element (acc[l][i], levels 0..6)
// folded into (t, r)
template <class F>
__device__ __forceinline__ void fold_acc(F f, const float (&acc)[kDig][4], int i, long long& t, uint32_t& r) {
  uint32_t b[kDig];
#pragma unroll
  for (int l = 0; l < kDig; ++l) b[l] = __float_as_uint(acc[l][i]);
  fold_bits(f, b, t, r);
}

// of seven exact level sums (the tcgen05 kernel)
__device__ __forceinline__ void fold_levels(const float (&lv)[kDig], long long& t, uint32_t& r) {
  int v[kDig];
#pragma unroll
  for (int l = 0; l < kDig; ++l) v[l] = __float2int_rn(lv[l]);
  fold_ints(Fold(), v, t, r);
}

// lane's ldmatrix address of the digits of the eight columns from n0
// ([digit][column][KS], a digit plane every dstride): matrices 0, 1 are the
// two k halves of a digit, 2, 3 of the next
__device__ __forceinline__ uint32_t tc_row_addr(const uint16_t* dig, size_t KS, size_t dstride, int n0, int lane) {
  return (uint32_t)__cvta_generic_to_shared(dig) +
         (uint32_t)(((lane >> 4) * dstride + (n0 + (lane & 7)) * KS + ((lane >> 3) & 1) * 8) * 2);
}

// the 28 digit products of one k-tile (table fragments af, digits at row;
// dst2 bytes between digit pairs), `first` of a chunk: on fresh accumulators
// (level 6: on acc's)
__device__ __forceinline__ void tc_ktile(const uint4 (&af)[kDig], uint32_t row, uint32_t dst2, float (&acc)[kDig][4],
                                         bool first) {
  uint32_t b0[kDig], b1[kDig];
#pragma unroll
  for (int k = 0; k + 1 < kDig; k += 2) ldsm_x4(row + (k / 2) * dst2, b0[k], b1[k], b0[k + 1], b1[k + 1]);
  ldsm_x2(row + (kDig / 2) * dst2, b0[kDig - 1], b1[kDig - 1]);
#pragma unroll
  for (int i = 0; i < kDig; ++i)
#pragma unroll
    for (int k = 0; k < kDig - i; ++k) {
      if (first && i == 0 && k < kDig - 1)
        mma_f16_16816_from(acc[k], af[i], b0[k], b1[k], __uint_as_float(kAccBits));
      else mma_f16_16816(acc[i + k], af[i], b0[k], b1[k]);
    }
}

__device__ __forceinline__ void tc_load_frags(uint4 (&af)[kDig], const uint4* __restrict__ A) {
#pragma unroll
  for (int i = 0; i < kDig; ++i) af[i] = __ldg(A + i * 32);
}

// level 6 of a chunk's accumulators: what the chunk before left of the sums
__device__ __forceinline__ void acc_begin(float (&acc)[kDig][4], const uint32_t (&R)[4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r) acc[kDig - 1][r] = __uint_as_float(kAccBits + R[r]);
}

static constexpr int kFragStep = kDig * 32;  // uint4 between the k-tiles of a table

// One exact digit GEMM tile of a fixed table A (fragment order
// [mt][KT][7][32][4]) against the smem digits of the eight columns from n0,
// over the k-tiles [k0, k1): exact level sums per chunk of at most `chunk`
// k-tiles, folded into (T, R) per accumulator element (R on entry: added to the
// sum).  The sum is t 2^(e_row + e_col - 64 + fs) and R a fraction of
// it, for operands scaled to 56-bit integers; an empty range gives T = 0.  PF: the table fragments of k-tile
// kt + 1 are loaded while kt's products run (tables that live in L2).
template <bool PF = false, class F>
__device__ __forceinline__ void tc_tile_range(F f, const uint4* __restrict__ A, int mt, int KT, int k0, int k1, int chunk,
                                              const uint16_t* dig, size_t KS, size_t dstride, int n0, int lane,
                                              long long (&T)[4], uint32_t (&R)[4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r) T[r] = 0;
  const uint4* Am = A + (size_t)mt * KT * kFragStep + lane;
  const uint32_t base = tc_row_addr(dig, KS, dstride, n0, lane);
  const uint32_t dst2 = (uint32_t)(4 * dstride);
  uint4 an[kDig];
  if (PF && k0 < k1) tc_load_frags(an, Am + (size_t)k0 * kFragStep);
  for (int kc = k0; kc < k1; kc += chunk) {
    float acc[kDig][4];
    acc_begin(acc, R);
    const int kend = min(k1, kc + chunk);
    auto tile = [&](int kt, bool first) {
      uint4 af[kDig];
      if (PF) {
#pragma unroll
        for (int i = 0; i < kDig; ++i) af[i] = an[i];
        tc_load_frags(an, Am + (size_t)min(kt + 1, k1 - 1) * kFragStep);
      } else {
        tc_load_frags(af, Am + (size_t)kt * kFragStep);
      }
      tc_ktile(af, base + (uint32_t)(kt * 32), dst2, acc, first);
    };
    tile(kc, true);
    for (int kt = kc + 1; kt < kend; ++kt) tile(kt, false);
#pragma unroll
    for (int r = 0; r < 4; ++r) fold_acc(f, acc, r, T[r], R[r]);
  }
}

template <bool PF = false, class F>
__device__ __forceinline__ void tc_tile(F f, const uint4* __restrict__ A, int mt, int KT, int chunk, const uint16_t* dig,
                                        size_t KS, size_t dstride, int n0, int lane, long long (&T)[4],
                                        uint32_t (&R)[4]) {
  tc_tile_range<PF>(f, A, mt, KT, 0, KT, chunk, dig, KS, dstride, n0, lane, T, R);
}

// The same whole tile as one of a sequence that a warp runs with few others
// on its SM, where nothing else hides the tables' L2 latency: pf holds the
// fragments of this tile's first two k-tiles on entry and of the next
// tile's (at An; null: none) on exit, so two k-tiles are always in flight.
// KT >= 2.
struct FragPair {
  uint4 f[2][kDig];
};
__device__ __forceinline__ void tc_stream_start(FragPair& pf, const uint4* __restrict__ Am) {
  tc_load_frags(pf.f[0], Am);
  tc_load_frags(pf.f[1], Am + kFragStep);
}
template <class F>
__device__ __forceinline__ void tc_tile_stream(F f, FragPair& pf, const uint4* __restrict__ Am, const uint4* __restrict__ An,
                                               int KT, uint32_t base, uint32_t dst2, long long (&T)[4], uint32_t (&R)[4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r) T[r] = 0;
  if (An == nullptr) An = Am;  // the last tile: loads that nothing uses
  for (int kc = 0; kc < KT; kc += kChunkKT) {
    float acc[kDig][4];
    acc_begin(acc, R);
    auto tile = [&](int kt, bool first) {
      uint4 af[kDig];
#pragma unroll
      for (int i = 0; i < kDig; ++i) {
        af[i] = pf.f[0][i];
        pf.f[0][i] = pf.f[1][i];
      }
      const int kn = kt + 2;
      tc_load_frags(pf.f[1], kn < KT ? Am + (size_t)kn * kFragStep : An + (size_t)(kn - KT) * kFragStep);
      tc_ktile(af, base + (uint32_t)(kt * 32), dst2, acc, first);
    };
    static_assert(kChunkKT == 2, "two k-tiles a chunk");
    tile(kc, true);
    if (kc + 1 < KT) tile(kc + 1, false);
#pragma unroll
    for (int r = 0; r < 4; ++r) fold_acc(f, acc, r, T[r], R[r]);
  }
}

// host: the exponent of a table row (its entries and their sum bounded)
int digit_row_exponent(const double* row, int K, int top = 256);

// host: digit table of a row-major matrix M[rows][K] in mma A-fragment order
// [MT][KT][7][32 lanes][4] (appended to frag), row exponents appended to ex;
// returns the k-tiles per chunk its level sums allow (0: none).  long_rows: set
// where a row's sum needs LongFold
int append_digit_table(const double* M, int rows, int K, int MT, int KT, std::vector<uint32_t>& frag,
                       std::vector<int>& ex, int top = 256, bool* long_rows = nullptr);

}  // namespace chn
