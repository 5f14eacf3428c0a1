// The pieces of the solve and its transpose for launches with few blocks
// (4-column tiles, one block per SM), where a block has its SM almost to
// itself and latency counts.
#pragma once

#include "chn_common.cuh"
#include "sizes.cuh"
#include "tc_common.cuh"

namespace chn {

__device__ __forceinline__ void copy8_async(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// the factors of the tile's columns (contiguous per kind, from system sys0
// on) into shared memory, in the background of the quadratures; the caller's
// few_contract waits for the copies
template <int NTHR, class S>
__device__ __forceinline__ void stage_factors(const Grid& g, const S& gsz, size_t sys0, int nx, double* luA, double* luB,
                                              double* rdA, double* rdB) {
  auto copy = [&](double* dst, const double* src, int n) {
    for (int i = threadIdx.x; i < n; i += NTHR) copy8_async(dst + i, src + i);
  };
  copy(luA, g.luA + sys0 * gsz.D() * 9, nx * gsz.D() * 9);
  copy(luB, g.luB + sys0 * gsz.R() * 5, nx * gsz.R() * 5);
  copy(rdA, g.rdA + sys0 * gsz.D(), nx * gsz.D());
  copy(rdB, g.rdB + sys0 * gsz.R(), nx * gsz.R());
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// One sweep over the M rows of an elimination chain by a group of NL lanes
// (NL: the band's reach), rows ascending or (DOWN) descending.  An FP64 warp
// instruction occupies its scheduler's FP64 unit for some 64 cycles however
// few lanes are active, so a lane per chain waits for every multiply-add of
// every row (279 a chain of the alpha band at 32x65x32: 23k cycles); here lane
// l of the group owns the rows congruent to l, a row's result goes to the
// group by shuffles and ONE multiply-add updates the next NL rows (8k).
// coef(m, t): what row m's result subtracts from the row t further on; scale(m):
// the pivot's reciprocal (SCALE).  steps: the longest chain's rows of the warp
// (every lane takes part in every shuffle); on: the group's stores.
template <int NL, bool DOWN, bool SCALE, class Coef, class Scale>
__device__ __forceinline__ void chain_sweep(int M, int steps, int l, bool on, double* b, int bstride, Coef coef,
                                            Scale scale) {
  auto row = [&](int n) { return min(max(DOWN ? M - 1 - n : n, 0), M - 1); };
  double acc = b[row(l) * bstride];
  double cf[NL], nb = 0.0, sc = 0.0;
  auto load = [&](int n0) {  // the group's values for steps n0 .. n0 + NL - 1
#pragma unroll
    for (int s = 0; s < NL; ++s) cf[s] = coef(row(n0 + s), NL - ((s - l) & (NL - 1)));
    nb = b[row(n0 + l + NL) * bstride];
    if (SCALE) sc = scale(row(n0 + l));
  };
  load(0);
  for (int n0 = 0; n0 < steps; n0 += NL) {
    double c[NL];
#pragma unroll
    for (int s = 0; s < NL; ++s) c[s] = cf[s];
    const double bn = nb, rs = sc;
    load(n0 + NL);
#pragma unroll
    for (int s = 0; s < NL; ++s) {
      const double v = SCALE ? acc * rs : acc;
      const double x = __shfl_sync(0xffffffffu, v, s, NL);
      if (l == s) {
        if (on && n0 + s < M) b[row(n0 + s) * bstride] = x;
        acc = bn;
      }
      acc = fma(-c[s], x, acc);
    }
  }
}

// Digit-table contractions over the planes of a 4-column tile, all inputs at
// once: load(y, o) gives the thread's column's inputs o[0..4] at plane y (o[2]
// and o[4] only with `all`); table w(q) of input q (digit tables Wt
// [5][ceil(R/16)][KT][7][32][4], exponents WE [5][R]); inputs 0..2 sum into Fa
// (rows < D), 3 and 4 into Fb (rows < R), comb(q, f, v) adding the second and
// third of a sum.  One pass of loads and three barriers for all inputs; a warp
// per 16 rows of Fa or of Fb runs its tables' k-tiles as one stream with two
// in flight.  Quadratures at 32x65x32, one instance: 62k -> 20k cycles a block
// for the forward inputs.  meancol: column 0 of inputs 3 and 4 is the (0, 0)
// line's.  dig: (all ? 5 : 3) inputs' digits and exponents; KP: plane pairs
// a thread holds (Q <= KP 2 NTHR / kTile).  Waits for the block's staged copies.
template <int kTile, int NTHR, int KP, class S, class Load, class Table, class Comb>
__device__ __forceinline__ void few_contract(const S& gsz, const uint32_t* __restrict__ Wt, const int* __restrict__ WE,
                                             bool all, int nx, bool meancol, uint16_t* dig, Load load, Table wq, Comb comb, cpx* Fa,
                                             cpx* Fb) {
  static_assert(kTile == 4, "one 8-column digit tile");
  constexpr int NC = 2 * kTile;
  const int KT = (gsz.Q() + 15) / 16, MTw = (gsz.R() + 15) / 16;
  const size_t KS = (size_t)KT * 16 + 8;
  const int nin = all ? 5 : 3;
  auto slot_of = [&](int q) { return all ? q : (q == 3 ? 2 : q); };
  int* exc = reinterpret_cast<int*>(dig + (size_t)nin * kDig * NC * KS);  // [nin][kTile], mean's Im [2]
  const int own0 = nin * kTile - 3;  // the slot of input q's mean Im: own0 + q
  for (int i = threadIdx.x; i < nin * kTile + 2; i += NTHR) exc[i] = 0;
  __syncthreads();
  const int col = threadIdx.x % kTile, y0 = 2 * (threadIdx.x / kTile);
  constexpr int kStep = 2 * (NTHR / kTile);
  cpx v[KP][2][5];
  {
    int e[5] = {0, 0, 0, 0, 0}, eim[5] = {0, 0, 0, 0, 0};
#pragma unroll
    for (int k = 0; k < KP; ++k)
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int y = y0 + p + k * kStep;
#pragma unroll
        for (int q = 0; q < 5; ++q) v[k][p][q] = cpx{0.0, 0.0};
        if (y < gsz.Q() && col < nx) load(y, v[k][p]);
#pragma unroll
        for (int q = 0; q < 5; ++q) column_exponents(v[k][p][q], q >= 3 && meancol && col == 0, e[q], eim[q]);
      }
    // lanes of a column lie kTile apart
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      if (!all && (q == 2 || q == 4)) continue;
#pragma unroll
      for (int o = 16; o >= kTile; o >>= 1) e[q] = max(e[q], __shfl_xor_sync(0xffffffffu, e[q], o));
      if ((threadIdx.x & 31) < kTile) atomicMax(&exc[slot_of(q) * kTile + col], e[q]);
      if (q >= 3 && eim[q]) atomicMax(&exc[own0 + q], eim[q]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    if (!all && (q == 2 || q == 4)) continue;
    const int ex = exc[slot_of(q) * kTile + col] - 1022;
    const int exi = q >= 3 && meancol && col == 0 ? exc[own0 + q] - 1022 : ex;
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int y = y0 + k * kStep;
      if (y >= KT * 16) break;
      uint32_t* d = reinterpret_cast<uint32_t*>(dig + ((size_t)slot_of(q) * kDig * NC + 2 * col) * KS + y);
      digits_pair(scaled56(v[k][0][q].re, ex), scaled56(v[k][1][q].re, ex), d, NC * KS / 2);
      digits_pair(scaled56(v[k][0][q].im, exi), scaled56(v[k][1][q].im, exi), d + KS / 2, NC * KS / 2);
    }
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  const uint4* __restrict__ W = reinterpret_cast<const uint4*>(Wt) + lane;
  for (int item = warp; item < 2 * MTw; item += NTHR / 32) {
    const bool toA = item < MTw;
    const int mt = toA ? item : item - MTw, N = toA ? gsz.D() : gsz.R();
    const int q0 = toA ? 0 : 3, q1 = toA ? (all ? 3 : 2) : (all ? 5 : 4);
    auto table = [&](int q) { return W + ((size_t)wq(q) * MTw + mt) * KT * kFragStep; };
    cpx f[2];
    FragPair pf;
    tc_stream_start(pf, table(q0));
    for (int q = q0; q < q1; ++q) {
      long long T[4];
      uint32_t R[4] = {0, 0, 0, 0};
      tc_tile_stream(LongFold(), pf, table(q), q + 1 < q1 ? table(q + 1) : nullptr, KT,
                     tc_row_addr(dig + (size_t)slot_of(q) * kDig * NC * KS, KS, (size_t)NC * KS, 0, lane),
                     (uint32_t)(4 * NC * KS), T, R);
      const int ecol = col_exp(exc[slot_of(q) * kTile + t]) - 64 + LongFold().shift();
      const int ecoli = q >= 3 && meancol && t == 0 ? col_exp(exc[own0 + q]) - 64 + LongFold().shift() : ecol;
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int row = min(mt * 16 + gq + 8 * rr, N - 1);
        const int e = WE[(size_t)wq(q) * gsz.R() + row];
        const cpx val = {round_sum(LongFold(), T[2 * rr], R[2 * rr], e + ecol),
                         round_sum(LongFold(), T[2 * rr + 1], R[2 * rr + 1], e + ecoli)};
        f[rr] = q == q0 ? val : comb(q, f[rr], val);
      }
    }
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      const int row = mt * 16 + gq + 8 * rr;
      if (row < N && t < nx) (toA ? Fa : Fb)[row * kTile + t] = f[rr];
    }
  }
  __syncthreads();
}

}  // namespace chn
