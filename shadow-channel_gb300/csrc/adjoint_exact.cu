// Exact discrete adjoint of the homogeneous tangent step: the transpose of
// one RK3 substage of the tangent (channel/channel.c:546-573 with
// channel/pass1.c:140-210 and channel/increproject*.c), taken with respect to
// the Euclidean inner product of the real and imaginary parts of every
// coefficient.  The reference's own adjoint (channel/channel.c:596-696) runs
// the continuous adjoint equations with reversed RK coefficients and is not
// this transpose; its dot products <lambda, T v> and <T^T lambda, v> agree
// only to the discretisation error.
//
// A tangent substage k maps (c_in, u_in) -> (c_out, u_out):
//   c1 = E_0 c_in (k == 0) or c_in,  F = Quad(H(u_in)),  c2 = c1 + dt c_k F,
//   x  = L_k^{-1} c2 (plus the homogeneous flux correction of the mean mode),
//   u_out = Recon(x),  c_out = E_{k+1} x + dt d_{k+1} F (k < 2) or x.
// k_solve_T runs the reverse of everything but the products:
//   x_bar = Recon^T(u_out_bar) + E_{k+1}^T c_out_bar (or c_out_bar),
//   F_bar = dt d_{k+1} c_out_bar,  x_bar <- flux^T x_bar,  c2_bar = L^{-T} x_bar,
//   F_bar += dt c_k c2_bar,  c_in_bar = E_0^T c2_bar (or c2_bar),
//   H_bar = Quad^T(F_bar)  (written pre-scaled for the inverse transform),
// and the products kernel (k_products_adj with `exact`) takes H_bar's
// physical fields to u_in_bar.
#include <type_traits>

#include "chn_common.cuh"
#include "few_tile.cuh"
#include "kernels.h"
#include "sizes.cuh"
#include "solve_common.cuh"
#include "tc_common.cuh"

namespace chn {

static constexpr int kThreads = 256;
static constexpr int kTile = 16;  // kx columns per block

__device__ __forceinline__ bool blocked_t(const uint32_t* status, int sdiv, int inst) {
  return status != nullptr && (status[inst / sdiv] & ST_CFL) != 0;
}

__device__ __forceinline__ void cfma_t(double w, const cpx& a, double& re, double& im) {
  re = fma(w, a.re, re);
  im = fma(w, a.im, im);
}

// row m of A^T y for a banded every-other-diagonal A (row i holds A[i][j] at
// column i + 2(j - dl), valid j as in channel/mvOps.c:198-220)
__device__ __forceinline__ cpx band_matvecT_row(const double* __restrict__ A, int w, int dl, int du, int N,
                                                const cpx* y, int ystride, int m) {
  double re = 0.0, im = 0.0;
  for (int j = 0; j <= dl + du; ++j) {
    const int i = m + 2 * (dl - j);
    if (i < 0 || i >= N) continue;
    int j0 = dl - i / 2;
    if (j0 < 0) j0 = 0;
    int j1 = (N - i + 1) / 2 + dl;
    if (j1 > dl + du + 1) j1 = dl + du + 1;
    if (j < j0 || j >= j1) continue;
    const double a = __ldg(A + (size_t)i * w + j);
    const cpx v = y[i * ystride];
    re = fma(a, v.re, re);
    im = fma(a, v.im, im);
  }
  return cpx{re, im};
}

// A^T y = b for one parity chain, A = L U the no-pivot factors of
// channel/mvOps.c:29-91 (L unit lower in columns j < dl, U in dl..dl+du):
// U^T w = b ascending, then L^T y = w descending; RD the reciprocal pivots
// (the forward chain multiplies by them too).  As band_solve_chain.
template <int W, int DL, int DU>
__device__ __forceinline__ void band_solveT_chain(const double* __restrict__ LU, const double* __restrict__ RD, int N,
                                   int par, double* b, int bstride) {
  const int M = (N - par + 1) / 2;  // rows of this parity: i = par + 2 m
  if (M <= 0) return;
  constexpr int G = kChainRows;
  {
    // f[q][t]: what the result of row n0 + q subtracts from the row t + 1 further on
    double f[G][DU], v[G], p[G], acc[DU];
    auto load = [&](int n0) {
#pragma unroll
      for (int q = 0; q < G; ++q) {
        const int m = min(n0 + q, M - 1);
#pragma unroll
        for (int t = 1; t <= DU; ++t) f[q][t - 1] = __ldg(LU + (size_t)(par + 2 * m) * W + DL + t);
        p[q] = __ldg(RD + par + 2 * m);
        v[q] = b[(par + 2 * min(m + DU, M - 1)) * bstride];
      }
    };
#pragma unroll
    for (int t = 0; t < DU; ++t) acc[t] = b[(par + 2 * min(t, M - 1)) * bstride];
    load(0);
    for (int n0 = 0; n0 < M; n0 += G) {
      double c[G][DU], w[G], r[G];
#pragma unroll
      for (int q = 0; q < G; ++q) {
#pragma unroll
        for (int t = 0; t < DU; ++t) c[q][t] = f[q][t];
        w[q] = v[q];
        r[q] = p[q];
      }
      load(n0 + G);
#pragma unroll
      for (int q = 0; q < G; ++q) {
        const double x = acc[0] * r[q];
#pragma unroll
        for (int t = 0; t + 1 < DU; ++t) acc[t] = fma(-c[q][t], x, acc[t + 1]);
        acc[DU - 1] = fma(-c[q][DU - 1], x, w[q]);
        if (n0 + q < M) b[(par + 2 * (n0 + q)) * bstride] = x;
      }
    }
  }
  {
    // f[q][t]: what the result of row n0 + q subtracts from the row t + 1 further on
    double f[G][DL], v[G], acc[DL];
    auto load = [&](int n0) {
#pragma unroll
      for (int q = 0; q < G; ++q) {
        const int m = max(M - 1 - (n0 + q), 0);
#pragma unroll
        for (int t = 1; t <= DL; ++t) f[q][t - 1] = __ldg(LU + (size_t)(par + 2 * m) * W + DL - t);
        v[q] = b[(par + 2 * max(m - DL, 0)) * bstride];
      }
    };
#pragma unroll
    for (int t = 0; t < DL; ++t) acc[t] = b[(par + 2 * max(M - 1 - t, 0)) * bstride];
    load(0);
    for (int n0 = 0; n0 < M; n0 += G) {
      double c[G][DL], w[G];
#pragma unroll
      for (int q = 0; q < G; ++q) {
#pragma unroll
        for (int t = 0; t < DL; ++t) c[q][t] = f[q][t];
        w[q] = v[q];
      }
      load(n0 + G);
#pragma unroll
      for (int q = 0; q < G; ++q) {
        const double x = acc[0];
#pragma unroll
        for (int t = 0; t + 1 < DL; ++t) acc[t] = fma(-c[q][t], x, acc[t + 1]);
        acc[DL - 1] = fma(-c[q][DL - 1], x, w[q]);
        if (n0 + q < M) b[(par + 2 * (M - 1 - (n0 + q))) * bstride] = x;
      }
    }
  }
}

struct SolveTSmem {
  cpx* hc;     // [Qh][kTile][6] parity-combined inputs of Recon^T
  cpx* ra;     // [R][kTile] alpha cotangents (aliases hc)
  cpx* rb;     // [R][kTile]
  cpx* Fa;     // [D][kTile] Recon^T alpha part, then F_bar alpha
  cpx* Fb;     // [R][kTile]
  // the FEW build's: digits (dig; hc unused), staged factors
  uint16_t* dig;
  double *luA, *luB, *rdA, *rdB;  // [tile][D][9], [tile][R][5], [tile][D], [tile][R]
};


// bytes of the tensor-core digits: Recon^T's [7][32][Q pad] (+ exponents),
// Quad^T's two [7][32][R pad] (+ exponents)
__host__ __device__ inline size_t solveT_tc_bytes(const Grid& g) {
  const size_t rq = (size_t)kDig * 32 * ((g.Q + 15) / 16 * 16 + 8) * 2 + (kTile + 1) * sizeof(int);
  const size_t qt = (size_t)2 * kDig * 32 * ((g.R + 15) / 16 * 16 + 8) * 2 + (2 * kTile + 1) * sizeof(int);
  return rq > qt ? rq : qt;
}

__host__ __device__ inline size_t solveT_hc_elems(const Grid& g) {
  size_t hc = (size_t)g.Qh * kTile * 6, r = 2 * (size_t)g.R * kTile;
  const size_t tc = (solveT_tc_bytes(g) + sizeof(cpx) - 1) / sizeof(cpx);
  if (tc > hc) hc = tc;
  return hc > r ? hc : r;
}

static size_t solveT_smem_bytes(const Grid& g) {
  return (solveT_hc_elems(g) + (size_t)g.D * kTile + (size_t)g.R * kTile) * sizeof(cpx);
}

// the FEW build's plan: digits (Recon^T's five inputs, then Quad^T's two),
// right-hand sides, F, the tile's factors
__host__ __device__ inline size_t solveT_few_dig_bytes(const Grid& g, int tile) {
  const size_t rt = (size_t)5 * kDig * 2 * tile * ((g.Q + 15) / 16 * 16 + 8) * 2;
  const size_t qt = (size_t)2 * kDig * 2 * tile * ((g.R + 15) / 16 * 16 + 8) * 2;
  return ((rt > qt ? rt : qt) + (5 * tile + 2) * sizeof(int) + 15) / 16 * 16;
}
static size_t solveT_few_smem_bytes(const Grid& g, int tile) {
  return solveT_few_dig_bytes(g, tile) + (size_t)tile * (3 * g.R + g.D) * sizeof(cpx) +
         (size_t)tile * (10 * g.D + 6 * g.R) * sizeof(double);
}
template <int TT>
__device__ inline SolveTSmem carve_solveT_few(const Grid& g, unsigned char* base) {
  SolveTSmem s;
  s.hc = nullptr;
  s.dig = reinterpret_cast<uint16_t*>(base);
  cpx* p = reinterpret_cast<cpx*>(base + solveT_few_dig_bytes(g, TT));
  s.ra = p; p += (size_t)g.R * TT;
  s.rb = p; p += (size_t)g.R * TT;
  s.Fa = p; p += (size_t)g.D * TT;
  s.Fb = p; p += (size_t)g.R * TT;
  s.luA = reinterpret_cast<double*>(p);
  s.luB = s.luA + (size_t)TT * g.D * 9;
  s.rdA = s.luB + (size_t)TT * g.R * 5;
  s.rdB = s.rdA + (size_t)TT * g.D;
  return s;
}

__device__ inline SolveTSmem carve_solveT(const Grid& g, unsigned char* base) {
  SolveTSmem s;
  cpx* p = reinterpret_cast<cpx*>(base);
  s.hc = p;
  s.ra = p;
  s.rb = p + (size_t)g.R * kTile;
  p += solveT_hc_elems(g);
  s.Fa = p; p += (size_t)g.D * kTile;
  s.Fb = p;
  return s;
}

// the mean line's: R^T (u + i w) and R'^T (du + i dw), both real lines (its
// imaginary parts never reach the fields); a non-finite one makes its line NaN
__device__ __forceinline__ cpx recon_T_mean_input(const cpx& u, const cpx& w) {
  return cpx{exp_field(u.im) == 0x7FF ? u.im : u.re, exp_field(w.im) == 0x7FF ? w.im : w.re};
}

// Recon^T of the velocity cotangent of columns x0.. (the mean line: recon_T_mean_input):
//   alpha_bar = Q^T v_bar - Q'^T Xp_bar + Q''^T dx_bar   (rows < D) -> s.Fa
//   beta_bar  = R^T Zp_bar + R'^T dz_bar                 (rows < R) -> s.Fb
// with Xp_bar = (i kx u_bar + i kz w_bar)/K2, Zp_bar = (i kz u_bar - i kx w_bar)/K2,
// dx_bar = -(i kx du_bar + i kz dw_bar)/K2, dz_bar = (i kz du_bar - i kx dw_bar)/K2
// (the transpose of channel/initAlphaBeta2.c:12-240).  The sums over the
// Gauss planes pair y with -y as the quadratures of k_solve do.
__device__ void recon_T_tile(const Grid& g, const cpx* __restrict__ Ub, int z, int x0, int nx, int xfirst,
                             SolveTSmem& s) {
  const int lx = threadIdx.x % kTile, grp = threadIdx.x / kTile, ngrp = blockDim.x / kTile;
  const size_t cs = (size_t)g.Q * g.X;
  const cpx* Uz = Ub + (size_t)z * 5 * cs;
  for (int phase = 0; phase < 2; ++phase) {
    const int nin = phase == 0 ? 3 : 2;
    for (int i = threadIdx.x; i < g.Qh * kTile; i += blockDim.x) {
      const int yp = i / kTile, l = i - yp * kTile;
      cpx* dst = s.hc + (size_t)i * 6;
      if (l >= nx) continue;
      const int x = x0 + l;
      const double ax = g.kxK2[(size_t)z * g.X + x], az = g.kzK2[(size_t)z * g.X + x];
      const int ya = yp, yb = g.Q - 1 - yp;
      cpx in[2][3];
      for (int side = 0; side < 2; ++side) {
        const int y = side ? yb : ya;
        const cpx u = Uz[0 * cs + (size_t)y * g.X + x], w = Uz[2 * cs + (size_t)y * g.X + x];
        const cpx du = Uz[3 * cs + (size_t)y * g.X + x], dw = Uz[4 * cs + (size_t)y * g.X + x];
        if (phase == 0) {
          in[side][0] = Uz[1 * cs + (size_t)y * g.X + x];
          in[side][1].re = -fma(ax, u.im, az * w.im);  // Xp_bar = i(ax u + az w)
          in[side][1].im = fma(ax, u.re, az * w.re);
          in[side][2].re = fma(ax, du.im, az * dw.im);  // dx_bar = -i(ax du + az dw)
          in[side][2].im = -fma(ax, du.re, az * dw.re);
        } else {
          in[side][0].re = fma(ax, w.im, -az * u.im);  // Zp_bar = i(az u - ax w)
          in[side][0].im = fma(az, u.re, -ax * w.re);
          in[side][1].re = fma(ax, dw.im, -az * du.im);  // dz_bar = i(az du - ax dw)
          in[side][1].im = fma(az, du.re, -ax * dw.re);
          if (l < xfirst) {
            in[side][0] = recon_T_mean_input(u, w);
            in[side][1] = recon_T_mean_input(du, dw);
          }
        }
      }
      for (int q = 0; q < nin; ++q) {
        if (ya == yb) {  // centre plane of an odd point count
          dst[2 * q] = in[0][q];
          dst[2 * q + 1] = in[0][q];
        } else {
          dst[2 * q].re = in[0][q].re + in[1][q].re;
          dst[2 * q].im = in[0][q].im + in[1][q].im;
          dst[2 * q + 1].re = in[0][q].re - in[1][q].re;
          dst[2 * q + 1].im = in[0][q].im - in[1][q].im;
        }
      }
    }
    __syncthreads();
    if (lx < nx) {
      const int N = phase == 0 ? g.D : g.R;
      constexpr int MAXR = 4;
      for (int ib = grp; ib < N; ib += ngrp * MAXR) {
        double sr[MAXR], si[MAXR];
#pragma unroll
        for (int m = 0; m < MAXR; ++m) { sr[m] = 0.0; si[m] = 0.0; }
        const bool even = (ib & 1) == 0;
        for (int yp = 0; yp < g.Qh; ++yp) {
          const cpx* src = s.hc + ((size_t)yp * kTile + lx) * 6;
          if (phase == 0) {
            // even rows: Q, Q'' (even bases) with "+", Q' (odd basis) with "-"
            const cpx V = src[even ? 0 : 1];
            const cpx Xp = src[even ? 3 : 2];
            const cpx Dx = src[even ? 4 : 5];
#pragma unroll
            for (int m = 0; m < MAXR; ++m) {
              const int i = ib + m * ngrp;
              if (i < N) {
                const size_t o = (size_t)yp * g.D + i;
                cfma_t(__ldg(g.Bq + o), V, sr[m], si[m]);
                cfma_t(-__ldg(g.Bqp + o), Xp, sr[m], si[m]);
                cfma_t(__ldg(g.Bqpp + o), Dx, sr[m], si[m]);
              }
            }
          } else {
            const cpx Zp = src[even ? 0 : 1];
            const cpx Dz = src[even ? 3 : 2];
#pragma unroll
            for (int m = 0; m < MAXR; ++m) {
              const int i = ib + m * ngrp;
              if (i < N) {
                const size_t o = (size_t)yp * g.R + i;
                cfma_t(__ldg(g.Br + o), Zp, sr[m], si[m]);
                cfma_t(__ldg(g.Brp + o), Dz, sr[m], si[m]);
              }
            }
          }
        }
#pragma unroll
        for (int m = 0; m < MAXR; ++m) {
          const int i = ib + m * ngrp;
          if (i >= N) continue;
          (phase == 0 ? s.Fa : s.Fb)[i * kTile + lx] = cpx{sr[m], si[m]};
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// the transposed contractions on the tensor cores (tc_common.cuh), the
// scheme of the forward quadratures (quad_rhs_tc in recon_solve.cu)
// ---------------------------------------------------------------------------

static constexpr int kTRegs = 8;  // plane inputs a thread keeps in registers (Q <= 128)

// comb(row, col, v) for rows < N and columns col < nx of the contraction of
// table b (row-major [rows][Q] digits: [b][ceil(R/16)][KT][7][32][4], row
// exponents TE[b * R + row]) with the per-column plane inputs in(y, col)
// (Re and Im as two GEMM columns sharing the column exponent; meancol: column 0
// is the (0, 0) line's, an exponent each)
template <class S, typename In, typename Comb>
__device__ void contract_planes_tc(const Grid& g, const S& gsz, const uint4* __restrict__ T, const int* __restrict__ TE,
                                   int b, int N, int nx, bool meancol, In input, Comb comb, uint16_t* dig, int* exc) {
  const int KT = (gsz.Q() + 15) / 16, MTw = (gsz.R() + 15) / 16;
  const size_t KS = (size_t)KT * 16 + 8;
  for (int i = threadIdx.x; i < kTile + 1; i += blockDim.x) exc[i] = 0;
  auto own = [&](int col) { return meancol && col == 0; };
  __syncthreads();
  if (KT <= kTRegs && blockDim.x == 16 * kTile) {
    const int col = threadIdx.x % kTile, y0 = 2 * (threadIdx.x / kTile);
    auto plane = [&](int k) { return y0 + 32 * (k >> 1) + (k & 1); };  // plane pairs, as quad_rhs_tc
    cpx vin[kTRegs];
    int emax = 0, eim = 0;
#pragma unroll
    for (int k = 0; k < kTRegs; ++k) {
      const int y = plane(k);
      vin[k] = (y < gsz.Q() && col < nx) ? input(y, col) : cpx{0.0, 0.0};
      column_exponents(vin[k], own(col), emax, eim);
    }
    if (emax) atomicMax(&exc[col], emax);
    if (eim) atomicMax(&exc[kTile], eim);
    __syncthreads();
    const int ex = exc[col] - 1022, exi = own(col) ? exc[kTile] - 1022 : ex;
#pragma unroll
    for (int k = 0; k < kTRegs; k += 2) {
      const int y = plane(k);
      if (y >= KT * 16) break;
      uint32_t* d = reinterpret_cast<uint32_t*>(dig + (size_t)(2 * col) * KS + y);
      digits_pair(scaled56(vin[k].re, ex), scaled56(vin[k + 1].re, ex), d, 16 * KS);
      digits_pair(scaled56(vin[k].im, exi), scaled56(vin[k + 1].im, exi), d + KS / 2, 16 * KS);
    }
  } else {
    for (int i = threadIdx.x; i < gsz.Q() * kTile; i += blockDim.x) {
      const int y = i / kTile, col = i - y * kTile;
      if (col >= nx) continue;
      const cpx v = input(y, col);
      int e = 0, eim = 0;
      column_exponents(v, own(col), e, eim);
      if (e) atomicMax(&exc[col], e);
      if (eim) atomicMax(&exc[kTile], eim);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < KT * 8 * kTile; i += blockDim.x) {
      const int y = 2 * (i / kTile), col = i % kTile;
      const cpx v0 = (y < gsz.Q() && col < nx) ? input(y, col) : cpx{0.0, 0.0};
      const cpx v1 = (y + 1 < gsz.Q() && col < nx) ? input(y + 1, col) : cpx{0.0, 0.0};
      const int ex = exc[col] - 1022, exi = own(col) ? exc[kTile] - 1022 : ex;
      uint32_t* d = reinterpret_cast<uint32_t*>(dig + (size_t)(2 * col) * KS + y);
      digits_pair(scaled56(v0.re, ex), scaled56(v1.re, ex), d, 16 * KS);
      digits_pair(scaled56(v0.im, exi), scaled56(v1.im, exi), d + KS / 2, 16 * KS);
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  const int NT = (2 * nx + 7) / 8, MTn = (N + 15) / 16;
  for (int item = warp; item < MTn * NT; item += blockDim.x >> 5) {
    const int mt = item / NT, nt = item - mt * NT;
    const int col = nt * 4 + t;
    const int ecol = col_exp(exc[min(col, kTile - 1)]) - 64 + LongFold().shift();
    const int ecoli = own(col) ? col_exp(exc[kTile]) - 64 + LongFold().shift() : ecol;
    long long sums[4];
    uint32_t R[4] = {0, 0, 0, 0};
    tc_tile(LongFold(), T + (size_t)b * MTw * KT * kDig * 32, mt, KT, kChunkKT, dig, KS, (size_t)32 * KS, nt * 8, lane, sums, R);
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      const int row = mt * 16 + gq + 8 * rr;
      if (row >= N || col >= nx) continue;
      const int e = TE[(size_t)b * gsz.R() + row];
      const cpx val = {round_sum(LongFold(), sums[2 * rr], R[2 * rr], e + ecol),
                       round_sum(LongFold(), sums[2 * rr + 1], R[2 * rr + 1], e + ecoli)};
      comb(row, col, val);
    }
  }
  __syncthreads();
}

// the derived plane inputs of Recon^T: o[1] Xp_bar = i(ax u + az w), o[2]
// dx_bar = -i(ax du + az dw), o[3] Zp_bar = i(az u - ax w), o[4] dz_bar =
// i(az du - ax dw)
__device__ __forceinline__ void recon_T_inputs(double ax, double az, const cpx& u, const cpx& w, const cpx& du,
                                               const cpx& dw, cpx (&o)[5]) {
  o[1] = cpx{-fma(ax, u.im, az * w.im), fma(ax, u.re, az * w.re)};
  o[2] = cpx{fma(ax, du.im, az * dw.im), -fma(ax, du.re, az * dw.re)};
  o[3] = cpx{fma(ax, w.im, -az * u.im), fma(az, u.re, -ax * w.re)};
  o[4] = cpx{fma(ax, dw.im, -az * du.im), fma(az, du.re, -ax * dw.re)};
}

// Recon^T (as recon_T_tile) with its five contractions on the tensor cores
template <class S>
__device__ void recon_T_tc(const Grid& g, const S& gsz, const cpx* __restrict__ Ub, int z, int x0, int nx, int xfirst,
                           SolveTSmem& s) {
  const size_t cs = (size_t)gsz.Q() * gsz.X();
  const cpx* Uz = Ub + (size_t)z * 5 * cs;
  uint16_t* dig = reinterpret_cast<uint16_t*>(s.hc);
  int* exc = reinterpret_cast<int*>(dig + (size_t)kDig * 32 * ((size_t)(gsz.Q() + 15) / 16 * 16 + 8));
  const uint4* T = reinterpret_cast<const uint4*>(g.tcBT);
  auto at = [&](int c, int y, int col) { return Uz[(size_t)c * cs + (size_t)y * gsz.X() + x0 + col]; };
  auto axz = [&](int col, double& ax, double& az) {
    ax = g.kxK2[(size_t)z * gsz.X() + x0 + col];
    az = g.kzK2[(size_t)z * gsz.X() + x0 + col];
  };
  // alpha_bar = Q^T v_bar - Q'^T Xp_bar + Q''^T dx_bar -> s.Fa
  contract_planes_tc(
      g, gsz, T, g.tcBTE, 0, gsz.D(), nx, false,
      [&](int y, int col) { return col < xfirst ? cpx{0.0, 0.0} : at(1, y, col); },
      [&](int row, int col, cpx v) { s.Fa[row * kTile + col] = v; }, dig, exc);
  contract_planes_tc(
      g, gsz, T, g.tcBTE, 1, gsz.D(), nx, false,
      [&](int y, int col) {
        if (col < xfirst) return cpx{0.0, 0.0};
        double ax, az;
        axz(col, ax, az);
        const cpx u = at(0, y, col), w = at(2, y, col);
        return cpx{-fma(ax, u.im, az * w.im), fma(ax, u.re, az * w.re)};  // Xp_bar = i(ax u + az w)
      },
      [&](int row, int col, cpx v) {
        cpx& f = s.Fa[row * kTile + col];
        f.re -= v.re;
        f.im -= v.im;
      },
      dig, exc);
  contract_planes_tc(
      g, gsz, T, g.tcBTE, 2, gsz.D(), nx, false,
      [&](int y, int col) {
        if (col < xfirst) return cpx{0.0, 0.0};
        double ax, az;
        axz(col, ax, az);
        const cpx du = at(3, y, col), dw = at(4, y, col);
        return cpx{fma(ax, du.im, az * dw.im), -fma(ax, du.re, az * dw.re)};  // dx_bar = -i(ax du + az dw)
      },
      [&](int row, int col, cpx v) {
        cpx& f = s.Fa[row * kTile + col];
        f.re += v.re;
        f.im += v.im;
      },
      dig, exc);
  // beta_bar = R^T Zp_bar + R'^T dz_bar -> s.Fb
  contract_planes_tc(
      g, gsz, T, g.tcBTE, 3, gsz.R(), nx, xfirst == 1,
      [&](int y, int col) {
        if (col < xfirst) return recon_T_mean_input(at(0, y, col), at(2, y, col));
        double ax, az;
        axz(col, ax, az);
        const cpx u = at(0, y, col), w = at(2, y, col);
        return cpx{fma(ax, w.im, -az * u.im), fma(az, u.re, -ax * w.re)};  // Zp_bar = i(az u - ax w)
      },
      [&](int row, int col, cpx v) { s.Fb[row * kTile + col] = v; }, dig, exc);
  contract_planes_tc(
      g, gsz, T, g.tcBTE, 4, gsz.R(), nx, xfirst == 1,
      [&](int y, int col) {
        if (col < xfirst) return recon_T_mean_input(at(3, y, col), at(4, y, col));
        double ax, az;
        axz(col, ax, az);
        const cpx du = at(3, y, col), dw = at(4, y, col);
        return cpx{fma(ax, dw.im, -az * du.im), fma(az, du.re, -ax * dw.re)};  // dz_bar = i(az du - ax dw)
      },
      [&](int row, int col, cpx v) {
        cpx& f = s.Fb[row * kTile + col];
        f.re += v.re;
        f.im += v.im;
      },
      dig, exc);
}

// Hz, Hx, Hy of one plane and column from pa = Qpw^T Fa, qa = Qw^T Fa, rb =
// Rw^T Fb, its roundings fixed (the builds agree bit for bit):
// Hx = -i kx pa - i kz rb, Hz = -i kz pa + i kx rb, Hy = -K2 qa, times scl
__device__ __forceinline__ void quad_T_combine(double kx, double kz, double k2, double scl, const cpx& pa, const cpx& qa,
                                               const cpx& rb, cpx* out, size_t cs) {
  out[0] = cpx{scl * fma(kz, pa.im, __dmul_rn(-kx, rb.im)), scl * fma(kx, rb.re, __dmul_rn(-kz, pa.re))};
  out[cs] = cpx{scl * fma(kx, pa.im, __dmul_rn(kz, rb.im)), -scl * fma(kx, pa.re, __dmul_rn(kz, rb.re))};
  out[2 * cs] = cpx{__dmul_rn(-scl, k2) * qa.re, __dmul_rn(-scl, k2) * qa.im};
}

// the mean line's: Hx.re = Rw^T fa, Hz.re = Rw^T fb, rb = Rw^T (fa + i fb)
__device__ __forceinline__ void quad_T_mean(double scl, const cpx& rb, cpx* out, size_t cs) {
  out[0] = cpx{scl * rb.im, 0.0};
  out[cs] = cpx{scl * rb.re, 0.0};
  out[2 * cs] = cpx{0.0, 0.0};
}

// H_bar = Quad^T(F_bar) on the tensor cores for the columns [0, nx):
// per plane y the contractions over the modes pa = Qpw^T Fa, qa = Qw^T Fa,
// rb = Rw^T Fb as GEMMs (rows: planes), then the combination of the FP64
// loop in k_solve_T (the mean column, whose two lines are Re and Im of Fb's
// column 0: quad_T_mean)
template <class S>
__device__ void quad_T_tc(const Grid& g, const S& gsz, int z, int x0, int nx, int xfirst, SolveTSmem& s, cpx* __restrict__ Hb) {
  const int KTr = (gsz.R() + 15) / 16, MTq = (gsz.Q() + 15) / 16;
  const size_t KS = (size_t)KTr * 16 + 8;
  uint16_t* dA = reinterpret_cast<uint16_t*>(s.hc);             // [7][32][KS] digits of Fa
  uint16_t* dB = dA + (size_t)kDig * 32 * KS;                    // digits of Fb
  int* exa = reinterpret_cast<int*>(dB + (size_t)kDig * 32 * KS);  // [2][kTile] column exponents, mean's Im
  auto own = [&](bool fb, int col) { return fb && col < xfirst; };
  for (int i = threadIdx.x; i < 2 * kTile + 1; i += blockDim.x) exa[i] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < (gsz.D() + gsz.R()) * kTile; i += blockDim.x) {
    const bool fb = i >= gsz.D() * kTile;
    const int j = fb ? i - gsz.D() * kTile : i, row = j / kTile, col = j - row * kTile;
    if (col >= nx || (col < xfirst && !fb)) continue;
    const cpx v = (fb ? s.Fb : s.Fa)[row * kTile + col];
    int e = 0, eim = 0;
    column_exponents(v, own(fb, col), e, eim);
    if (e) atomicMax(&exa[(fb ? kTile : 0) + col], e);
    if (eim) atomicMax(&exa[2 * kTile], eim);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * KTr * 8 * kTile; i += blockDim.x) {
    const bool fb = i >= KTr * 8 * kTile;
    const int j = fb ? i - KTr * 8 * kTile : i, row = 2 * (j / kTile), col = j % kTile;
    const int N = fb ? gsz.R() : gsz.D();
    auto at = [&](int r) {
      return (r < N && col < nx && (col >= xfirst || fb)) ? (fb ? s.Fb : s.Fa)[r * kTile + col] : cpx{0.0, 0.0};
    };
    const cpx v0 = at(row), v1 = at(row + 1);
    const int ex = exa[(fb ? kTile : 0) + col] - 1022, exi = own(fb, col) ? exa[2 * kTile] - 1022 : ex;
    uint32_t* d = reinterpret_cast<uint32_t*>((fb ? dB : dA) + (size_t)(2 * col) * KS + row);
    digits_pair(scaled56(v0.re, ex), scaled56(v1.re, ex), d, 16 * KS);
    digits_pair(scaled56(v0.im, exi), scaled56(v1.im, exi), d + KS / 2, 16 * KS);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  const int NT = (2 * nx + 7) / 8;
  const uint4* __restrict__ W = reinterpret_cast<const uint4*>(g.tcWT);
  const size_t cs = (size_t)gsz.Q() * gsz.X();
  const double kz = g.Kz[z];
  for (int item = warp; item < MTq * NT; item += blockDim.x >> 5) {
    const int mt = item / NT, nt = item - mt * NT;
    const int col = nt * 4 + t;
    double v[3][4];  // pa, qa, rb at (rows gq, gq + 8) x (Re, Im)
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const uint16_t* d = b < 2 ? dA : dB;
      const int ecol = col_exp(exa[(b < 2 ? 0 : kTile) + min(col, kTile - 1)]) - 64 + LongFold().shift();
      const int ecoli = own(b == 2, col) ? col_exp(exa[2 * kTile]) - 64 + LongFold().shift() : ecol;
      long long sums[4];
      uint32_t R[4] = {0, 0, 0, 0};
      tc_tile(LongFold(), W + (size_t)b * MTq * KTr * kDig * 32, mt, KTr, kChunkKT, d, KS, (size_t)32 * KS, nt * 8, lane, sums, R);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int y = min(mt * 16 + gq + 8 * (r >> 1), gsz.Q() - 1);
        v[b][r] = round_sum(LongFold(), sums[r], R[r], g.tcWTE[(size_t)b * gsz.Q() + y] + (r & 1 ? ecoli : ecol));
      }
    }
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      const int y = mt * 16 + gq + 8 * rr;
      if (y >= gsz.Q() || col >= nx) continue;
      const int x = x0 + col;
      if (col < xfirst) {
        quad_T_mean(g.norm, cpx{v[2][2 * rr], v[2][2 * rr + 1]}, Hb + (size_t)y * gsz.X(), cs);
        continue;
      }
      quad_T_combine(g.Kx[x], kz, g.K2[(size_t)z * gsz.X() + x], x == 0 ? g.norm : 0.5 * g.norm,
                     cpx{v[0][2 * rr], v[0][2 * rr + 1]}, cpx{v[1][2 * rr], v[1][2 * rr + 1]},
                     cpx{v[2][2 * rr], v[2][2 * rr + 1]}, Hb + ((size_t)z * 5 * gsz.Q() + y) * gsz.X() + x, cs);
    }
  }
}

// quad_T_tc for launches with few blocks: a 4-column tile, a warp per 16
// planes, its three tables' k-tiles as one stream.  KP: row pairs of Fa or Fb
// a thread holds (R <= 64 KP).
template <int KP, class S>
__device__ __forceinline__ void quad_T_few(const Grid& g, const S& gsz, int z, int x0, int nx, int xfirst, SolveTSmem& s,
                                           cpx* __restrict__ Hb) {
  constexpr int TT = 4, NTHR = 256, NC = 2 * TT;
  const int KTr = (gsz.R() + 15) / 16, MTq = (gsz.Q() + 15) / 16;
  const size_t KS = (size_t)KTr * 16 + 8;
  int* exc = reinterpret_cast<int*>(s.dig + (size_t)2 * kDig * NC * KS);  // [2][TT], mean's Im
  if (threadIdx.x < 2 * TT + 1) exc[threadIdx.x] = 0;
  __syncthreads();
  {
    // threads [0, 128) take Fa, the rest Fb; row pairs 2 (t / TT) + 64 k
    const int cls = threadIdx.x >> 7, col = threadIdx.x % TT, j0 = 2 * ((threadIdx.x & 127) / TT);
    const int N = cls ? gsz.R() : gsz.D();
    const cpx* F = cls ? s.Fb : s.Fa;
    const bool on = col < nx && (col >= xfirst || cls), own = cls && col < xfirst;
    cpx v[KP][2];
    int e = 0, eim = 0;
#pragma unroll
    for (int k = 0; k < KP; ++k)
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int j = j0 + p + 64 * k;
        v[k][p] = (on && j < N) ? F[j * TT + col] : cpx{0.0, 0.0};
        column_exponents(v[k][p], own, e, eim);
      }
#pragma unroll
    for (int o = 16; o >= TT; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    if ((threadIdx.x & 31) < TT) atomicMax(&exc[cls * TT + col], e);
    if (eim) atomicMax(&exc[2 * TT], eim);
    __syncthreads();
    const int ex = exc[cls * TT + col] - 1022, exi = own ? exc[2 * TT] - 1022 : ex;
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int j = j0 + 64 * k;
      if (j >= KTr * 16) break;
      uint32_t* d = reinterpret_cast<uint32_t*>(s.dig + ((size_t)cls * kDig * NC + 2 * col) * KS + j);
      digits_pair(scaled56(v[k][0].re, ex), scaled56(v[k][1].re, ex), d, NC * KS / 2);
      digits_pair(scaled56(v[k][0].im, exi), scaled56(v[k][1].im, exi), d + KS / 2, NC * KS / 2);
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  const uint4* __restrict__ W = reinterpret_cast<const uint4*>(g.tcWT) + lane;
  const size_t cs = (size_t)gsz.Q() * gsz.X();
  const int x = x0 + min(t, nx - 1);
  auto table = [&](int mt, int b) { return W + ((size_t)b * MTq + mt) * KTr * kFragStep; };
  FragPair pf;
  if (warp < MTq) tc_stream_start(pf, table(warp, 0));
  for (int mt = warp; mt < MTq; mt += NTHR / 32) {
    cpx v[3][2];  // pa, qa, rb at rows gq, gq + 8
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const int cls = b < 2 ? 0 : 1, nm = mt + NTHR / 32;
      long long T[4];
      uint32_t R[4] = {0, 0, 0, 0};
      tc_tile_stream(LongFold(), pf, table(mt, b), b < 2 ? table(mt, b + 1) : (nm < MTq ? table(nm, 0) : nullptr), KTr,
                     tc_row_addr(s.dig + (size_t)cls * kDig * NC * KS, KS, (size_t)NC * KS, 0, lane),
                     (uint32_t)(4 * NC * KS), T, R);
      const int ecol = col_exp(exc[cls * TT + t]) - 64 + LongFold().shift();
      const int ecoli = cls && t < xfirst ? col_exp(exc[2 * TT]) - 64 + LongFold().shift() : ecol;
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int e = g.tcWTE[(size_t)b * gsz.Q() + min(mt * 16 + gq + 8 * rr, gsz.Q() - 1)];
        v[b][rr] = cpx{round_sum(LongFold(), T[2 * rr], R[2 * rr], e + ecol),
                       round_sum(LongFold(), T[2 * rr + 1], R[2 * rr + 1], e + ecoli)};
      }
    }
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      const int y = mt * 16 + gq + 8 * rr;
      if (y >= gsz.Q() || t >= nx) continue;
      if (t < xfirst) quad_T_mean(g.norm, v[2][rr], Hb + (size_t)y * gsz.X(), cs);
      else quad_T_combine(g.Kx[x], g.Kz[z], g.K2[(size_t)z * gsz.X() + x], x == 0 ? g.norm : 0.5 * g.norm, v[0][rr], v[1][rr],
                     v[2][rr], Hb + ((size_t)z * 5 * gsz.Q() + y) * gsz.X() + x, cs);
    }
  }
}

// Recon^T (as recon_T_tc) for launches with few blocks
template <int KP, class S>
__device__ __forceinline__ void recon_T_few(const Grid& g, const S& gsz, const cpx* __restrict__ Ub, int z, int x0,
                                            int nx, int xfirst, SolveTSmem& s) {
  constexpr int TT = 4, NTHR = 256;
  const size_t cs = (size_t)gsz.Q() * gsz.X();
  const int col = threadIdx.x % TT, x = x0 + min(col, nx - 1);
  const cpx* Uc = Ub + (size_t)z * 5 * cs + x;
  const double ax = g.kxK2[(size_t)z * gsz.X() + x], az = g.kzK2[(size_t)z * gsz.X() + x];
  few_contract<TT, NTHR, KP>(
      gsz, g.tcBT, g.tcBTE, true, nx, xfirst == 1, s.dig,
      [&](int y, cpx (&o)[5]) {
        const cpx* b = Uc + (size_t)y * gsz.X();
        if (col < xfirst) {
          o[3] = recon_T_mean_input(b[0], b[2 * cs]);
          o[4] = recon_T_mean_input(b[3 * cs], b[4 * cs]);
          return;
        }
        recon_T_inputs(ax, az, b[0], b[2 * cs], b[3 * cs], b[4 * cs], o);
        o[0] = b[cs];
      },
      [](int q) { return q; },
      [](int q, const cpx& f, const cpx& v) {
        if (q == 1) return cpx{f.re - v.re, f.im - v.im};
        return cpx{f.re + v.re, f.im + v.im};
      },
      s.Fa, s.Fb);
}

// the chains of a few-block tile (as solve_chains_few): U^T then L^T
template <int TT, class S>
__device__ __forceinline__ void solveT_chains_few(const Grid& g, const S& gsz, int bidx, int nx, int xfirst,
                                                  const SolveTSmem& s) {
  static_assert(TT == 4, "the thread map");
  const int tid = threadIdx.x;
  auto run = [&](auto nl, const double* LU, const double* RD, int W, int N, int par, bool on, double* b) {
    constexpr int NL = decltype(nl)::value;
    const int M = max((N - par + 1) / 2, 1), steps = (N + 1) / 2, l = tid & (NL - 1);
    double* bp = b + (N > par ? par * 2 * TT : 0);
    on = on && N > par;
    chain_sweep<NL, false, true>(M, steps, l, on, bp, 4 * TT,
                                 [&](int m, int t) { return LU[(size_t)(par + 2 * m) * W + NL + t]; },
                                 [&](int m) { return RD[par + 2 * m]; });
    __syncwarp();
    chain_sweep<NL, true, false>(M, steps, l, on, bp, 4 * TT,
                                 [&](int m, int t) { return LU[(size_t)(par + 2 * m) * W + NL - t]; },
                                 [](int) { return 1.0; });
  };
  if (tid < 64) {
    const int ch = tid / 4, l = ch / 4, lc = min(l, nx - 1);
    run(std::integral_constant<int, 4>(), s.luA + (size_t)lc * gsz.D() * 9, s.rdA + (size_t)lc * gsz.D(), 9, gsz.D(),
        ch & 1, l < nx && l >= xfirst, reinterpret_cast<double*>(s.ra + lc) + ((ch >> 1) & 1));
  } else if (tid < 96) {
    const int ch = (tid - 64) / 2, l = ch / 4, lc = min(l, nx - 1);
    run(std::integral_constant<int, 2>(), s.luB + (size_t)lc * gsz.R() * 5, s.rdB + (size_t)lc * gsz.R(), 5, gsz.R(),
        ch & 1, l < nx && l >= xfirst, reinterpret_cast<double*>(s.rb + lc) + ((ch >> 1) & 1));
  } else if (tid < 128 && xfirst) {
    const int ch = ((tid - 96) / 2) & 7;
    run(std::integral_constant<int, 2>(), g.lu0 + (size_t)bidx * gsz.R() * 5, g.rd0 + (size_t)bidx * gsz.R(), 5, gsz.R(),
        ch & 1, tid < 112, reinterpret_cast<double*>(ch < 4 ? s.ra : s.rb) + ((ch >> 1) & 1));
  }
}

// Block z ntx + tx: kx tile tx of line z; the mean line is column 0 of the
// kz = 0 line's first tile, its parts as Re and Im of the beta class (as in
// k_solve).  S: the sizes (SizesRT, or SizesCT for a specialised grid); TT kx
// columns per block; FEW (the row and plane pairs a thread holds): the build
// for launches with few blocks (TT 4)
template <bool MULTI, class S, int TT = kTile, int FEW = 0>
__global__ void __launch_bounds__(kThreads, FEW ? 1 : 2) k_solve_T(const __grid_constant__ Grid g0, SolveTArgs a) {
  const int ntx = (g0.X + TT - 1) / TT;
  const int z = blockIdx.x / ntx, tx = blockIdx.x - z * ntx;
  const int inst = blockIdx.y;
  CHN_INSTANCE_GRID(g0, a.grids, inst);
  const S gsz(g);
  if (z >= gsz.Nz() || tx * TT >= gsz.X()) return;
  if (blocked_t(a.status, a.sdiv, inst)) return;
  const int x0 = tx * TT;
  const int nx = min(TT, gsz.X() - x0);
  cpx* __restrict__ Cc = a.Cc.at(inst);
  auto cidx = [&](int v, int r, int x) { return (((size_t)z * 2 + v) * gsz.R() + r) * gsz.X() + x; };
  extern __shared__ __align__(16) unsigned char smem[];
  // deterministic block sum of the Re parts into this block's slot
  __shared__ double gred[kThreads / 32];
  auto add_re_part = [&](double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) gred[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += gred[w];
      a.gacc[(long long)inst * a.gstride + 1 + blockIdx.x] += t;
    }
  };
  if (z == gsz.Nz() / 2) {
    // the tangent zeroes this line every substage (channel/channel.c:460-467)
    if (!a.final_only)
      for (int i = threadIdx.x; i < 2 * gsz.R() * nx; i += blockDim.x) {
        const int v = i / (gsz.R() * nx), r = (i / nx) % gsz.R(), x = x0 + i % nx;
        Cc[cidx(v, r, x)] = cpx{0.0, 0.0};
      }
    return;
  }
  const cpx* __restrict__ Ub = a.Ub.at(inst);
  const int xfirst = (z == 0 && x0 == 0) ? 1 : 0;
  SolveTSmem s;
  if constexpr (FEW) {
    s = carve_solveT_few<TT>(g, smem);
    if (!a.final_only)
      stage_factors<kThreads>(g, gsz, ((size_t)a.k * gsz.Nz() + z) * gsz.X() + x0, nx, s.luA, s.luB, s.rdA, s.rdB);
    recon_T_few<FEW>(g, gsz, Ub, z, x0, nx, xfirst, s);
  } else {
    s = carve_solveT(g, smem);
    if (g.tc) recon_T_tc(g, gsz, Ub, z, x0, nx, xfirst, s);
    else recon_T_tile(g, Ub, z, x0, nx, xfirst, s);
  }
  if (a.final_only) {
    // the sweep's start state: IU = Recon(IC), so IC_bar += Recon^T(IU_bar)
    for (int i = threadIdx.x; i < gsz.R() * TT; i += blockDim.x) {
      const int r = i / TT, l = i - r * TT;
      if (l >= nx) continue;
      const int x = x0 + l;
      if (l < xfirst) {  // real lines: R^T u_bar + R'^T du_bar to alpha, of w_bar to beta
        const cpx f = s.Fb[r * TT];
        Cc[cidx(0, r, 0)].re += f.re;
        Cc[cidx(1, r, 0)].re += f.im;
        continue;
      }
      if (r < gsz.D()) {
        const cpx f = s.Fa[r * TT + l];
        Cc[cidx(0, r, x)].re += f.re;
        Cc[cidx(0, r, x)].im += f.im;
      }
      const cpx f = s.Fb[r * TT + l];
      Cc[cidx(1, r, x)].re += f.re;
      Cc[cidx(1, r, x)].im += f.im;
    }
    return;
  }
  const int k = a.k;
  const double dt = g.dt;
  // forward coefficients c = {1/2, 1/3, 1}, d = {0, -1/6, -2/3}; b[k] is LU index k
  const double ck = k == 0 ? 1. / 2 : (k == 1 ? 1. / 3. : 1.);
  const double dnext = k == 0 ? -1. / 6 : (k == 1 ? -2. / 3 : 0.0);
  const int bidx = k;
  const int aidx_next = (k == 0) ? 1 : 0;  // a[1] = -1/2, a[2] = 1/3
  // x_bar = Recon^T part + E_{k+1}^T c_out_bar (or c_out_bar); F_bar = dt d_{k+1} c_out_bar
  for (int i = threadIdx.x; i < gsz.R() * TT; i += blockDim.x) {
    const int r = i / TT, l = i - r * TT;
    if (l >= nx) continue;
    const int x = x0 + l;
    const size_t zx = (size_t)z * gsz.X() + x;
    cpx xa, xb;
    if (l < xfirst) {
      const cpx rec = s.Fb[r * TT], coa = Cc[cidx(0, r, 0)], cob = Cc[cidx(1, r, 0)];
      xa = coa;
      xb = cob;
      if (k < 2) {
        const double* E = g.ex0 + (size_t)aidx_next * gsz.R() * 5;
        xa = band_matvecT_row(E, 5, 2, 2, gsz.R(), Cc + cidx(0, 0, 0), gsz.X(), r);
        xb = band_matvecT_row(E, 5, 2, 2, gsz.R(), Cc + cidx(1, 0, 0), gsz.X(), r);
        s.Fb[r * TT] = cpx{dt * dnext * coa.re, dt * dnext * cob.re};  // the mean right-hand side is real
      } else {
        s.Fb[r * TT] = cpx{0.0, 0.0};
      }
      xa.re += rec.re;
      xb.re += rec.im;
      s.ra[r * TT] = xa;
      s.rb[r * TT] = xb;
      continue;
    }
    if (r < gsz.D()) {
      const cpx rec = s.Fa[r * TT + l];
      const cpx co = Cc[cidx(0, r, x)];
      if (k < 2) {
        const double* E = g.exA + ((size_t)aidx_next * gsz.Nz() * gsz.X() + zx) * gsz.D() * 9;
        xa = band_matvecT_row(E, 9, 4, 4, gsz.D(), Cc + cidx(0, 0, x), gsz.X(), r);
        s.Fa[r * TT + l] = cpx{dt * dnext * co.re, dt * dnext * co.im};
      } else {
        xa = co;
        s.Fa[r * TT + l] = cpx{0.0, 0.0};
      }
      xa.re += rec.re;
      xa.im += rec.im;
    } else {
      xa = Cc[cidx(0, r, x)];  // alpha rows >= Ny-4 ride along unchanged
    }
    {
      const cpx rec = s.Fb[r * TT + l];
      const cpx co = Cc[cidx(1, r, x)];
      if (k < 2) {
        const double* E = g.exB + ((size_t)aidx_next * gsz.Nz() * gsz.X() + zx) * gsz.R() * 5;
        xb = band_matvecT_row(E, 5, 2, 2, gsz.R(), Cc + cidx(1, 0, x), gsz.X(), r);
        s.Fb[r * TT + l] = cpx{dt * dnext * co.re, dt * dnext * co.im};
      } else {
        xb = co;
        s.Fb[r * TT + l] = cpx{0.0, 0.0};
      }
      xb.re += rec.re;
      xb.im += rec.im;
    }
    s.ra[r * TT + l] = xa;
    s.rb[r * TT + l] = xb;
  }
  __syncthreads();
  const bool want_g = a.gacc != nullptr;
  if (xfirst) {
    // the mean line's flux correction x = xs - 0.5 add (rwsum . xs.re),
    // transposed: xs_bar.re = x_bar.re - 0.5 rwsum (add . x_bar.re); warp 0
    if (threadIdx.x < 32) {
      double part = 0.0;
      for (int i = threadIdx.x; i < gsz.R(); i += 32) part = fma(g.add0[i], s.ra[i * TT].re, part);
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      // the forced tangent adds 0.5 * 2.0 * add to this line's real part
      // (channel/increproject0.c:209-214): its cotangent is <add, x_bar.re>
      if (want_g && threadIdx.x == 0) a.gacc[(long long)inst * a.gstride] += part;
      for (int i = threadIdx.x; i < gsz.R(); i += 32) s.ra[i * TT].re = fma(-0.5 * part, g.rwsum[i], s.ra[i * TT].re);
    }
    __syncthreads();
  }
  if constexpr (FEW) {
    solveT_chains_few<TT>(g, gsz, bidx, nx, xfirst, s);
  } else {
    // L^{-T}: per column 4 chains for alpha, 4 for beta (parity x re/im), the
    // alpha chains in threads [0, 4 TT), the beta ones from a warp boundary, the
    // mean line's from the next
    constexpr int kHalf = 4 * TT;
    const int sec = (int)threadIdx.x / kHalf, t = (int)threadIdx.x - sec * kHalf, l = t / 4;
    const int par = t & 1, part = (t >> 1) & 1;
    if (sec < 2 && l < nx && l >= xfirst) {
      const size_t sys = ((size_t)bidx * gsz.Nz() + z) * gsz.X() + x0 + l;
      if (sec == 0)
        band_solveT_chain<9, 4, 4>(g.luA + sys * gsz.D() * 9, g.rdA + sys * gsz.D(), gsz.D(), par,
                                   reinterpret_cast<double*>(s.ra + l) + part, 2 * TT);
      else
        band_solveT_chain<5, 2, 2>(g.luB + sys * gsz.R() * 5, g.rdB + sys * gsz.R(), gsz.R(), par,
                                   reinterpret_cast<double*>(s.rb + l) + part, 2 * TT);
    } else if (sec == 2 && xfirst && t < 8) {
      band_solveT_chain<5, 2, 2>(g.lu0 + (size_t)bidx * gsz.R() * 5, g.rd0 + (size_t)bidx * gsz.R(), gsz.R(), par,
                                 reinterpret_cast<double*>(t < 4 ? s.ra : s.rb) + part, 2 * TT);
    }
  }
  __syncthreads();
  // dJ/dRe: <c2_bar, f_Re> of this block's columns (the forcing of
  // recon_solve.cu's kind 3 rebuilt from the stored primal states)
  double gpart = 0.0;
  const double re2 = g.re * g.re;
  const double akf = k == 1 ? -1. / 2 : 1. / 3.;                  // forward a_k
  const double bkf = k == 0 ? 1. / 6 : (k == 1 ? 2. / 3 : 0.0);  // forward b_k
  if (want_g) {
    const int xs = a.xslot.slot();
    const cpx* xk = a.Xf + (long long)inst * a.xstride + (long long)xs * a.xslot.stride;
    const double ft1 = a.Ftr ? a.Ftr[(long long)inst * a.ftr_stride + xs + 1] : 0.0;
    const size_t csz = coef_size(g);
    for (int i = threadIdx.x; i < gsz.R() * TT; i += blockDim.x) {
      const int r = i / TT, l = i - r * TT;
      if (l >= nx) continue;
      const int x = x0 + l;
      if (l < xfirst) {
        // D0 = -Rps on the primal's solved mean flow before its flux
        // correction, MC[3n + k + 1] - 0.5 flux_t add
        const cpx p0 = band_matvec_row(g.Rps, 5, 2, 2, gsz.R(), xk + cidx(0, 0, 0), gsz.X(), r);
        cpx p1 = band_matvec_row(g.Rps, 5, 2, 2, gsz.R(), xk + csz + cidx(0, 0, 0), gsz.X(), r);
        p1.re -= 0.5 * ft1 * rps_row_real(g, g.add0, r);
        const cpx q0 = band_matvec_row(g.Rps, 5, 2, 2, gsz.R(), xk + cidx(1, 0, 0), gsz.X(), r);
        const cpx q1 = band_matvec_row(g.Rps, 5, 2, 2, gsz.R(), xk + csz + cidx(1, 0, 0), gsz.X(), r);
        const cpx c2a = s.ra[r * TT], c2b = s.rb[r * TT];
        gpart += re2 * dt * (c2a.re * (akf * p0.re + bkf * p1.re) + c2a.im * (akf * p0.im + bkf * p1.im));
        gpart += re2 * dt * (c2b.re * (akf * q0.re + bkf * q1.re) + c2b.im * (akf * q0.im + bkf * q1.im));
        continue;
      }
      const double k2 = g.K2[(size_t)z * gsz.X() + x];
      if (r < gsz.D()) {
        const cpx d0 = visc_v_row(g, k2, xk + cidx(0, 0, x), gsz.X(), r);
        const cpx d1 = visc_v_row(g, k2, xk + csz + cidx(0, 0, x), gsz.X(), r);
        const cpx c2 = s.ra[r * TT + l];
        gpart -= re2 * dt * (c2.re * (akf * d0.re + bkf * d1.re) + c2.im * (akf * d0.im + bkf * d1.im));
      }
      const cpx d0 = visc_g_row(g, k2, xk + cidx(1, 0, x), gsz.X(), r);
      const cpx d1 = visc_g_row(g, k2, xk + csz + cidx(1, 0, x), gsz.X(), r);
      const cpx c2 = s.rb[r * TT + l];
      gpart += re2 * dt * (c2.re * (akf * d0.re + bkf * d1.re) + c2.im * (akf * d0.im + bkf * d1.im));
    }
  }
  // F_bar += dt c_k c2_bar; c_in_bar = E_0^T c2_bar (k == 0) or c2_bar
  for (int i = threadIdx.x; i < gsz.R() * TT; i += blockDim.x) {
    const int r = i / TT, l = i - r * TT;
    if (l >= nx) continue;
    const int x = x0 + l;
    const size_t zx = (size_t)z * gsz.X() + x;
    if (l < xfirst) {
      const cpx c2a = s.ra[r * TT], c2b = s.rb[r * TT];
      cpx& f = s.Fb[r * TT];
      f = cpx{fma(dt * ck, c2a.re, f.re), fma(dt * ck, c2b.re, f.im)};
      Cc[cidx(0, r, 0)] = k == 0 ? band_matvecT_row(g.ex0, 5, 2, 2, gsz.R(), s.ra, TT, r) : c2a;
      Cc[cidx(1, r, 0)] = k == 0 ? band_matvecT_row(g.ex0, 5, 2, 2, gsz.R(), s.rb, TT, r) : c2b;
      continue;
    }
    if (r < gsz.D()) {
      const cpx c2 = s.ra[r * TT + l];
      s.Fa[r * TT + l].re += dt * ck * c2.re;
      s.Fa[r * TT + l].im += dt * ck * c2.im;
      Cc[cidx(0, r, x)] = k == 0 ? band_matvecT_row(g.exA + zx * gsz.D() * 9, 9, 4, 4, gsz.D(), s.ra + l, TT, r) : c2;
    } else {
      Cc[cidx(0, r, x)] = s.ra[r * TT + l];
    }
    const cpx c2 = s.rb[r * TT + l];
    s.Fb[r * TT + l].re += dt * ck * c2.re;
    s.Fb[r * TT + l].im += dt * ck * c2.im;
    Cc[cidx(1, r, x)] = k == 0 ? band_matvecT_row(g.exB + zx * gsz.R() * 5, 5, 2, 2, gsz.R(), s.rb + l, TT, r) : c2;
  }
  __syncthreads();
  if (want_g) add_re_part(gpart);
  // H_bar = Quad^T(F_bar) (transpose of channel/project.c:97-115, 177-191):
  //   Hx_bar = -i kx Qpw^T Fa_bar - i kz Rw^T Fb_bar
  //   Hz_bar = -i kz Qpw^T Fa_bar + i kx Rw^T Fb_bar,  Hy_bar = -K2 Qw^T Fa_bar
  // Scaled for the inverse transform that follows: the forward transform's 1/(px pz),
  // halved off the kx = 0 column (the transpose of the real-to-complex x
  // transform).  Plane pairs (y, -y) share the sums: weights of even type
  // (Qw, Rw) give E + O / E - O, of odd type (Qpw) E + O / O - E.
  if constexpr (FEW) {
    quad_T_few<FEW>(g, gsz, z, x0, nx, xfirst, s, a.Hb.at(inst));
    return;
  }
  if (g.tc) {
    quad_T_tc(g, gsz, z, x0, nx, xfirst, s, a.Hb.at(inst));
    return;
  }
  const int lx = threadIdx.x % TT, grp = threadIdx.x / TT, ngrp = blockDim.x / TT;
  if (lx >= nx) return;
  const int x = x0 + lx;
  const double kx = g.Kx[x], kz = g.Kz[z], k2 = g.K2[(size_t)z * gsz.X() + x];
  const double scl = x == 0 ? g.norm : 0.5 * g.norm;
  cpx* __restrict__ Hb = a.Hb.at(inst);
  const size_t cs = (size_t)gsz.Q() * gsz.X();
  for (int yp = grp; yp < gsz.Qh(); yp += ngrp) {
    const int y1 = yp, y2 = gsz.Q() - 1 - yp;
    // E/O sums over even/odd rows: [0] Qpw^T Fa, [1] Qw^T Fa, [2] Rw^T Fb
    double er[3] = {0, 0, 0}, ei[3] = {0, 0, 0}, orr[3] = {0, 0, 0}, oi[3] = {0, 0, 0};
    {
      int i = 0;
      for (; i + 1 < gsz.D(); i += 2) {
        const cpx f0 = s.Fa[i * TT + lx], f1 = s.Fa[(i + 1) * TT + lx];
        cfma_t(__ldg(g.Wqp + (size_t)i * gsz.Q() + yp), f0, er[0], ei[0]);
        cfma_t(__ldg(g.Wqp + (size_t)(i + 1) * gsz.Q() + yp), f1, orr[0], oi[0]);
        cfma_t(__ldg(g.Wq + (size_t)i * gsz.Q() + yp), f0, er[1], ei[1]);
        cfma_t(__ldg(g.Wq + (size_t)(i + 1) * gsz.Q() + yp), f1, orr[1], oi[1]);
      }
      if (i < gsz.D()) {
        const cpx f0 = s.Fa[i * TT + lx];
        cfma_t(__ldg(g.Wqp + (size_t)i * gsz.Q() + yp), f0, er[0], ei[0]);
        cfma_t(__ldg(g.Wq + (size_t)i * gsz.Q() + yp), f0, er[1], ei[1]);
      }
      i = 0;
      for (; i + 1 < gsz.R(); i += 2) {
        const cpx f0 = s.Fb[i * TT + lx], f1 = s.Fb[(i + 1) * TT + lx];
        cfma_t(__ldg(g.Wr + (size_t)i * gsz.Q() + yp), f0, er[2], ei[2]);
        cfma_t(__ldg(g.Wr + (size_t)(i + 1) * gsz.Q() + yp), f1, orr[2], oi[2]);
      }
      if (i < gsz.R()) cfma_t(__ldg(g.Wr + (size_t)i * gsz.Q() + yp), s.Fb[i * TT + lx], er[2], ei[2]);
    }
    for (int side = 0; side < 2; ++side) {
      if (side == 1 && y2 == y1) break;
      const int y = side ? y2 : y1;
      auto val = [&](int c, bool odd_basis) {
        cpx r;
        if (!side) { r.re = er[c] + orr[c]; r.im = ei[c] + oi[c]; }
        else if (!odd_basis) { r.re = er[c] - orr[c]; r.im = ei[c] - oi[c]; }
        else { r.re = orr[c] - er[c]; r.im = oi[c] - ei[c]; }
        return r;
      };
      if (lx < xfirst) quad_T_mean(scl, val(2, false), Hb + (size_t)y * gsz.X(), cs);
      else
        quad_T_combine(kx, kz, k2, scl, val(0, true), val(1, false), val(2, false),
                     Hb + ((size_t)z * 5 * gsz.Q() + y) * gsz.X() + x, cs);
    }
  }
}

// Ca[i] += src[i] over each instance's coefficient array (the per-step
// source of a time-summed objective)
template <bool MULTI>
__global__ void __launch_bounds__(kThreads) k_add_source(const __grid_constant__ Grid g0, Batch<const cpx> src,
                                                         Batch<cpx> ca, const Grid* grids) {
  const int inst = blockIdx.y;
  CHN_INSTANCE_GRID(g0, grids, inst);
  const size_t n = coef_size(g);
  const cpx* __restrict__ s = src.at(inst);
  cpx* __restrict__ c = ca.at(inst);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    c[i].re += s[i].re;
    c[i].im += s[i].im;
  }
}

cudaError_t launch_add_source(const Grid& g, Batch<const cpx> src, Batch<cpx> ca, int ninst, cudaStream_t st,
                              const Grid* grids) {
  if (ninst <= 0) return cudaSuccess;
  const size_t n = coef_size(g);
  int blocks = (int)((n + kThreads - 1) / kThreads);
  if (blocks > 152 * 4) blocks = 152 * 4;
  if (grids) k_add_source<true><<<dim3(blocks, ninst), kThreads, 0, st>>>(g, src, ca, grids);
  else k_add_source<false><<<dim3(blocks, ninst), kThreads, 0, st>>>(g, src, ca, grids);
  return cudaGetLastError();
}

static int s_solveT_optin = 0;

// launches of at most kFewTiles 4-column tiles take the FEW build (where
// CHN_SOLVE_TILE does not ask for a tile)
static bool solveT_few(const Grid& g, const SolveTArgs& a) {
  if (a.grids || !g.tc || g.sfixed || g.R <= 16 || g.R > 128 || g.Q > 256) return false;
  if ((long long)g.Nz * ((g.X + 3) / 4) * a.ninst > kFewTiles) return false;
  return solveT_few_smem_bytes(g, 4) + 1024 <= (size_t)s_solveT_optin;
}

cudaError_t launch_solve_T(const Grid& g, const SolveTArgs& a, cudaStream_t st) {
  if (a.ninst <= 0) return cudaSuccess;
  if (solveT_few(g, a)) {
    const dim3 grid(g.Nz * ((g.X + 3) / 4), a.ninst);
    const size_t sm = solveT_few_smem_bytes(g, 4);
    const bool fx = (g.fixed & FIXED_SOLVE) != 0;  // the solve's fixed-size choice covers its transpose
    if (fx && sizes_match<Sizes32>(g)) k_solve_T<false, Sizes32, 4, 1><<<grid, kThreads, sm, st>>>(g, a);
    else if (fx && sizes_match<Sizes16>(g)) k_solve_T<false, Sizes16, 4, 1><<<grid, kThreads, sm, st>>>(g, a);
    else if (g.Q <= 128 && g.R <= 64) k_solve_T<false, SizesRT, 4, 1><<<grid, kThreads, sm, st>>>(g, a);
    else k_solve_T<false, SizesRT, 4, 2><<<grid, kThreads, sm, st>>>(g, a);
    return cudaGetLastError();
  }
  const dim3 grid(g.Nz * ((g.X + kTile - 1) / kTile), a.ninst);
  const size_t sm = solveT_smem_bytes(g);
  const bool fx = (g.fixed & FIXED_SOLVE) && !a.grids;
  if (a.grids) k_solve_T<true, SizesRT><<<grid, kThreads, sm, st>>>(g, a);
  else if (fx && sizes_match<Sizes32>(g)) k_solve_T<false, Sizes32><<<grid, kThreads, sm, st>>>(g, a);
  else if (fx && sizes_match<Sizes16>(g)) k_solve_T<false, Sizes16><<<grid, kThreads, sm, st>>>(g, a);
  else k_solve_T<false, SizesRT><<<grid, kThreads, sm, st>>>(g, a);
  return cudaGetLastError();
}

void prepare_solve_T(int optin) {
  s_solveT_optin = optin;
  allow_max_smem(k_solve_T<false, SizesRT>, optin);
  allow_max_smem(k_solve_T<true, SizesRT>, optin);
  allow_max_smem(k_solve_T<false, Sizes32>, optin);
  allow_max_smem(k_solve_T<false, Sizes16>, optin);
  allow_max_smem(k_solve_T<false, SizesRT, 4, 1>, optin);
  allow_max_smem(k_solve_T<false, SizesRT, 4, 2>, optin);
  allow_max_smem(k_solve_T<false, Sizes32, 4, 1>, optin);
  allow_max_smem(k_solve_T<false, Sizes16, 4, 1>, optin);
}

}  // namespace chn
