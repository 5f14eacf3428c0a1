// Banded row operations shared by the implicit solve (recon_solve.cu) and
// its transpose (adjoint_exact.cu): the every-other-diagonal matrices of
// channel/mvOps.c and the viscous operators of the Re forcing.
#pragma once

#include "chn_common.cuh"

namespace chn {

// out[i] = sum_j A[i][j] y[i + 2(j - DL)] over the valid band (channel/mvOps.c:198-220),
// band layout (width W, lower DL, upper DU) known at compile time: the band
// loop unrolls with per-term predicates (the loads issue together), the
// multiply-adds keep the ascending order
template <int W, int DL, int DU>
__device__ __forceinline__ cpx band_matvec_row_t(const double* __restrict__ A, int N, const cpx* y, int ystride,
                                                 int i) {
  int j0 = DL - i / 2;
  if (j0 < 0) j0 = 0;
  int j1 = (N - i + 1) / 2 + DL;
  if (j1 > DL + DU + 1) j1 = DL + DU + 1;
  double re = 0.0, im = 0.0;
#pragma unroll
  for (int j = 0; j < DL + DU + 1; ++j) {
    if (j < j0 || j >= j1) continue;
    const double a = __ldg(A + (size_t)i * W + j);
    const cpx v = y[(i - 2 * (DL - j)) * ystride];
    re = fma(a, v.re, re);
    im = fma(a, v.im, im);
  }
  return cpx{re, im};
}

// the same for the two band layouts in use, chosen by the arguments
__device__ __forceinline__ cpx band_matvec_row(const double* __restrict__ A, int w, int dl, int du, int N,
                                               const cpx* y, int ystride, int i) {
  if (w == 9 && dl == 4 && du == 4) return band_matvec_row_t<9, 4, 4>(A, N, y, ystride, i);
  if (w == 5 && dl == 2 && du == 2) return band_matvec_row_t<5, 2, 2>(A, N, y, ystride, i);
  int j0 = dl - i / 2;
  if (j0 < 0) j0 = 0;
  int j1 = (N - i + 1) / 2 + dl;
  if (j1 > dl + du + 1) j1 = dl + du + 1;
  double re = 0.0, im = 0.0;
  for (int j = j0; j < j1; ++j) {
    const double a = __ldg(A + (size_t)i * w + j);
    const cpx v = y[(i - 2 * (dl - j)) * ystride];
    re = fma(a, v.re, re);
    im = fma(a, v.im, im);
  }
  return cpx{re, im};
}

// One elimination chain (fixed parity, real or imaginary part) of the
// no-pivot every-other-diagonal LU solve (channel/mvOps.c:29-91); W, DL, DU
// the band layout (width, lower, upper), RD the reciprocal pivots; entries
// outside the matrix are zero.  The last DL or DU results stay in registers
// and the multiply-adds run from the oldest to the newest, so a row waits for
// one multiply-add (and the pivot's product) of the row before it.  The
// factors of the next kChainRows rows load while a group's rows run (GLOBAL:
// from global memory; else they are staged in shared memory): 32x65x32, one
// instance, 36k -> 9k cycles of a block's 260k.
static constexpr int kChainRows = 4;

template <bool GLOBAL>
__device__ __forceinline__ double band_load(const double* p) {
  return GLOBAL ? __ldg(p) : *p;
}

template <int W, int DL, int DU, bool GLOBAL>
__device__ __forceinline__ void band_solve_chain(const double* __restrict__ LU, const double* __restrict__ RD, int N,
                                                 int par, double* b, int bstride) {
  const int M = (N - par + 1) / 2;  // rows of this parity: i = par + 2 m
  if (M <= 0) return;
  constexpr int G = kChainRows;
  {
    double f[G][DL], v[G], x[DL];
    auto load = [&](int m0) {
#pragma unroll
      for (int q = 0; q < G; ++q) {
        const int i = par + 2 * min(m0 + q, M - 1);
#pragma unroll
        for (int j = 0; j < DL; ++j) f[q][j] = band_load<GLOBAL>(LU + (size_t)i * W + j);
        v[q] = b[i * bstride];
      }
    };
#pragma unroll
    for (int t = 0; t < DL; ++t) x[t] = 0.0;  // x[t]: the result t + 1 rows back
    load(0);
    for (int m0 = 0; m0 < M; m0 += G) {
      double c[G][DL], w[G];
#pragma unroll
      for (int q = 0; q < G; ++q) {
#pragma unroll
        for (int j = 0; j < DL; ++j) c[q][j] = f[q][j];
        w[q] = v[q];
      }
      load(m0 + G);
#pragma unroll
      for (int q = 0; q < G; ++q) {
        double acc = w[q];
#pragma unroll
        for (int j = 0; j < DL; ++j) acc = fma(-c[q][j], x[DL - 1 - j], acc);
#pragma unroll
        for (int t = DL - 1; t > 0; --t) x[t] = x[t - 1];
        x[0] = acc;
        if (m0 + q < M) b[(par + 2 * (m0 + q)) * bstride] = acc;
      }
    }
  }
  {
    double f[G][DU], v[G], p[G], x[DU];
    auto load = [&](int n0) {  // rows from the last one down
#pragma unroll
      for (int q = 0; q < G; ++q) {
        const int i = par + 2 * max(M - 1 - (n0 + q), 0);
#pragma unroll
        for (int j = 0; j < DU; ++j) f[q][j] = band_load<GLOBAL>(LU + (size_t)i * W + DL + 1 + j);
        p[q] = band_load<GLOBAL>(RD + i);
        v[q] = b[i * bstride];
      }
    };
#pragma unroll
    for (int t = 0; t < DU; ++t) x[t] = 0.0;
    load(0);
    for (int n0 = 0; n0 < M; n0 += G) {
      double c[G][DU], w[G], r[G];
#pragma unroll
      for (int q = 0; q < G; ++q) {
#pragma unroll
        for (int j = 0; j < DU; ++j) c[q][j] = f[q][j];
        w[q] = v[q];
        r[q] = p[q];
      }
      load(n0 + G);
#pragma unroll
      for (int q = 0; q < G; ++q) {
        double acc = w[q];
#pragma unroll
        for (int j = DU - 1; j >= 0; --j) acc = fma(-c[q][j], x[j], acc);
        acc *= r[q];
#pragma unroll
        for (int t = DU - 1; t > 0; --t) x[t] = x[t - 1];
        x[0] = acc;
        if (n0 + q < M) b[(par + 2 * (M - 1 - (n0 + q))) * bstride] = acc;
      }
    }
  }
}

// row r of (K2^2 Qs + 2 K2 Qps + Qpps) y and of (Rps + K2 Rs) y, the viscous
// operators of the alpha and beta systems (channel/tangent_forcing.c:38-68)
__device__ __forceinline__ cpx visc_v_row(const Grid& g, double k2, const cpx* y, int ystride, int r) {
  const int dl = 4, du = 4, N = g.D;
  int j0 = dl - r / 2;
  if (j0 < 0) j0 = 0;
  int j1 = (N - r + 1) / 2 + dl;
  if (j1 > dl + du + 1) j1 = dl + du + 1;
  const double sq = k2 * k2;
  double re = 0.0, im = 0.0;
  for (int j = j0; j < j1; ++j) {
    const size_t o = (size_t)r * 9 + j;
    const double m = sq * __ldg(g.Qs + o) + 2. * k2 * __ldg(g.Qps + o) + __ldg(g.Qpps + o);
    const cpx v = y[(r - 2 * (dl - j)) * ystride];
    re = fma(m, v.re, re);
    im = fma(m, v.im, im);
  }
  return cpx{re, im};
}

__device__ __forceinline__ cpx visc_g_row(const Grid& g, double k2, const cpx* y, int ystride, int r) {
  const int dl = 2, du = 2, N = g.R;
  int j0 = dl - r / 2;
  if (j0 < 0) j0 = 0;
  int j1 = (N - r + 1) / 2 + dl;
  if (j1 > dl + du + 1) j1 = dl + du + 1;
  double re = 0.0, im = 0.0;
  for (int j = j0; j < j1; ++j) {
    const size_t o = (size_t)r * 5 + j;
    const double m = __ldg(g.Rps + o) + k2 * __ldg(g.Rs + o);
    const cpx v = y[(r - 2 * (dl - j)) * ystride];
    re = fma(m, v.re, re);
    im = fma(m, v.im, im);
  }
  return cpx{re, im};
}

// row r of Rps y for a real vector y (stride 1)
__device__ __forceinline__ double rps_row_real(const Grid& g, const double* y, int r) {
  const int dl = 2, du = 2, N = g.R;
  int j0 = dl - r / 2;
  if (j0 < 0) j0 = 0;
  int j1 = (N - r + 1) / 2 + dl;
  if (j1 > dl + du + 1) j1 = dl + du + 1;
  double acc = 0.0;
  for (int j = j0; j < j1; ++j) acc = fma(__ldg(g.Rps + (size_t)r * 5 + j), y[r - 2 * (dl - j)], acc);
  return acc;
}

}  // namespace chn
