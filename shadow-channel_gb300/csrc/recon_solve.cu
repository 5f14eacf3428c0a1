// Legendre-direction kernels.
//
//   k_recon  coefficients -> velocity at every quadrature plane
//            (channel/initAlphaBeta2.c:12-240, same arithmetic as the
//            reconstruction tail of channel/project.c:231-332)
//   k_solve  one RK3 substage of the implicit Galerkin step for a kz line:
//            quadrature right-hand side, banded solve, trajectory store and
//            next-substage right-hand side (channel/project.c:24-405,
//            project0.c:22-271, increproject*.c, adjproject*.c)
//
// Both exploit the parity of the Legendre bases on the symmetric Gauss
// points: Q_n, Q_n'', R_n are even/odd as (-1)^n and Q_n', R_n' as
// (-1)^(n+1), so for the plane pair (y, -y) a contraction splits into an
// even-index sum E and an odd-index sum O with values E +- O.  This halves
// the FP64 multiply-adds of every quadrature and reconstruction.
#include <type_traits>

#include "chn_common.cuh"
#include "kernels.h"
#include "solve_common.cuh"
#include "sizes.cuh"
#include "few_tile.cuh"
#include "tc_common.cuh"

namespace chn {

static constexpr int kThreads = 256;
static constexpr int kTile = 16;   // kx columns per block
static constexpr int kQuadRegs = 8;  // quadrature inputs a thread keeps in registers (Q <= 128)

__device__ __forceinline__ bool blocked(const uint32_t* status, int sdiv, int inst) {
  return status != nullptr && (status[inst / sdiv] & ST_CFL) != 0;
}

__device__ __forceinline__ void cfma(double w, const cpx& a, double& re, double& im) {
  re = fma(w, a.re, re);
  im = fma(w, a.im, im);
}

// ---------------------------------------------------------------------------
// reconstruction
// ---------------------------------------------------------------------------

template <bool MULTI>
__global__ void __launch_bounds__(kThreads) k_recon(const __grid_constant__ Grid g0, ReconArgs a) {
  const int ntx = (g0.X + kTile - 1) / kTile;
  const int z = blockIdx.x / ntx, tx = blockIdx.x - z * ntx;
  const int inst = blockIdx.y;
  CHN_INSTANCE_GRID(g0, a.grids, inst);
  if (z >= g.Nz || tx * kTile >= g.X) return;
  if (z == g.Nz / 2) return;  // never read (channel/pass1.c:51-85 skips it)
  if (blocked(a.status, a.sdiv, inst)) return;
  const int x0 = tx * kTile;
  const int nx = min(kTile, g.X - x0);
  extern __shared__ __align__(16) unsigned char smem[];
  cpx* cs = reinterpret_cast<cpx*>(smem);  // [2][R][kTile]
  const cpx* __restrict__ C = a.C.at(inst);
  if (a.slot.stride) C += (long long)a.slot.slot() * a.slot.stride;
  for (int i = threadIdx.x; i < 2 * g.R * kTile; i += blockDim.x) {
    const int v = i / (g.R * kTile), r = (i / kTile) % g.R, x = i % kTile;
    cpx val = {0.0, 0.0};
    if (x < nx) val = C[(((size_t)z * 2 + v) * g.R + r) * g.X + x0 + x];
    cs[i] = val;
  }
  __syncthreads();
  const int lx = threadIdx.x % kTile, grp = threadIdx.x / kTile;
  const int ngrp = blockDim.x / kTile;
  if (lx >= nx) return;
  const int x = x0 + lx;
  cpx* __restrict__ U = a.U.at(inst);
  const cpx* al = cs;                     // alpha_j at al[j*kTile + lx]
  const cpx* be = cs + g.R * kTile;       // beta_j
  const bool mean = (z == 0 && x == 0);
  const double ax = g.kxK2[z * g.X + x], az = g.kzK2[z * g.X + x];
  for (int yp = grp; yp < g.Qh; yp += ngrp) {
    const int y1 = yp, y2 = g.Q - 1 - yp;
    // E/O sums: [0] Q alpha (v), [1] Q' alpha, [2] Q'' alpha, [3] R beta, [4] R' beta
    double er[5] = {0, 0, 0, 0, 0}, ei[5] = {0, 0, 0, 0, 0};
    double orr[5] = {0, 0, 0, 0, 0}, oi[5] = {0, 0, 0, 0, 0};
    if (!mean) {
      const double* bq = g.Bq + (size_t)y1 * g.D;
      const double* bqp = g.Bqp + (size_t)y1 * g.D;
      const double* bqpp = g.Bqpp + (size_t)y1 * g.D;
      int j = 0;
      for (; j + 1 < g.D; j += 2) {
        const cpx c0 = al[j * kTile + lx], c1 = al[(j + 1) * kTile + lx];
        const double q0 = __ldg(bq + j), q1 = __ldg(bq + j + 1);
        const double p0 = __ldg(bqp + j), p1 = __ldg(bqp + j + 1);
        const double s0 = __ldg(bqpp + j), s1 = __ldg(bqpp + j + 1);
        cfma(q0, c0, er[0], ei[0]); cfma(q1, c1, orr[0], oi[0]);
        cfma(p0, c0, er[1], ei[1]); cfma(p1, c1, orr[1], oi[1]);
        cfma(s0, c0, er[2], ei[2]); cfma(s1, c1, orr[2], oi[2]);
      }
      if (j < g.D) {
        const cpx c0 = al[j * kTile + lx];
        cfma(__ldg(bq + j), c0, er[0], ei[0]);
        cfma(__ldg(bqp + j), c0, er[1], ei[1]);
        cfma(__ldg(bqpp + j), c0, er[2], ei[2]);
      }
    }
    {
      const double* br = g.Br + (size_t)y1 * g.R;
      const double* brp = g.Brp + (size_t)y1 * g.R;
      // mean mode: R a and R' a land in slots 1/2 (u, du), R b and R' b in 3/4
      const cpx* src0 = mean ? al : be;
      int j = 0;
      for (; j + 1 < g.R; j += 2) {
        const double r0 = __ldg(br + j), r1 = __ldg(br + j + 1);
        const double p0 = __ldg(brp + j), p1 = __ldg(brp + j + 1);
        const cpx b0 = be[j * kTile + lx], b1 = be[(j + 1) * kTile + lx];
        cfma(r0, b0, er[3], ei[3]); cfma(r1, b1, orr[3], oi[3]);
        cfma(p0, b0, er[4], ei[4]); cfma(p1, b1, orr[4], oi[4]);
        if (mean) {
          const cpx c0 = src0[j * kTile + lx], c1 = src0[(j + 1) * kTile + lx];
          cfma(r0, c0, er[1], ei[1]); cfma(r1, c1, orr[1], oi[1]);
          cfma(p0, c0, er[2], ei[2]); cfma(p1, c1, orr[2], oi[2]);
        }
      }
      if (j < g.R) {
        const double r0 = __ldg(br + j), p0 = __ldg(brp + j);
        const cpx b0 = be[j * kTile + lx];
        cfma(r0, b0, er[3], ei[3]);
        cfma(p0, b0, er[4], ei[4]);
        if (mean) {
          const cpx c0 = src0[j * kTile + lx];
          cfma(r0, c0, er[1], ei[1]);
          cfma(p0, c0, er[2], ei[2]);
        }
      }
    }
    for (int side = 0; side < 2; ++side) {
      if (side == 1 && y2 == y1) break;
      const int y = side ? y2 : y1;
      // even-parity bases: E + O / E - O;  odd-parity (Q', R'): E + O / -(E - O)
      auto val = [&](int c, bool odd_basis) {
        cpx r;
        if (!side) { r.re = er[c] + orr[c]; r.im = ei[c] + oi[c]; }
        else if (!odd_basis) { r.re = er[c] - orr[c]; r.im = ei[c] - oi[c]; }
        else { r.re = orr[c] - er[c]; r.im = oi[c] - ei[c]; }
        return r;
      };
      cpx u, v, w, du, dw;
      if (mean) {
        // (kx,kz) = (0,0): u = R a, du = R' a, v = 0, w = R b, dw = R' b
        u = val(1, false); du = val(2, true); w = val(3, false); dw = val(4, true);
        v.re = 0.0; v.im = 0.0;
      } else {
        v = val(0, false);
        const cpx qp = val(1, true);          // Q' alpha, f = -Q' alpha
        const cpx qpp = val(2, false);
        const cpx g_ = val(3, false);         // g = R beta
        const cpx rp = val(4, true);
        const cpx f = {-qp.re, -qp.im};
        // u = (kx Im f + kz Im g)/K2 - i (kx Re f + kz Re g)/K2, etc.
        u.re = fma(ax, f.im, az * g_.im);
        u.im = -fma(ax, f.re, az * g_.re);
        w.re = fma(-ax, g_.im, az * f.im);
        w.im = fma(ax, g_.re, -az * f.re);
        du.re = fma(-ax, qpp.im, az * rp.im);
        du.im = fma(ax, qpp.re, -az * rp.re);
        dw.re = -fma(ax, rp.im, az * qpp.im);
        dw.im = fma(ax, rp.re, az * qpp.re);
      }
      cpx* out = U + ((size_t)z * 5 * g.Q + y) * g.X + x;
      const size_t cs_ = (size_t)g.Q * g.X;
      out[0] = u;
      out[cs_] = v;
      out[2 * cs_] = w;
      out[3 * cs_] = du;
      out[4 * cs_] = dw;
    }
  }
}

size_t recon_smem_bytes(const Grid& g) { return (size_t)2 * g.R * kTile * sizeof(cpx); }

cudaError_t launch_recon(const Grid& g, const ReconArgs& a, cudaStream_t st) {
  if (a.ninst <= 0) return cudaSuccess;
  if (g.tc) return launch_recon_tc(g, a, st);
  const int ntx = (g.X + kTile - 1) / kTile;
  if (a.grids) k_recon<true><<<dim3(g.Nz * ntx, a.ninst), kThreads, recon_smem_bytes(g), st>>>(g, a);
  else k_recon<false><<<dim3(g.Nz * ntx, a.ninst), kThreads, recon_smem_bytes(g), st>>>(g, a);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// implicit solve
// ---------------------------------------------------------------------------

struct RKc {
  double b, c, dnext;
  int bidx, aidx0, aidx_next;
};

__device__ __forceinline__ RKc rk_coeffs(int k, int adjoint) {
  // forward  a = {1/3,-1/2,1/3}, b = {1/6,2/3,0}, c = {1/2,1/3,1}, d = {0,-1/6,-2/3}
  // adjoint  a = {1/3,-1/2,1/3}, b = {2/3,1/6,0}, c = {1,1/3,1/2}, d = {0,-2/3,-1/6}
  RKc r;
  if (!adjoint) {
    r.bidx = k;
    r.c = k == 0 ? 1. / 2 : (k == 1 ? 1. / 3. : 1.);
    r.dnext = k == 0 ? -1. / 6 : (k == 1 ? -2. / 3 : 0.0);
  } else {
    r.bidx = k == 0 ? 1 : (k == 1 ? 0 : 2);
    r.c = k == 0 ? 1. : (k == 1 ? 1. / 3. : 1. / 2.);
    r.dnext = k == 0 ? -2. / 3 : (k == 1 ? -1. / 6 : 0.0);
  }
  r.b = r.bidx == 0 ? 1. / 6 : (r.bidx == 1 ? 2. / 3 : 0.);
  r.aidx0 = 0;                         // a[0] = 1/3
  r.aidx_next = (k == 0) ? 1 : 0;      // a[1] = -1/2, a[2] = 1/3
  return r;
}

struct SolveSmem {
  cpx* hc;    // [Qh][kTile][6] parity-combined inputs (live during a quadrature)
  cpx* ra;    // [R][kTile] alpha right-hand side / solution (aliases hc: live between quadratures)
  cpx* rb;    // [R][kTile]
  cpx* Fa;    // [D][kTile]
  cpx* Fb;    // [R][kTile]
  // the FEW build's: digits of all inputs (dig; hc unused), staged factors
  uint16_t* dig;
  double *luA, *luB, *rdA, *rdB;  // [kTile][D][9], [kTile][R][5], [kTile][D], [kTile][R]
};

// The solve's functions below take the block's tile width (kx columns per
// block, 16 or 8: the autotuner's choice, Grid::stile) as the template
// parameter kTile, which stands for the file's 16 inside them.

// digits of one quadrature input for the tensor-core quadrature:
// [7][2 kTile columns][KS] fp16 + kTile exponents and the mean line's second
__host__ __device__ inline size_t solve_tc_kstride(const Grid& g) { return (size_t)((g.Q + 15) / 16) * 16 + 8; }

// the FP64 quadrature's parity-combined inputs only where it runs (g.tc = 0)
template <int kTile>
__host__ __device__ inline size_t solve_hc_elems(const Grid& g) {
  size_t hc = g.tc ? 0 : (size_t)g.Qh * kTile * 6, r = 2 * (size_t)g.R * kTile;
  const size_t tc =
      ((size_t)kDig * 2 * kTile * solve_tc_kstride(g) * 2 + (kTile + 1) * sizeof(int) + sizeof(cpx) - 1) / sizeof(cpx);
  if (r > hc) hc = r;
  return tc > hc ? tc : hc;
}

template <int kTile>
size_t solve_smem_bytes_t(const Grid& g) {
  return (solve_hc_elems<kTile>(g) + (size_t)g.D * kTile + (size_t)g.R * kTile) * sizeof(cpx);
}

// the widest tile's (the fit check of a grid)
size_t solve_smem_bytes(const Grid& g) { return solve_smem_bytes_t<16>(g); }
// what a grid is accepted by: eight doubles per coefficient row above the
// blocks' plan (the mean line's own arrays, when it had some), so that the
// range of Ny (up to 179) stays
size_t solve_smem_limit(const Grid& g) { return solve_smem_bytes(g) + (size_t)8 * g.R * sizeof(double); }

template <int kTile>
__device__ inline SolveSmem carve_solve(const Grid& g, unsigned char* base) {
  SolveSmem s;
  cpx* p = reinterpret_cast<cpx*>(base);
  s.hc = p;
  s.ra = p;
  s.rb = p + (size_t)g.R * kTile;
  p += solve_hc_elems<kTile>(g);
  s.Fa = p; p += (size_t)g.D * kTile;
  s.Fb = p;
  return s;
}

// The FEW build's plan: digits of the 3 inputs (5 for the adjoint), right-
// hand sides, F, the tile's factors
__host__ __device__ inline size_t solve_few_dig_bytes(const Grid& g, int tile, bool adj) {
  return ((size_t)(adj ? 5 : 3) * kDig * 2 * tile * solve_tc_kstride(g) * 2 + (5 * tile + 2) * sizeof(int) + 15) / 16 * 16;
}
inline size_t solve_few_smem_bytes(const Grid& g, int tile, bool adj) {
  return solve_few_dig_bytes(g, tile, adj) + (size_t)tile * (3 * g.R + g.D) * sizeof(cpx) +
         (size_t)tile * (10 * g.D + 6 * g.R) * sizeof(double);
}
template <int kTile>
__device__ inline SolveSmem carve_solve_few(const Grid& g, unsigned char* base, bool adj) {
  SolveSmem s;
  s.hc = nullptr;
  s.dig = reinterpret_cast<uint16_t*>(base);
  cpx* p = reinterpret_cast<cpx*>(base + solve_few_dig_bytes(g, kTile, adj));
  s.ra = p; p += (size_t)g.R * kTile;
  s.rb = p; p += (size_t)g.R * kTile;
  s.Fa = p; p += (size_t)g.D * kTile;
  s.Fb = p; p += (size_t)g.R * kTile;
  s.luA = reinterpret_cast<double*>(p);
  s.luB = s.luA + (size_t)kTile * g.D * 9;
  s.rdA = s.luB + (size_t)kTile * g.R * 5;
  s.rdB = s.rdA + (size_t)kTile * g.D;
  return s;
}

// the mean line's stand-ins for G and Sb (its two real quadratures as Re, Im)
__device__ __forceinline__ cpx mean_input(const cpx& u, const cpx& v, double sign) { return cpx{u.re, sign * v.re}; }

// Quadrature right-hand side for columns x0..x0+nx-1 of line z from terms H:
//   Fa = Qpw . i(kx Hx + kz Hz) - K2 Qw . Hy  [+ Qppw . -i(kz Sx - kx Sz)]
//   Fb = Rw . i(kz Hx - kx Hz)                [+ Rpw  .  i(kz Sz + kx Sx)]
// (channel/project.c:97-115, 177-191; channel/adjproject.c:113-134, 218-234)
template <int kTile>
__device__ void quad_rhs(const Grid& g, const cpx* __restrict__ H, int z, int x0, int nx, bool adj,
                         SolveSmem& s) {
  const int lx = threadIdx.x % kTile, grp = threadIdx.x / kTile, ngrp = blockDim.x / kTile;
  const double kz = g.Kz[z];
  const size_t cs = (size_t)g.Q * g.X;
  const cpx* Hz_ = H + (size_t)z * 5 * cs;  // slot c at Hz_ + c*cs + y*X + x
  for (int phase = 0; phase < 2; ++phase) {
    // phase 0: inputs of Fa (P, Hy, Sa); phase 1: inputs of Fb (G, Sb)
    const int nin = phase == 0 ? (adj ? 3 : 2) : (adj ? 2 : 1);
    for (int i = threadIdx.x; i < g.Qh * kTile; i += blockDim.x) {
      const int yp = i / kTile, l = i - yp * kTile;
      cpx* dst = s.hc + (size_t)i * 6;
      if (l >= nx) continue;
      const int x = x0 + l;
      const double kx = g.Kx[x];
      const int ya = yp, yb = g.Q - 1 - yp;
      cpx in[2][3];
      for (int side = 0; side < 2; ++side) {
        const int y = side ? yb : ya;
        const cpx hz = Hz_[0 * cs + (size_t)y * g.X + x];
        const cpx hx = Hz_[1 * cs + (size_t)y * g.X + x];
        if (phase == 0) {
          const cpx hy = Hz_[2 * cs + (size_t)y * g.X + x];
          in[side][0].re = -kx * hx.im - kz * hz.im;   // P = i(kx Hx + kz Hz)
          in[side][0].im = kx * hx.re + kz * hz.re;
          in[side][1] = hy;
          if (adj) {
            const cpx sx = Hz_[3 * cs + (size_t)y * g.X + x], sz = Hz_[4 * cs + (size_t)y * g.X + x];
            in[side][2].re = kz * sx.im - kx * sz.im;  // Sa = -i(kz Sx - kx Sz)
            in[side][2].im = -kz * sx.re + kx * sz.re;
          }
        } else {
          const bool mean = z == 0 && x == 0;
          in[side][0].re = -kz * hx.im + kx * hz.im;   // G = i(kz Hx - kx Hz)
          in[side][0].im = kz * hx.re - kx * hz.re;
          if (mean) in[side][0] = mean_input(hx, hz, 1.0);
          if (adj) {
            const cpx sx = Hz_[3 * cs + (size_t)y * g.X + x], sz = Hz_[4 * cs + (size_t)y * g.X + x];
            in[side][1].re = -kz * sz.im - kx * sx.im;  // Sb = i(kz Sz + kx Sx)
            in[side][1].im = kz * sz.re + kx * sx.re;
            if (mean) in[side][1] = mean_input(sz, sx, -1.0);
          }
        }
      }
      for (int q = 0; q < nin; ++q) {
        if (ya == yb) {  // centre plane of an odd point count
          dst[2 * q] = in[0][q];
          dst[2 * q + 1] = in[0][q];
        } else {
          dst[2 * q].re = in[0][q].re + in[1][q].re;      // "+" combination
          dst[2 * q].im = in[0][q].im + in[1][q].im;
          dst[2 * q + 1].re = in[0][q].re - in[1][q].re;  // "-" combination
          dst[2 * q + 1].im = in[0][q].im - in[1][q].im;
        }
      }
    }
    __syncthreads();
    if (lx < nx) {
      const int x = x0 + lx;
      const double k2 = g.K2[z * g.X + x];
      const int N = phase == 0 ? g.D : g.R;
      // rows i = grp, grp + ngrp, ... share the parity of grp (ngrp is even)
      constexpr int MAXR = 4;
      for (int ib = grp; ib < N; ib += ngrp * MAXR) {
        double sr[MAXR][3], si[MAXR][3];
#pragma unroll
        for (int m = 0; m < MAXR; ++m)
#pragma unroll
          for (int q = 0; q < 3; ++q) { sr[m][q] = 0.0; si[m][q] = 0.0; }
        const bool even = (ib & 1) == 0;
        for (int yp = 0; yp < g.Qh; ++yp) {
          const cpx* src = s.hc + ((size_t)yp * kTile + lx) * 6;
          if (phase == 0) {
            // even rows: Qpw (odd basis) pairs with "-", Qw and Qppw with "+"
            const cpx P = src[even ? 1 : 0];
            const cpx Hy = src[even ? 2 : 3];
            const cpx Sa = adj ? src[even ? 4 : 5] : cpx{0.0, 0.0};
#pragma unroll
            for (int m = 0; m < MAXR; ++m) {
              const int i = ib + m * ngrp;
              if (i < N) {
                const size_t o = (size_t)i * g.Q + yp;
                cfma(__ldg(g.Wqp + o), P, sr[m][0], si[m][0]);
                cfma(__ldg(g.Wq + o), Hy, sr[m][1], si[m][1]);
                if (adj) cfma(__ldg(g.Wqpp + o), Sa, sr[m][2], si[m][2]);
              }
            }
          } else {
            // even rows: Rw with "+", Rpw (odd basis) with "-"
            const cpx G = src[even ? 0 : 1];
            const cpx Sb = adj ? src[even ? 3 : 2] : cpx{0.0, 0.0};
#pragma unroll
            for (int m = 0; m < MAXR; ++m) {
              const int i = ib + m * ngrp;
              if (i < N) {
                const size_t o = (size_t)i * g.Q + yp;
                cfma(__ldg(g.Wr + o), G, sr[m][0], si[m][0]);
                if (adj) cfma(__ldg(g.Wrp + o), Sb, sr[m][1], si[m][1]);
              }
            }
          }
        }
#pragma unroll
        for (int m = 0; m < MAXR; ++m) {
          const int i = ib + m * ngrp;
          if (i >= N) continue;
          cpx f;
          if (phase == 0) {
            f.re = fma(-k2, sr[m][1], sr[m][0]) + sr[m][2];
            f.im = fma(-k2, si[m][1], si[m][0]) + si[m][2];
            s.Fa[i * kTile + lx] = f;
          } else {
            f.re = sr[m][0] + sr[m][1];
            f.im = si[m][0] + si[m][1];
            s.Fb[i * kTile + lx] = f;
          }
        }
      }
    }
    __syncthreads();
  }
}

// i (a u + b v), its roundings fixed: the builds of the quadratures agree bit for bit
__device__ __forceinline__ cpx imul_sum(double a, const cpx& u, double b, const cpx& v) {
  return cpx{-fma(a, u.im, __dmul_rn(b, v.im)), fma(a, u.re, __dmul_rn(b, v.re))};
}

// The same right-hand side on the tensor cores (tc_common.cuh): each input
// vector over the Q planes, per column, as base-256 digits (shared memory
// of the FP64 version's parity-combined inputs), times the digit tables of
// the weighted transposes; one FP64 rounding per contraction.
//   Fa = Qpw P - K2 Qw Hy [+ Qppw Sa],   Fb = Rw G [+ Rpw Sb]
template <int kTile, int NTHR, class S>
__device__ void quad_rhs_tc(const Grid& g, const S& gsz, const cpx* __restrict__ H, int z, int x0, int nx, bool adj,
                            SolveSmem& s) {
  constexpr int NC = 2 * kTile;  // digit columns: Re, Im of each kx column
  const int KT = (gsz.Q() + 15) / 16, MTw = (gsz.R() + 15) / 16;
  const size_t KS = (size_t)((gsz.Q() + 15) / 16) * 16 + 8;  // solve_tc_kstride
  uint16_t* dig = reinterpret_cast<uint16_t*>(s.hc);             // [7][NC][KS]
  int* exc = reinterpret_cast<int*>(dig + (size_t)kDig * NC * KS);  // [kTile], mean's Im
  const bool meancol = z == 0 && x0 == 0;
  const double kz = g.Kz[z];
  const size_t cs = (size_t)gsz.Q() * gsz.X();
  const cpx* Hz_ = H + (size_t)z * 5 * cs;  // slot c at Hz_ + c*cs + y*X + x
  // input q: 0 P = i(kx Hx + kz Hz), 1 Hy, 2 Sa = -i(kz Sx - kx Sz), 3 G = i(kz Hx - kx Hz),
  // 4 Sb = i(kz Sz + kx Sx); weight table: Qpw 1, Qw 0, Qppw 2, Rw 3, Rpw 4
  auto input = [&](int q, int y, int col) -> cpx {
    const int x = x0 + col;
    const double kx = g.Kx[x];
    const cpx* b = Hz_ + (size_t)y * gsz.X() + x;
    if (q >= 3 && z == 0 && x == 0) return q == 3 ? mean_input(b[cs], b[0], 1.0) : mean_input(b[4 * cs], b[3 * cs], -1.0);
    switch (q) {
      case 0: return imul_sum(kx, b[cs], kz, b[0]);
      case 1: return b[2 * cs];
      case 2: return imul_sum(-kz, b[3 * cs], kx, b[4 * cs]);
      case 3: return imul_sum(kz, b[cs], -kx, b[0]);
      default: return imul_sum(kz, b[4 * cs], kx, b[3 * cs]);
    }
  };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  const int NT = (2 * nx + 7) / 8;
  const uint4* __restrict__ W = reinterpret_cast<const uint4*>(g.tcW);
  const int qs[5] = {0, 1, 3, 2, 4};
  const int nq = adj ? 5 : 3;
  for (int iq = 0; iq < nq; ++iq) {
    const int q = adj ? iq : qs[iq];
    const int w = q == 0 ? 1 : (q == 1 ? 0 : q);
    const bool toA = q < 3;
    const int N = toA ? gsz.D() : gsz.R();
    cpx* F = toA ? s.Fa : s.Fb;
    const bool first = (q == 0 || q == 3);
    for (int i = threadIdx.x; i < kTile + 1; i += NTHR) exc[i] = 0;
    auto own = [&](int col) { return meancol && q >= 3 && col == 0; };
    __syncthreads();
    if (KT <= kQuadRegs && NTHR == 16 * kTile) {
      // thread t holds column t % kTile and the plane pairs 2 (t / kTile) +
      // 32 k, + 1 (entries 2 k, 2 k + 1): its inputs stay in registers from the
      // exponent maximum to the digits, which pack two planes a word
      const int col = threadIdx.x % kTile, y0 = 2 * (threadIdx.x / kTile);
      auto plane = [&](int k) { return y0 + 32 * (k >> 1) + (k & 1); };
      cpx vin[kQuadRegs];
      int emax = 0, eim = 0;
#pragma unroll
      for (int k = 0; k < kQuadRegs; ++k) {
        const int y = plane(k);
        vin[k] = (y < gsz.Q() && col < nx) ? input(q, y, col) : cpx{0.0, 0.0};
        column_exponents(vin[k], own(col), emax, eim);
      }
      if (emax) atomicMax(&exc[col], emax);
      if (eim) atomicMax(&exc[kTile], eim);
      __syncthreads();
      const int ex = exc[col] - 1022, exi = own(col) ? exc[kTile] - 1022 : ex;
#pragma unroll
      for (int k = 0; k < kQuadRegs; k += 2) {
        const int y = plane(k);
        if (y >= KT * 16) break;
        uint32_t* d = reinterpret_cast<uint32_t*>(dig + (size_t)(2 * col) * KS + y);
        digits_pair(scaled56(vin[k].re, ex), scaled56(vin[k + 1].re, ex), d, kTile * KS);
        digits_pair(scaled56(vin[k].im, exi), scaled56(vin[k + 1].im, exi), d + KS / 2, kTile * KS);
      }
    } else {
      for (int i = threadIdx.x; i < gsz.Q() * kTile; i += NTHR) {
        const int y = i / kTile, col = i - y * kTile;
        if (col >= nx) continue;
        const cpx v = input(q, y, col);
        int e = 0, eim = 0;
        column_exponents(v, own(col), e, eim);
        if (e) atomicMax(&exc[col], e);
        if (eim) atomicMax(&exc[kTile], eim);
      }
      __syncthreads();
      for (int i = threadIdx.x; i < KT * 8 * kTile; i += NTHR) {
        const int y = 2 * (i / kTile), col = i % kTile;
        const cpx v0 = (y < gsz.Q() && col < nx) ? input(q, y, col) : cpx{0.0, 0.0};
        const cpx v1 = (y + 1 < gsz.Q() && col < nx) ? input(q, y + 1, col) : cpx{0.0, 0.0};
        const int ex = exc[col] - 1022, exi = own(col) ? exc[kTile] - 1022 : ex;
        uint32_t* d = reinterpret_cast<uint32_t*>(dig + (size_t)(2 * col) * KS + y);
        digits_pair(scaled56(v0.re, ex), scaled56(v1.re, ex), d, kTile * KS);
        digits_pair(scaled56(v0.im, exi), scaled56(v1.im, exi), d + KS / 2, kTile * KS);
      }
    }
    __syncthreads();
    const int MTn = (N + 15) / 16;
    for (int item = warp; item < MTn * NT; item += NTHR >> 5) {
      const int mt = item / NT, nt = item - mt * NT;
      const int col = nt * 4 + t;
      const int ecol = col_exp(exc[min(col, kTile - 1)]) - 64 + LongFold().shift();
      const int ecoli = own(col) ? col_exp(exc[kTile]) - 64 + LongFold().shift() : ecol;
      long long T[4];
      uint32_t R[4] = {0, 0, 0, 0};
      tc_tile<true>(LongFold(), W + (size_t)w * MTw * KT * kDig * 32, mt, KT, kChunkKT, dig, KS, (size_t)NC * KS, nt * 8, lane, T,
                    R);
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int row = mt * 16 + gq + 8 * rr;
        if (row >= N || col >= nx) continue;
        const int e = g.tcWE[(size_t)w * gsz.R() + row];
        const cpx val = {round_sum(LongFold(), T[2 * rr], R[2 * rr], e + ecol),
                         round_sum(LongFold(), T[2 * rr + 1], R[2 * rr + 1], e + ecoli)};
        cpx& f = F[row * kTile + col];
        if (first) {
          f = val;
        } else if (q == 1) {
          const double k2 = g.K2[(size_t)z * gsz.X() + x0 + col];
          f.re = fma(-k2, val.re, f.re);
          f.im = fma(-k2, val.im, f.im);
        } else {
          f.re += val.re;
          f.im += val.im;
        }
      }
    }
    __syncthreads();
  }
}


// quad_rhs_tc for launches with few blocks (few_contract)
template <int kTile, int NTHR, int KP, class S>
__device__ void quad_rhs_few(const Grid& g, const S& gsz, const cpx* __restrict__ H, int z, int x0, int nx, bool adj,
                             SolveSmem& s) {
  const int col = threadIdx.x % kTile, x = x0 + min(col, nx - 1);
  const double kx = g.Kx[x], kz = g.Kz[z];
  const size_t cs = (size_t)gsz.Q() * gsz.X();
  const cpx* Hc = H + (size_t)z * 5 * cs + x;
  const bool mean = z == 0 && x == 0;
  const int lx = x0 + min((int)(threadIdx.x & 3), nx - 1);
  const double k2 = g.K2[(size_t)z * gsz.X() + lx];  // of this lane's output column
  few_contract<kTile, NTHR, KP>(
      gsz, g.tcW, g.tcWE, adj, nx, z == 0 && x0 == 0, s.dig,
      [&](int y, cpx (&o)[5]) {
        const cpx* b = Hc + (size_t)y * gsz.X();
        const cpx hz = b[0], hx = b[cs];
        o[0] = imul_sum(kx, hx, kz, hz);   // P
        o[1] = b[2 * cs];                  // Hy
        o[3] = mean ? mean_input(hx, hz, 1.0) : imul_sum(kz, hx, -kx, hz);  // G
        if (adj) {
          const cpx sx = b[3 * cs], sz = b[4 * cs];
          o[2] = imul_sum(-kz, sx, kx, sz);                                   // Sa
          o[4] = mean ? mean_input(sz, sx, -1.0) : imul_sum(kz, sz, kx, sx);  // Sb
        }
      },
      [](int q) { return q == 0 ? 1 : (q == 1 ? 0 : q); },  // Qpw P, Qw Hy, Qppw Sa, Rw G, Rpw Sb
      [&](int q, const cpx& f, const cpx& v) {
        if (q == 1) return cpx{fma(-k2, v.re, f.re), fma(-k2, v.im, f.im)};
        return cpx{f.re + v.re, f.im + v.im};
      },
      s.Fa, s.Fb);
}

// the banded solves of a tile: per column 4 chains for alpha, 4 for beta
// (parity x re/im), threads [0, 4 kTile) the alpha chains, as many from a
// warp boundary the beta ones: a warp holds one system (no divergence between
// the two bands).
template <int kTile, class S>
__device__ __forceinline__ void solve_chains(const Grid& g, const S& gsz, int bidx, int z, int x0, int nx, int xfirst,
                                             const SolveSmem& s) {
  constexpr int kHalf = 4 * kTile < 32 ? 32 : 4 * kTile;
  if (xfirst && (int)threadIdx.x >= 2 * kHalf) {  // the mean line's two, in a warp of their own
    const int t = (int)threadIdx.x - 2 * kHalf;
    if (t < 8)
      band_solve_chain<5, 2, 2>(g.lu0 + (size_t)bidx * gsz.R() * 5, g.rd0 + (size_t)bidx * gsz.R(), gsz.R(), t & 1,
                                      reinterpret_cast<double*>(t < 4 ? s.ra : s.rb) + ((t >> 1) & 1), 2 * kTile);
    return;
  }
  const bool beta = (int)threadIdx.x >= kHalf;
  const int t = beta ? (int)threadIdx.x - kHalf : (int)threadIdx.x, l = t / 4, par = t & 1, part = (t >> 1) & 1;
  if (t >= 4 * kTile || l >= nx || l < xfirst) return;
  const size_t sys = ((size_t)bidx * gsz.Nz() + z) * gsz.X() + x0 + l;
  if (!beta)
    band_solve_chain<9, 4, 4>(g.luA + sys * gsz.D() * 9, g.rdA + sys * gsz.D(), gsz.D(), par,
                              reinterpret_cast<double*>(s.ra + l) + part, 2 * kTile);
  else
    band_solve_chain<5, 2, 2>(g.luB + sys * gsz.R() * 5, g.rdB + sys * gsz.R(), gsz.R(), par,
                              reinterpret_cast<double*>(s.rb + l) + part, 2 * kTile);
}

// the same for the few-block build: chains of four lanes (alpha, warps 0 and
// 1) and of two (beta, warp 2; the mean line's, warp 3), the factors staged
template <int kTile, class S>
__device__ __forceinline__ void solve_chains_few(const Grid& g, const S& gsz, int bidx, int nx, int xfirst,
                                                 const SolveSmem& s) {
  static_assert(kTile == 4, "the thread map");
  const int tid = threadIdx.x;
  auto run = [&](auto nl, const double* LU, const double* RD, int W, int N, int par, bool on, double* b) {
    constexpr int NL = decltype(nl)::value;
    const int M = max((N - par + 1) / 2, 1), steps = (N + 1) / 2, l = tid & (NL - 1);
    double* bp = b + (N > par ? par * 2 * kTile : 0);
    on = on && N > par;
    chain_sweep<NL, false, false>(M, steps, l, on, bp, 4 * kTile, [&](int m, int t) {
      return LU[(size_t)(par + 2 * min(m + t, M - 1)) * W + NL - t]; }, [](int) { return 1.0; });
    __syncwarp();
    chain_sweep<NL, true, true>(M, steps, l, on, bp, 4 * kTile, [&](int m, int t) {
      return LU[(size_t)(par + 2 * max(m - t, 0)) * W + NL + t]; }, [&](int m) { return RD[par + 2 * m]; });
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

// The (kx, kz) = (0, 0) line (channel/project0.c, increproject0.c,
// adjproject0.c) is column 0 of the kz = 0 line's first tile: two real systems
// of the R basis (alpha and beta hold u and w), whose quadratures fa = Rw Hx
// [+ Rpw Sz] and fb = Rw Hz [- Rpw Sx] come out of the tile's beta contraction
// as Re and Im of Fb's column 0 (mean_input); they took one warp 115k cycles of
// the tile's block, more than the rest of it.

// Block z ntx + tx: kx tile tx of line z.  S: the sizes (SizesRT, or SizesCT for a specialised grid); NTHR
// threads (256, or 128 with the 8-column tile), MINB blocks per SM; FEW: the
// build for launches with few blocks (quad_rhs_few, staged factors)
template <bool MULTI, int kTile, class S, int NTHR = kThreads, int MINB = 2, int FEW = 0>
__global__ void __launch_bounds__(NTHR, MINB) k_solve(const __grid_constant__ Grid g0, SolveArgs a) {
  const int ntx = (g0.X + kTile - 1) / kTile;
  const int z = blockIdx.x / ntx, tx = blockIdx.x - z * ntx;
  const int inst = blockIdx.y;
  CHN_INSTANCE_GRID(g0, a.grids, inst);
  const S gsz(g);
  if (z >= gsz.Nz() || tx * kTile >= gsz.X()) return;
  if (blocked(a.status, a.sdiv, inst)) return;
  const int x0 = tx * kTile;
  const int nx = min(kTile, gsz.X() - x0);
  const size_t csz = coef_size(g);
  cpx* __restrict__ Cc = a.Cc.at(inst);
  cpx* __restrict__ So = a.Sout.at(inst);
  cpx* Tst = nullptr;
  int tslot = -1;
  if (a.T.base && (inst % a.tdiv) == a.tsel) {
    tslot = a.slot.slot();
    if (tslot >= 0) Tst = a.T.base + (long long)(inst / a.tdiv) * a.T.stride + (long long)tslot * a.slot.stride;
  }
  int mean_mode = a.mean_mode;
  if (mean_mode == MEAN_TAN_HOMOG && ((a.forced_mask >> (inst % a.mdiv)) & 1u)) mean_mode = MEAN_TAN_FORCED;
  auto cidx = [&](int v, int r, int x) { return (((size_t)z * 2 + v) * gsz.R() + r) * gsz.X() + x; };
  if (z == gsz.Nz() / 2) {
    // the Nz/2 line is zeroed every substage and never stored (channel/channel.c:460-467)
    for (int i = threadIdx.x; i < 2 * gsz.R() * nx; i += NTHR) {
      const int v = i / (gsz.R() * nx), r = (i / nx) % gsz.R(), x = x0 + i % nx;
      Cc[cidx(v, r, x)] = cpx{0.0, 0.0};
      So[cidx(v, r, x)] = cpx{0.0, 0.0};
    }
    return;
  }
  extern __shared__ __align__(16) unsigned char smem[];
  const RKc rk = rk_coeffs(a.k, a.adjoint);
  const bool adj = a.adjoint != 0;
  const double dt = g.dt;
  const int xfirst = (z == 0 && x0 == 0) ? 1 : 0;  // the mean mode has its own system
  // Re-sensitivity forcing of this tangent (kind 2: the reference's forcing
  // reconnected, channel/tangent_forcing.c + increproject.c:61-104, at the
  // first substage; kind 3: the exact derivative of the discrete step,
  // -re^2 dt (a_k D x_k + b_k D x_{k+1}) in every substage's right-hand side)
  int fkind = 0;
  const cpx* xk = nullptr;
  double ft1 = 0.0;
  if (a.re2_mask | a.re3_mask) {
    const uint32_t bit = 1u << (inst % a.mdiv);
    fkind = (a.re3_mask & bit) ? 3 : ((a.re2_mask & bit) ? 2 : 0);
    if (fkind) {
      const int xs = a.xslot.slot();
      xk = a.Xf.at(inst / a.xdiv) + (long long)xs * a.xslot.stride;
      if (a.Ftr) ft1 = a.Ftr[(long long)(inst / a.xdiv) * a.ftr_stride + xs + 1];
    }
  }
  const cpx* __restrict__ H = a.H.at(inst);
  SolveSmem s;
  if constexpr (FEW) {
    s = carve_solve_few<kTile>(g, smem, adj);
    stage_factors<NTHR>(g, gsz, (size_t)rk.bidx * gsz.Nz() * gsz.X() + (size_t)z * gsz.X() + x0, nx, s.luA, s.luB, s.rdA, s.rdB);
    quad_rhs_few<kTile, NTHR, FEW>(g, gsz, H, z, x0, nx, adj, s);
  } else {
    s = carve_solve<kTile>(g, smem);
    if (g.tc) quad_rhs_tc<kTile, NTHR>(g, gsz, H, z, x0, nx, adj, s);
    else quad_rhs<kTile>(g, H, z, x0, nx, adj, s);
  }
  const double re2 = g.re * g.re;
  const double ak = a.k == 1 ? -1. / 2 : 1. / 3.;  // forward a_k; b_k is rk.b
  if (fkind == 2 && a.k == 0) {
    // C += dt Mass^-1 F MC[3n+1] with F_alpha = -re^2 Dv, F_beta = re^2 (Rps + K2 Rs)
    __syncthreads();
    const cpx* x1 = xk + csz;
    for (int i = threadIdx.x; i < gsz.R() * kTile; i += NTHR) {
      const int r = i / kTile, l = i - r * kTile;
      if (l >= nx) continue;
      const int x = x0 + l;
      if (l < xfirst) {  // tangent_forcing0.c:31-41
        const cpx p = band_matvec_row(g.Rps, 5, 2, 2, gsz.R(), x1 + cidx(0, 0, 0), gsz.X(), r);
        const cpx q = band_matvec_row(g.Rps, 5, 2, 2, gsz.R(), x1 + cidx(1, 0, 0), gsz.X(), r);
        s.ra[r * kTile] = cpx{re2 * p.re, re2 * p.im};
        s.rb[r * kTile] = cpx{re2 * q.re, re2 * q.im};
        continue;
      }
      const double k2 = g.K2[(size_t)z * gsz.X() + x];
      if (r < gsz.D()) {
        const cpx v = visc_v_row(g, k2, x1 + cidx(0, 0, x), gsz.X(), r);
        s.ra[r * kTile + l] = cpx{-re2 * v.re, -re2 * v.im};
      }
      const cpx w = visc_g_row(g, k2, x1 + cidx(1, 0, x), gsz.X(), r);
      s.rb[r * kTile + l] = cpx{re2 * w.re, re2 * w.im};
    }
    __syncthreads();
    solve_chains<kTile>(g, gsz, 2, z, x0, nx, xfirst, s);  // mass matrices: the b = 0 factors
    __syncthreads();
    for (int i = threadIdx.x; i < gsz.R() * kTile; i += NTHR) {
      const int r = i / kTile, l = i - r * kTile;
      if (l >= nx) continue;
      const int x = x0 + l;
      if (r < gsz.D() || l < xfirst) {
        const cpx f = s.ra[r * kTile + l];
        Cc[cidx(0, r, x)].re += dt * f.re;
        Cc[cidx(0, r, x)].im += dt * f.im;
      }
      const cpx f = s.rb[r * kTile + l];
      Cc[cidx(1, r, x)].re += dt * f.re;
      Cc[cidx(1, r, x)].im += dt * f.im;
    }
    __syncthreads();
  }
  // right-hand sides (channel/project.c:60-81, 125-130, 143-163, 202-207)
  for (int i = threadIdx.x; i < gsz.R() * kTile; i += NTHR) {
    const int r = i / kTile, l = i - r * kTile;
    if (l >= nx) continue;
    const int x = x0 + l;
    const size_t zx = (size_t)z * gsz.X() + x;
    cpx va, vb;
    if (l < xfirst) {
      if (a.k == 0) {
        const double* E = g.ex0 + (size_t)rk.aidx0 * gsz.R() * 5;
        va = band_matvec_row(E, 5, 2, 2, gsz.R(), Cc + cidx(0, 0, 0), gsz.X(), r);
        vb = band_matvec_row(E, 5, 2, 2, gsz.R(), Cc + cidx(1, 0, 0), gsz.X(), r);
      } else {
        va = Cc[cidx(0, r, 0)];
        vb = Cc[cidx(1, r, 0)];
      }
      const cpx f = s.Fb[r * kTile];
      va.re += dt * rk.c * f.re;
      vb.re += dt * rk.c * f.im;
      if (fkind == 3) {
        // D0 = -Rps; the implicit term acts on the primal's solved mean flow
        // before its flux correction: MC[3n+k+1] - 0.5 flux_t add
        const cpx p0 = band_matvec_row(g.Rps, 5, 2, 2, gsz.R(), xk + cidx(0, 0, 0), gsz.X(), r);
        cpx p1 = band_matvec_row(g.Rps, 5, 2, 2, gsz.R(), xk + csz + cidx(0, 0, 0), gsz.X(), r);
        p1.re -= 0.5 * ft1 * rps_row_real(g, g.add0, r);
        const cpx q0 = band_matvec_row(g.Rps, 5, 2, 2, gsz.R(), xk + cidx(1, 0, 0), gsz.X(), r);
        const cpx q1 = band_matvec_row(g.Rps, 5, 2, 2, gsz.R(), xk + csz + cidx(1, 0, 0), gsz.X(), r);
        va.re += re2 * dt * ak * p0.re;
        va.im += re2 * dt * ak * p0.im;
        va.re += re2 * dt * rk.b * p1.re;
        va.im += re2 * dt * rk.b * p1.im;
        vb.re += re2 * dt * ak * q0.re;
        vb.im += re2 * dt * ak * q0.im;
        vb.re += re2 * dt * rk.b * q1.re;
        vb.im += re2 * dt * rk.b * q1.im;
      }
      s.ra[r * kTile] = va;
      s.rb[r * kTile] = vb;
      continue;
    }
    if (r < gsz.D()) {
      if (a.k == 0) {
        const double* E = g.exA + ((size_t)rk.aidx0 * gsz.Nz() * gsz.X() + zx) * gsz.D() * 9;
        va = band_matvec_row(E, 9, 4, 4, gsz.D(), Cc + cidx(0, 0, x), gsz.X(), r);
      } else {
        va = Cc[cidx(0, r, x)];
      }
      const cpx f = s.Fa[r * kTile + l];
      va.re += dt * rk.c * f.re;
      va.im += dt * rk.c * f.im;
      if (fkind == 3) {
        const double k2 = g.K2[zx];
        const cpx d0 = visc_v_row(g, k2, xk + cidx(0, 0, x), gsz.X(), r);
        const cpx d1 = visc_v_row(g, k2, xk + csz + cidx(0, 0, x), gsz.X(), r);
        va.re -= re2 * dt * ak * d0.re;
        va.im -= re2 * dt * ak * d0.im;
        va.re -= re2 * dt * rk.b * d1.re;
        va.im -= re2 * dt * rk.b * d1.im;
      }
    } else {
      va = Cc[cidx(0, r, x)];  // alpha rows >= Ny-4 ride along unchanged
    }
    if (a.k == 0) {
      const double* E = g.exB + ((size_t)rk.aidx0 * gsz.Nz() * gsz.X() + zx) * gsz.R() * 5;
      vb = band_matvec_row(E, 5, 2, 2, gsz.R(), Cc + cidx(1, 0, x), gsz.X(), r);
    } else {
      vb = Cc[cidx(1, r, x)];
    }
    const cpx f = s.Fb[r * kTile + l];
    vb.re += dt * rk.c * f.re;
    vb.im += dt * rk.c * f.im;
    if (fkind == 3) {  // beta: D = -(Rps + K2 Rs)
      const double k2 = g.K2[zx];
      const cpx d0 = visc_g_row(g, k2, xk + cidx(1, 0, x), gsz.X(), r);
      const cpx d1 = visc_g_row(g, k2, xk + csz + cidx(1, 0, x), gsz.X(), r);
      vb.re += re2 * dt * ak * d0.re;
      vb.im += re2 * dt * ak * d0.im;
      vb.re += re2 * dt * rk.b * d1.re;
      vb.im += re2 * dt * rk.b * d1.im;
    }
    s.ra[r * kTile + l] = va;
    s.rb[r * kTile + l] = vb;
  }
  __syncthreads();
  if constexpr (FEW) solve_chains_few<kTile>(g, gsz, rk.bidx, nx, xfirst, s);
  else solve_chains<kTile>(g, gsz, rk.bidx, z, x0, nx, xfirst, s);
  __syncthreads();
  if (xfirst) {
    // constant mass flux: a += 0.5 * flux_t * add (channel/project0.c:153-168), warp 0
    if (threadIdx.x < 32) {
      double part = 0.0;
      for (int i = threadIdx.x; i < gsz.R(); i += 32) part = fma(g.rwsum[i], s.ra[i * kTile].re, part);
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      double flux_t;
      if (mean_mode == MEAN_PRIMAL) flux_t = g.flux - part;
      else if (mean_mode == MEAN_TAN_FORCED) flux_t = 2.0 - part;
      else flux_t = -part;
      const double* add = g.add0 + (size_t)(adj ? 1 + rk.bidx : 0) * gsz.R();
      if (mean_mode == MEAN_PRIMAL && a.Fts && Tst && threadIdx.x == 0)
        a.Fts[(long long)(inst / a.tdiv) * a.fts_stride + tslot] = flux_t;
      for (int i = threadIdx.x; i < gsz.R(); i += 32) {
        double& v = s.ra[i * kTile].re;
        v = v + flux_t * add[i] * 0.5;
      }
    }
    __syncthreads();
  }
  // state rows: alpha from the solve (rows >= Ny-4 carried), beta from the solve
  for (int i = threadIdx.x; i < gsz.R() * kTile; i += NTHR) {
    const int r = i / kTile, l = i - r * kTile;
    if (l >= nx) continue;
    const int x = x0 + l;
    const cpx va = s.ra[r * kTile + l], vb = s.rb[r * kTile + l];
    So[cidx(0, r, x)] = va;
    So[cidx(1, r, x)] = vb;
    if (Tst) {
      Tst[cidx(0, r, x)] = va;
      Tst[cidx(1, r, x)] = vb;
    }
  }
  __syncthreads();
  if (a.k == 2) {
    // the carried array is the state after the last substage
    for (int i = threadIdx.x; i < gsz.R() * kTile; i += NTHR) {
      const int r = i / kTile, l = i - r * kTile;
      if (l >= nx) continue;
      const int x = x0 + l;
      Cc[cidx(0, r, x)] = So[cidx(0, r, x)];
      Cc[cidx(1, r, x)] = So[cidx(1, r, x)];
    }
    return;
  }
  // next-substage right-hand side: M(a[k+1]) state + dt d[k+1] F
  // (channel/project.c:352-404; adjoint F from the previous-stage terms,
  //  channel/adjproject.c:393-549)
  if (adj) {
    __syncthreads();
    if constexpr (FEW) {
      quad_rhs_few<kTile, NTHR, FEW>(g, gsz, a.Hprev.at(inst), z, x0, nx, true, s);
    } else {
      if (g.tc) quad_rhs_tc<kTile, NTHR>(g, gsz, a.Hprev.at(inst), z, x0, nx, true, s);
      else quad_rhs<kTile>(g, a.Hprev.at(inst), z, x0, nx, true, s);
    }
    __syncthreads();
  }
  // the solved state of this tile (So) is still in ra, rb unless the
  // adjoint's second quadrature overwrote them (they share its digit buffer)
  for (int i = threadIdx.x; i < gsz.R() * kTile; i += NTHR) {
    const int r = i / kTile, l = i - r * kTile;
    if (l >= nx) continue;
    const int x = x0 + l;
    const size_t zx = (size_t)z * gsz.X() + x;
    const cpx* ya = adj ? So + cidx(0, 0, x) : s.ra + l;
    const cpx* yb = adj ? So + cidx(1, 0, x) : s.rb + l;
    const int ys = adj ? gsz.X() : kTile;
    const bool mean = l < xfirst;
    const cpx f = s.Fb[r * kTile + l];
    cpx va = ya[r * ys];  // alpha rows >= Ny-4 carried
    if (mean) {
      va = band_matvec_row_t<5, 2, 2>(g.ex0 + (size_t)rk.aidx_next * gsz.R() * 5, gsz.R(), ya, ys, r);
      va.re += dt * rk.dnext * f.re;
    } else if (r < gsz.D()) {
      const double* E = g.exA + ((size_t)rk.aidx_next * gsz.Nz() * gsz.X() + zx) * gsz.D() * 9;
      va = band_matvec_row_t<9, 4, 4>(E, gsz.D(), ya, ys, r);
      const cpx fa = s.Fa[r * kTile + l];
      va.re += dt * rk.dnext * fa.re;
      va.im += dt * rk.dnext * fa.im;
    }
    const double* E = mean ? g.ex0 + (size_t)rk.aidx_next * gsz.R() * 5
                           : g.exB + ((size_t)rk.aidx_next * gsz.Nz() * gsz.X() + zx) * gsz.R() * 5;
    cpx vb = band_matvec_row_t<5, 2, 2>(E, gsz.R(), yb, ys, r);
    vb.re += dt * rk.dnext * (mean ? f.im : f.re);
    if (!mean) vb.im += dt * rk.dnext * f.im;
    Cc[cidx(0, r, x)] = va;
    Cc[cidx(1, r, x)] = vb;
  }
}

// The build for few blocks (4-column tiles, one block per SM): where its
// tiles are at most kFewTiles, CHN_SOLVE_TILE does not ask for a tile
// and the grid's tables and shared memory allow it.
static int s_solve_optin = 0;
static bool solve_few(const Grid& g, const SolveArgs& a) {
  if (a.grids || !g.tc || g.sfixed || g.Q <= 16 || g.Q > 256) return false;  // (a stream takes two k-tiles or more)
  if ((long long)g.Nz * ((g.X + 3) / 4) * a.ninst > kFewTiles) return false;
  return solve_few_smem_bytes(g, 4, a.adjoint != 0) + 1024 <= (size_t)s_solve_optin;
}

template <int T, class S, int NTHR = kThreads, int MINB = 2>
static void launch_solve_t(const Grid& g, const SolveArgs& a, cudaStream_t st) {
  const int ntx = (g.X + T - 1) / T;
  const dim3 grid(g.Nz * ntx, a.ninst);
  if (a.grids) k_solve<true, T, SizesRT, NTHR, MINB><<<grid, NTHR, solve_smem_bytes_t<T>(g), st>>>(g, a);
  else k_solve<false, T, S, NTHR, MINB><<<grid, NTHR, solve_smem_bytes_t<T>(g), st>>>(g, a);
}

// Grid::stile 16 or 8 columns in 256-thread blocks, or 8 columns in
// 128-thread blocks at 4 per SM (Grid::sthr 128)
template <class S>
static void launch_solve_s(const Grid& g, const SolveArgs& a, cudaStream_t st) {
  if (g.stile == 8 && g.sthr == 128) launch_solve_t<8, S, 128, 4>(g, a, st);
  else if (g.stile == 8) launch_solve_t<8, S>(g, a, st);
  else launch_solve_t<16, S>(g, a, st);
}

// the block tile of Grid::stile (8 or 16 kx columns; the same results), the
// build compiled for the grid's sizes where Grid::fixed & FIXED_SOLVE
cudaError_t launch_solve(const Grid& g, const SolveArgs& a, cudaStream_t st) {
  if (a.ninst <= 0) return cudaSuccess;
  if (solve_few(g, a)) {
    const dim3 grid(g.Nz * ((g.X + 3) / 4), a.ninst);
    const size_t sm = solve_few_smem_bytes(g, 4, a.adjoint != 0);
    const bool fx = (g.fixed & FIXED_SOLVE) != 0;
    if (fx && sizes_match<Sizes32>(g)) k_solve<false, 4, Sizes32, 256, 1, 1><<<grid, 256, sm, st>>>(g, a);
    else if (fx && sizes_match<Sizes16>(g)) k_solve<false, 4, Sizes16, 256, 1, 1><<<grid, 256, sm, st>>>(g, a);
    else if (g.Q <= 128) k_solve<false, 4, SizesRT, 256, 1, 1><<<grid, 256, sm, st>>>(g, a);
    else k_solve<false, 4, SizesRT, 256, 1, 2><<<grid, 256, sm, st>>>(g, a);
    return cudaGetLastError();
  }
  const bool fx = (g.fixed & FIXED_SOLVE) && !a.grids;
  if (fx && sizes_match<Sizes32>(g)) launch_solve_s<Sizes32>(g, a, st);
  else if (fx && sizes_match<Sizes16>(g)) launch_solve_s<Sizes16>(g, a, st);
  else launch_solve_s<SizesRT>(g, a, st);
  return cudaGetLastError();
}

void prepare_recon_solve(int optin) {
  s_solve_optin = optin;
  allow_max_smem(k_solve<false, 4, SizesRT, 256, 1, 1>, optin);
  allow_max_smem(k_solve<false, 4, SizesRT, 256, 1, 2>, optin);
  allow_max_smem(k_solve<false, 4, Sizes32, 256, 1, 1>, optin);
  allow_max_smem(k_solve<false, 4, Sizes16, 256, 1, 1>, optin);
  allow_max_smem(k_recon<false>, optin);
  allow_max_smem(k_recon<true>, optin);
  allow_max_smem(k_solve<false, 16, SizesRT>, optin);
  allow_max_smem(k_solve<true, 16, SizesRT>, optin);
  allow_max_smem(k_solve<false, 8, SizesRT>, optin);
  allow_max_smem(k_solve<true, 8, SizesRT>, optin);
  allow_max_smem(k_solve<false, 16, Sizes32>, optin);
  allow_max_smem(k_solve<false, 8, Sizes32>, optin);
  allow_max_smem(k_solve<false, 16, Sizes16>, optin);
  allow_max_smem(k_solve<false, 8, Sizes16>, optin);
  allow_max_smem(k_solve<false, 8, SizesRT, 128, 4>, optin);
  allow_max_smem(k_solve<true, 8, SizesRT, 128, 4>, optin);
  allow_max_smem(k_solve<false, 8, Sizes32, 128, 4>, optin);
  allow_max_smem(k_solve<false, 8, Sizes16, 128, 4>, optin);
}

}  // namespace chn
