// The transforms of grids whose planes do not fit one block (64x65x64,
// 128x129x128) as exact digit GEMMs: a z pass and an x pass with the spectral
// columns in an HBM intermediate
//   T[inst][c][Q][pz][X]   (c: field or product component),
// rounded to FP64 there.  The same tables, digits and folds as the one-block
// kernels (phys_tc.cu); a block takes 16 columns of one pass of one plane and
// component.  The FFT passes they replace are bound by the FP64 unit; the
// digit products, 28 a k-tile, run on the tensor cores and leave the FP64 unit
// the products and one conversion an output.  One instance at 128x129x128,
// six fields inverse / three products forward / six adjoint:
// 2.66 / 1.55 / 3.07 ms with the FFT passes, 1.52 / 0.87 / 1.50 here (the
// forward passes 1.21 / 2.22 before they were split radix-2).
#include <algorithm>

#include "chn_common.cuh"
#include "kernels.h"
#include "phys_common.cuh"
#include "phys_tc.cuh"
#include "setup.h"
#include "sizes.cuh"
#include "tc_common.cuh"

namespace chn {

static constexpr int kThreads = 256;
static constexpr int kWarps = kThreads / 32;
static constexpr int kCols = 16;    // columns per block of the z passes and the forward x pass
static constexpr int kRowsX = 32;   // rows m per block of the inverse x pass

__device__ __forceinline__ size_t t_plane(const Grid& g, int il, int nc, int c, int y) {
  return (((size_t)il * nc + c) * g.Q + y) * g.pz * g.X;
}

// ---------------------------------------------------------------------------
// inverse
// ---------------------------------------------------------------------------

static size_t z_inv_smem(const Grid& g) {
  const PhysTcDims d = phys_tc_dims(g, 1);
  return (size_t)kDig * kCols * d.KSz * 2 + (size_t)kCols * (g.Nz - 1) * sizeof(cpx) + kCols * sizeof(int);
}

// Z[m][x] = sum_kz F[kz][x] exp(+2 pi i m zp(kz)/pz) of kCols columns of one
// field and plane (the z stage of k_phys_inverse_tc)
__global__ void __launch_bounds__(kThreads, 2) k_z_inv_tc(const __grid_constant__ Grid g, PhysArgs a, int inst0, cpx* T) {
  const int y = blockIdx.x, il = blockIdx.y, inst = inst0 + il;
  const int nxc = (g.X + kCols - 1) / kCols, f = blockIdx.z / nxc, x0 = (blockIdx.z - f * nxc) * kCols;
  if (a.skip_blocked && blocked(a.status, a.sdiv, inst)) return;
  const PhysTcDims d = phys_tc_dims(g, 1);
  const int nx = min(kCols, g.X - x0), Kk = g.Nz - 1;
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* dig = reinterpret_cast<uint16_t*>(smem);
  cpx* Fin = reinterpret_cast<cpx*>(smem + (size_t)kDig * kCols * d.KSz * 2);  // [kk][column]
  int* exz = reinterpret_cast<int*>(Fin + (size_t)kCols * Kk);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  if (threadIdx.x < kCols) exz[threadIdx.x] = 0;
  __syncthreads();
  const cpx* __restrict__ U = a.U.at(inst);
  {
    const int n = threadIdx.x % kCols;
    int e = 0;
    for (int kk = threadIdx.x / kCols; kk < Kk; kk += kThreads / kCols) {
      cpx v = {0.0, 0.0};
      if (n < nx) v = field_value(g, U, f, kk < g.Nz / 2 ? kk : kk + 1, y, x0 + n);
      Fin[(size_t)kk * kCols + n] = v;
      e = max(e, max(exp_field(v.re), exp_field(v.im)));
    }
    e = max(e, __shfl_xor_sync(0xffffffffu, e, 16));
    if (lane < kCols) atomicMax(&exz[n], e);
  }
  __syncthreads();
  const size_t dstride = (size_t)kCols * d.KSz;
  {
    // lanes of a warp: 8 columns x 4 words, conflict-free stores of 16-byte-strided rows
    const int KW = d.KTz * 8;
    uint32_t* dw = reinterpret_cast<uint32_t*>(dig);
    for (int i = threadIdx.x; i < kCols * KW; i += kThreads) {
      const int n = (i & 7) + 8 * ((i >> 5) & 1), w = ((i >> 3) & 3) + 4 * (i >> 6);
      const int kk = g.tcZM[w];
      cpx v = {0.0, 0.0};
      if (kk >= 0) v = Fin[(size_t)kk * kCols + n];
      const int ex = exz[n] - 1022;
      digits_pair(scaled56(v.re, ex), scaled56(v.im, ex), dw + (size_t)n * d.KSz / 2 + w, dstride / 2);
    }
  }
  __syncthreads();
  const uint4* __restrict__ Az = reinterpret_cast<const uint4*>(g.tcZ);
  cpx* Tp = T + t_plane(g, il, a.nfields, f, y);
  const int NT = (nx + 7) / 8;
  for (int item = warp; item < d.MTz * NT; item += kWarps) {
    const int mt = item / NT, nt = item - mt * NT;
    long long TE[4], TO[4];
    uint32_t RE[4] = {0, 0, 0, 0}, RO[4] = {0, 0, 0, 0};
    tc_tile_range<true>(LongFold(), Az, mt, d.KTz, 0, d.KTzE, g.tcch, dig, d.KSz, dstride, nt * 8, lane, TE, RE);
    const Rests<true, LongFold> rE(RE);
    tc_tile_range<true>(LongFold(), Az, mt, d.KTz, d.KTzE, d.KTz, g.tcch, dig, d.KSz, dstride, nt * 8, lane, TO, RO);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = mt * 16 + gq + 8 * (r >> 1), n = nt * 8 + 2 * t + (r & 1);
      if (row >= 2 * d.pzh || n >= nx) continue;
      const int e = kZRowExp + col_exp(exz[n]) - 64 + LongFold().shift();
      const int im = row >= d.pzh, m = im ? row - d.pzh : row;
      bool bad = false;
      reinterpret_cast<double*>(Tp + (size_t)m * g.X + x0 + n)[im] = round_plus(LongFold(), TE[r], rE[r], TO[r], RO[r], e, bad);
      if (d.Rz == 2)
        reinterpret_cast<double*>(Tp + (size_t)(m + d.pzh) * g.X + x0 + n)[im] =
            round_minus(LongFold(), TE[r], rE[r], TO[r], RO[r], e, bad);
    }
  }
}

static size_t x_inv_smem(const Grid& g) {
  const PhysTcDims d = phys_tc_dims(g, 1);
  return (size_t)kDig * kRowsX * d.KSx * 2 + kRowsX * sizeof(int);
}

// P[m][xp] = Re Z[m][0] + 2 sum_{0<j<X} Re(Z[m][j] exp(+2 pi i j xp/px)) of
// kRowsX rows of one field and plane (the x stage of k_phys_inverse_tc)
__global__ void __launch_bounds__(kThreads, 3) k_x_inv_tc(const __grid_constant__ Grid g, PhysArgs a, int inst0,
                                                          const cpx* T) {
  const int y = blockIdx.x, il = blockIdx.y, inst = inst0 + il;
  const int nmc = (g.pz + kRowsX - 1) / kRowsX, f = blockIdx.z / nmc, m0 = (blockIdx.z - f * nmc) * kRowsX;
  if (a.skip_blocked && blocked(a.status, a.sdiv, inst)) return;
  const PhysTcDims d = phys_tc_dims(g, 1);
  const int nm = min(kRowsX, g.pz - m0);
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* dig = reinterpret_cast<uint16_t*>(smem);
  int* exx = reinterpret_cast<int*>(smem + (size_t)kDig * kRowsX * d.KSx * 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  const cpx* __restrict__ Tr = T + t_plane(g, il, a.nfields, f, y) + (size_t)m0 * g.X;
  // column exponents, a warp per row (not the imaginary part of the kx = 0
  // bin, which c2r ignores)
  for (int n = warp; n < kRowsX; n += kWarps) {
    int e = 0;
    for (int x = lane; x < g.X; x += 32) {
      const cpx v = n < nm ? Tr[(size_t)n * g.X + x] : cpx{0.0, 0.0};
      e = max(e, max(exp_field(v.re), x == 0 ? 0 : exp_field(v.im)));
    }
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) exx[n] = e;
  }
  __syncthreads();
  const size_t dstride = (size_t)kRowsX * d.KSx;
  {
    // K words: the even j, then the odd j; threads over j (coalesced)
    uint32_t* dw = reinterpret_cast<uint32_t*>(dig);
    const int KW = d.KTx * 8, WE = d.KTxE * 8;
    FlatRC rc(threadIdx.x, kThreads, KW);
    for (int i = threadIdx.x; i < kRowsX * KW; i += kThreads, rc.next()) {
      const int n = rc.r, w = rc.c;
      const int j = w < WE ? (w < d.nxE ? d.Rx * w : -1) : (w - WE < d.nxO ? 2 * (w - WE) + 1 : -1);
      cpx v = {0.0, 0.0};
      if (j >= 0 && n < nm) v = Tr[(size_t)n * g.X + j];
      if (j == 0) v.im = 0.0;
      const int ex = exx[n] - 1022;
      digits_pair(scaled56(v.re, ex), scaled56(v.im, ex), dw + (size_t)n * d.KSx / 2 + w, dstride / 2);
    }
  }
  __syncthreads();
  const uint4* __restrict__ Ax = reinterpret_cast<const uint4*>(g.tcX);
  double* __restrict__ P = a.P.at(inst);
  if (a.pslot.stride) P += (long long)a.pslot.slot() * a.pslot.stride;
  double* Pm = P + ((size_t)f * g.Q + y) * g.pz * g.px + (size_t)m0 * g.px;
  const int NT = (nm + 7) / 8;
  bool nonfinite = false;
  for (int item = warp; item < d.MTx * NT; item += kWarps) {
    const int mt = item / NT, nt = item - mt * NT;
    long long TE[4], TO[4];
    uint32_t RE[4] = {0, 0, 0, 0}, RO[4] = {0, 0, 0, 0};
    tc_tile_range(LongFold(), Ax, mt, d.KTx, 0, d.KTxE, g.tcch, dig, d.KSx, dstride, nt * 8, lane, TE, RE);
    const Rests<true, LongFold> rE(RE);
    tc_tile_range(LongFold(), Ax, mt, d.KTx, d.KTxE, d.KTx, g.tcch, dig, d.KSx, dstride, nt * 8, lane, TO, RO);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int xp = mt * 16 + gq + 8 * (r >> 1), n = nt * 8 + 2 * t + (r & 1);
      if (xp >= d.pxh || n >= nm) continue;
      const int e = g.tcXE[xp] + col_exp(exx[n]) - 64 + LongFold().shift();
      Pm[(size_t)n * g.px + xp] = round_plus(LongFold(), TE[r], rE[r], TO[r], RO[r], e, nonfinite);
      if (d.Rx == 2) Pm[(size_t)n * g.px + xp + d.pxh] = round_minus(LongFold(), TE[r], rE[r], TO[r], RO[r], e, nonfinite);
    }
  }
  if (nonfinite && a.status) atomicOr(&a.status[inst / a.sdiv], ST_NONFINITE);
}

// ---------------------------------------------------------------------------
// products and forward transforms
// ---------------------------------------------------------------------------

static size_t x_fwd_smem(const Grid& g) {
  const FwdTcDims d = fwd_tc_dims(g);
  return (size_t)kDig * kCols * d.KSx * 2 + (size_t)kCols * g.px * sizeof(double) + kCols * sizeof(int);
}

// component q of the products on kCols rows zp of a plane and their x
// transform Y[zp][kx] (the products and x stage of k_products_tc)
__global__ void __launch_bounds__(kThreads, 2) k_x_fwd_tc(const __grid_constant__ Grid g, ProdArgs a, int mode, int inst0,
                                                          cpx* T) {
  const int y = blockIdx.x, il = blockIdx.y, inst = inst0 + il;
  const int ncomp = mode >= 2 ? 6 : 3;
  const int q = blockIdx.z % ncomp, z0 = (blockIdx.z / ncomp) * kCols;  // components of the same rows side by side
  if (blocked(a.status, a.sdiv, inst)) return;
  const FwdTcDims d = fwd_tc_dims(g);
  const int nz = min(kCols, g.pz - z0);
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* dig = reinterpret_cast<uint16_t*>(smem);
  double* st = reinterpret_cast<double*>(smem + (size_t)kDig * kCols * d.KSx * 2);  // [zp][xp]
  int* exx = reinterpret_cast<int*>(st + (size_t)kCols * g.px);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  const size_t plane = (size_t)g.pz * g.px, fs = (size_t)g.Q * plane;
  const size_t off = (size_t)y * plane + (size_t)z0 * g.px;
  const double* __restrict__ Pp = a.Pp.base + (long long)(inst / a.pdiv) * a.Pp.stride + off +
                                  (a.pslot.stride ? (long long)a.pslot.slot() * a.pslot.stride : 0LL);
  const double* __restrict__ Pt = a.Pt.base ? a.Pt.at(inst) + off : nullptr;
  // a warp per row: products, the row's exponent
  for (int n = warp; n < kCols; n += kWarps) {
    int e = 0;
    for (int xp = lane; xp < g.px; xp += 32) {
      const double v = n < nz ? split_product(mode, Pp, Pt, fs, (size_t)n * g.px + xp, q) : 0.0;
      st[(size_t)n * g.px + xp] = v;
      e = max(e, exp_field(v));
    }
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) exx[n] = e;
  }
  __syncthreads();
  const size_t dstride = (size_t)kCols * d.KSx;
  {
    FlatRC rc(threadIdx.x, kThreads, d.KTxc * 8);
    for (int i = threadIdx.x; i < kCols * (d.KTxc * 8); i += kThreads, rc.next())
      fwd_x_digits(d, st + (size_t)rc.r * g.px, 2 * rc.c, true, exx[rc.r] - 1022,
                   reinterpret_cast<uint32_t*>(dig + (size_t)rc.r * d.KSx), dstride / 2);
  }
  __syncthreads();
  const uint4* __restrict__ Ax = reinterpret_cast<const uint4*>(mode == 3 ? g.tcFXU : g.tcFX);
  const int* __restrict__ AxE = mode == 3 ? g.tcFXUE : g.tcFXE;
  cpx* Tp = T + t_plane(g, il, ncomp, q, y) + (size_t)z0 * g.X;
  const int NT = (nz + 7) / 8;
  for (int item = warp; item < d.MTx * NT; item += kWarps) {
    const int mt = item / NT, nt = item - mt * NT;
    long long S[4];
    uint32_t R[4] = {0, 0, 0, 0};
    tc_tile<true>(LongFold(), Ax, mt, d.KTxc, kChunkKT, dig + (mt >= d.MTxE ? d.KTxc * 16 : 0), d.KSx, dstride, nt * 8, lane, S, R);
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      FwdRow row;
      if (!fwd_row(mt, gq + 8 * rr, d.MTxE, d.nxE, d.nxO, row)) continue;
      const int kx = 2 * row.e + row.cls, er = AxE[2 * (row.cls * d.nxE + row.e) + row.part] - 64 + LongFold().shift();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int n = nt * 8 + 2 * t + c;
        if (n >= nz) continue;
        reinterpret_cast<double*>(Tp + (size_t)n * g.X + kx)[row.part] = round_sum(LongFold(), S[2 * rr + c], R[2 * rr + c], er + col_exp(exx[n]));
      }
    }
  }
}

static size_t z_fwd_smem(const Grid& g) {
  const FwdTcDims d = fwd_tc_dims(g);
  return (size_t)kDig * kCols * d.KSz * 2 + kCols * sizeof(int);
}

// F[kz][kx] = sum_zp Y[zp][kx] exp(-2 pi i zp(kz) zp/pz) of kCols columns (the
// z stage of k_products_tc); modes 0, 1 into H, the adjoint modes over the
// columns just read (their kept rows first), for k_assemble
__global__ void __launch_bounds__(kThreads, 2) k_z_fwd_tc(const __grid_constant__ Grid g, ProdArgs a, int mode, int inst0,
                                                          cpx* T) {
  const int y = blockIdx.x, il = blockIdx.y, inst = inst0 + il;
  const int ncomp = mode >= 2 ? 6 : 3, nxc = (g.X + kCols - 1) / kCols;
  const int q = blockIdx.z / nxc, x0 = (blockIdx.z - q * nxc) * kCols;
  if (blocked(a.status, a.sdiv, inst)) return;
  const FwdTcDims d = fwd_tc_dims(g);
  const int nx = min(kCols, g.X - x0);
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* dig = reinterpret_cast<uint16_t*>(smem);
  int* exz = reinterpret_cast<int*>(smem + (size_t)kDig * kCols * d.KSz * 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  cpx* Tc = T + t_plane(g, il, ncomp, q, y) + x0;
  if (threadIdx.x < kCols) exz[threadIdx.x] = 0;
  __syncthreads();
  {
    const int n = threadIdx.x % kCols;
    int e = 0;
    if (n < nx)
      for (int zp = threadIdx.x / kCols; zp < g.pz; zp += kThreads / kCols) {
        const cpx v = Tc[(size_t)zp * g.X + n];
        e = max(e, max(exp_field(v.re), exp_field(v.im)));
      }
    e = max(e, __shfl_xor_sync(0xffffffffu, e, 16));
    if (lane < kCols) atomicMax(&exz[n], e);
  }
  __syncthreads();
  const size_t dstride = (size_t)kCols * d.KSz;
  {
    const int KW = d.KTzc * 8;
    uint32_t* dw = reinterpret_cast<uint32_t*>(dig);
    for (int i = threadIdx.x; i < kCols * KW; i += kThreads) {
      const int n = (i & 7) + 8 * ((i >> 5) & 1), zp = ((i >> 3) & 3) + 4 * (i >> 6), ex = exz[n] - 1022;
      auto input = [&](int z) {
        const cpx v = (n < nx && zp < d.pzh) ? Tc[(size_t)z * g.X + n] : cpx{0.0, 0.0};
        return make_longlong2(scaled56(v.re, ex), scaled56(v.im, ex));
      };
      const longlong2 u = input(zp), v = d.Rz == 2 ? input(zp + d.pzh) : u;
      fwd_z_digits(d, zp, u, v, dw + (size_t)n * d.KSz / 2, dstride / 2);
    }
  }
  __syncthreads();
  const uint4* __restrict__ Az = reinterpret_cast<const uint4*>(g.tcFZ);
  cpx* __restrict__ H = a.H.at(inst);
  const int NT = (nx + 7) / 8;
  for (int item = warp; item < d.MTz * NT; item += kWarps) {
    const int mt = item / NT, nt = item - mt * NT;
    long long S[4];
    uint32_t R[4] = {0, 0, 0, 0};
    tc_tile<true>(LongFold(), Az, mt, d.KTzc, kChunkKT, dig + (mt >= d.MTzE ? d.KTzc * 16 : 0), d.KSz, dstride, nt * 8, lane, S, R);
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      FwdRow row;
      if (!fwd_row(mt, gq + 8 * rr, d.MTzE, d.nzE, d.nzO, row)) continue;
      const int er = g.tcFZE[2 * (row.cls * d.nzE + row.e) + row.part] - 64 + LongFold().shift();
      const int kk = fwd_z_mode(g.Nz, d.Rz, row.cls, row.e), z = kk < g.Nz / 2 ? kk : kk + 1;
      cpx* out = mode < 2 ? H + (((size_t)z * 5 + q) * g.Q + y) * g.X + x0 : Tc + (size_t)kk * g.X;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int n = nt * 8 + 2 * t + c;
        if (n < nx) reinterpret_cast<double*>(out + n)[row.part] = round_sum(LongFold(), S[2 * rr + c], R[2 * rr + c], er + col_exp(exz[n]));
      }
    }
  }
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------

bool phys_tcs_fits(const Grid& g, int optin) {
  const size_t room = (size_t)optin - 1024;
  return z_inv_smem(g) <= room && x_inv_smem(g) <= room && x_fwd_smem(g) <= room && z_fwd_smem(g) <= room;
}

// Narrow planes that fit one block of the FFT kernels (X <= 8 from about Nz = 112
// on) fill few of a z pass's 16 columns, and their DFTs' work grows with Nz^2: batches
// of them run the FFTs.  A launch of few planes, one FFT block each, leaves the
// chip idle and takes the passes.  Inverse of instances of 4x17x128, FFTs against
// passes: 2 (50 planes) 0.049 / 0.066 ms, 64 0.374 / 1.85; 8x17x128: 2 0.087 /
// 0.066, 4 0.102 / 0.121, 64 0.78 / 1.91; 12x17x128: 4 (100 planes) 0.124 / 0.126,
// 32 0.78 / 1.01; 16x33x128 (X = 8, radix 2 and 3): 8 0.562 / 0.519, 32 1.88 /
// 1.98; 16x17x112 (radix 7): 32 1.11 / 0.93; 20x17x108: 32 1.41 / 1.16.
bool split_tc_inverse(const Grid& g, int ninst) {
  const long long planes = (long long)g.Q * ninst;
  if (!g.fused || g.X > 8) return true;
  if (g.X == 8) return g.general || planes <= 3 * 152;
  return planes <= 16 * g.X;
}

cudaError_t launch_phys_inverse_tcs(const Grid& g, const PhysArgs& a, cudaStream_t st) {
  const int cap = a.tmp_inst * 6 / a.nfields;
  for (int i0 = 0; i0 < a.ninst; i0 += cap) {
    const int n = std::min(cap, a.ninst - i0);
    k_z_inv_tc<<<dim3(g.Q, n, a.nfields * ((g.X + kCols - 1) / kCols)), kThreads, z_inv_smem(g), st>>>(g, a, i0, a.tmp);
    k_x_inv_tc<<<dim3(g.Q, n, a.nfields * ((g.pz + kRowsX - 1) / kRowsX)), kThreads, x_inv_smem(g), st>>>(g, a, i0, a.tmp);
  }
  if (a.cfl_check) launch_cfl(g, a, st);
  return cudaGetLastError();
}

cudaError_t launch_products_tcs(const Grid& g, const ProdArgs& a, int mode, cudaStream_t st) {
  const int nc = mode >= 2 ? 6 : 3, cap = a.tmp_inst * 6 / nc;
  for (int i0 = 0; i0 < a.ninst; i0 += cap) {
    const int n = std::min(cap, a.ninst - i0);
    k_x_fwd_tc<<<dim3(g.Q, n, nc * ((g.pz + kCols - 1) / kCols)), kThreads, x_fwd_smem(g), st>>>(g, a, mode, i0, a.tmp);
    k_z_fwd_tc<<<dim3(g.Q, n, nc * ((g.X + kCols - 1) / kCols)), kThreads, z_fwd_smem(g), st>>>(g, a, mode, i0, a.tmp);
    if (mode >= 2) launch_assemble(g, a, mode == 3, i0, n, st);
  }
  return cudaGetLastError();
}

void prepare_phys_tcs(int optin) {
  allow_max_smem(k_z_inv_tc, optin);
  allow_max_smem(k_x_inv_tc, optin);
  allow_max_smem(k_x_fwd_tc, optin);
  allow_max_smem(k_z_fwd_tc, optin);
}

}  // namespace chn
