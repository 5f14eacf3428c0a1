// The inverse 3/2-padded transforms (channel/pass1.c:42-114,
// channel/spec2phys.c:39-76) as exact digit GEMMs on the tensor cores.
//
// One block per (instance, plane y), one or two fields per pass:
//   z stage   Z[m][x] = sum_kz F[kz][x] exp(+2 pi i m zp(kz)/pz) over the
//             Nz - 1 kept rows, one column per (field, x);
//   x stage   P[m][xp] = Re Z[m][0] + 2 sum_{0<j<X} Re(Z[m][j] exp(+2 pi i j xp/px))
//             (the complex-to-real transform; the imaginary part of the
//             kx = 0 bin is ignored as by c2r), one column per m.
// Each stage is split radix-2 where its length n is even: with
// exp(2 pi i k (m + n/2)/n) = (-1)^k exp(2 pi i k m/n), the outputs m and
// m + n/2 are E + O and E - O for the sums E, O over the even and odd k, so
// a stage is one GEMM with half the rows (m < n/2) whose K holds the even
// modes and then the odd ones; the two partial sums stay exact 64-bit
// integers (the E and O rows of a table share their row exponent) and their
// sum and difference are rounded once each.  z stage: rows Re, Im of
// Z[m < pz/2] (2 pz/2 rows), K = Re, Im of the even-zp and odd-zp modes;
// x stage: rows xp < px/2, K = Re, Im of the even and odd j.  An odd length
// keeps one class (the full DFT).
// The DFT matrices hold the FFT's own twiddle doubles; operands are base-256
// digits with exact FP32 level sums (tc_common.cuh), so each output is the
// (faithfully) rounded value of the exact sum of the 56-bit operands.  The
// intermediate Z stays a folded 64-bit sum in shared memory between the stages.  Same outputs,
// CFL check and status bits as k_phys_inverse.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>
#include <vector>

#include "chn_common.cuh"
#include "kernels.h"
#include "phys_common.cuh"
#include "setup.h"
#include "phys_tc.cuh"
#include "sizes.cuh"
#include "tc_common.cuh"

namespace chn {

static constexpr int kThreads = 256;

// ---------------------------------------------------------------------------
// host tables
// ---------------------------------------------------------------------------

// the kept kz modes of one class of the z stage's radix-2 split (padded
// index zp even or odd; the only class for an odd pz)
static void z_class_modes(int Nz, int pz, int cls, std::vector<int>& kk_of) {
  kk_of.clear();
  for (int kk = 0; kk < Nz - 1; ++kk) {
    const int zp = kk < Nz / 2 ? kk : kk + 1 + Nz / 2;  // padded row of kept kz index kk
    if (pz % 2 || (zp & 1) == cls) kk_of.push_back(kk);
  }
}

// the two stages' matrices (rows x K words of Re, Im) and the z stage's
// K-word -> kept kz map, shared by the mma.sync tables below and the
// tcgen05 tables of phys_tc5.cu
bool phys_tc_matrices(const HostTables& h, std::vector<double>& Az, std::vector<double>& Ax,
                      std::vector<int>& zmap, int& zrows, int& Kz, int& xrows, int& Kx) {
  const int pz = h.pz, px = h.px, Nz = h.Nz, X = h.X;
  const int Rz = pz % 2 ? 1 : 2, Rx = px % 2 ? 1 : 2, pzh = pz / Rz, pxh = px / Rx;
  std::vector<int> zE, zO;
  z_class_modes(Nz, pz, 0, zE);
  if (Rz == 2) z_class_modes(Nz, pz, 1, zO);
  int nE = 0, nO = 0;
  z_class_counts(Nz, pz, nE, nO);  // the kernel's closed form
  if (nE != (int)zE.size() || nO != (int)zO.size()) return false;
  const int nxE = (X + Rx - 1) / Rx, nxO = X - nxE;
  const int KTzE = (2 * (int)zE.size() + 15) / 16, KTzO = (2 * (int)zO.size() + 15) / 16;
  const int KTxE = (2 * nxE + 15) / 16, KTxO = (2 * nxO + 15) / 16;
  Kz = (KTzE + KTzO) * 16;
  Kx = (KTxE + KTxO) * 16;
  zrows = 2 * pzh;
  xrows = pxh;
  // z stage: rows Re Z[m], Im Z[m] (m < pzh); K words: even modes, then odd
  Az.assign((size_t)2 * pzh * Kz, 0.0);
  Ax.assign((size_t)pxh * Kx, 0.0);
  zmap.assign((size_t)Kz / 2, -1);
  for (int c = 0; c < 2; ++c) {
    const std::vector<int>& modes = c ? zO : zE;
    const int w0 = c ? KTzE * 8 : 0;
    for (int e = 0; e < (int)modes.size(); ++e) {
      const int kk = modes[e], zp = kk < Nz / 2 ? kk : kk + 1 + Nz / 2, w = w0 + e;
      zmap[w] = kk;
      for (int m = 0; m < pzh; ++m) {
        const int idx = (int)(((long long)m * zp) % pz);
        const double cs = h.twz[2 * idx], sn = -h.twz[2 * idx + 1];  // exp(+i theta) = conj(exp(-i theta))
        Az[(size_t)m * Kz + 2 * w] = cs;
        Az[(size_t)m * Kz + 2 * w + 1] = -sn;
        Az[(size_t)(pzh + m) * Kz + 2 * w] = sn;
        Az[(size_t)(pzh + m) * Kz + 2 * w + 1] = cs;
      }
    }
  }
  // x stage: rows xp < pxh; K words: j = Rx e (even), then j = 2 o + 1 (odd)
  for (int w = 0; w < Kx / 2; ++w) {
    int j;
    if (w < KTxE * 8) {
      if (w >= nxE) continue;
      j = Rx * w;
    } else {
      const int o = w - KTxE * 8;
      if (o >= nxO) continue;
      j = 2 * o + 1;
    }
    for (int xp = 0; xp < pxh; ++xp) {
      if (j == 0) {
        Ax[(size_t)xp * Kx + 2 * w] = 1.0;
        continue;
      }
      const int idx = (int)(((long long)j * xp) % px);
      const double cs = h.twx[2 * idx], sn = -h.twx[2 * idx + 1];
      Ax[(size_t)xp * Kx + 2 * w] = 2.0 * cs;
      Ax[(size_t)xp * Kx + 2 * w + 1] = -2.0 * sn;
    }
  }
  return true;
}

int build_phys_tc_tables(const HostTables& h, std::vector<uint32_t>& zfrag, std::vector<int>& zex,
                         std::vector<uint32_t>& xfrag, std::vector<int>& xex, std::vector<int>& zmap, bool& long_rows) {
  long_rows = false;
  std::vector<double> Az, Ax;
  int zrows = 0, Kz = 0, xrows = 0, Kx = 0;
  if (!phys_tc_matrices(h, Az, Ax, zmap, zrows, Kz, xrows, Kx)) return 0;
  zfrag.clear(); zex.clear(); xfrag.clear(); xex.clear();
  // one table per stage with both classes in its K: a row's exponent covers
  // its even and odd parts, so their integer sums add exactly
  const int cz = append_digit_table(Az.data(), zrows, Kz, (zrows + 15) / 16, Kz / 16, zfrag, zex, 256, &long_rows);
  const int cx = append_digit_table(Ax.data(), xrows, Kx, (xrows + 15) / 16, Kx / 16, xfrag, xex, 256, &long_rows);
  for (int e : zex)
    if (e != kZRowExp) return 0;  // (every row holds a 1: exp(0) of kz = 0)
  return std::min(cz, cx);
}

// forward transforms (channel/pass1.c:312-339): x stage Y[zp][kx] =
// norm sum_xp p[zp][xp] exp(-2 pi i kx xp/px) for kx < X (rows 2kx, 2kx+1 =
// Re, Im; the 1/(px pz) scaling folded in, Ax; the exact transpose's products
// take an unscaled copy, Au), z stage F[kz][kx] = sum_zp
// Y[zp][kx] exp(-2 pi i zp(kz) zp/pz) for the Nz - 1 kept rows (Az: rows 2kk,
// 2kk+1; K = 2 pz with Re, Im of Y interleaved)
static void fwd_tc_matrices(const HostTables& h, std::vector<double>& Ax, std::vector<double>& Au, std::vector<double>& Az) {
  const int pz = h.pz, px = h.px, Nz = h.Nz, X = h.X, Kk = Nz - 1;
  const double norm = 1.0 / ((3. * h.Nx / 2.) * (3. * h.Nz / 2.));
  Ax.assign((size_t)2 * X * px, 0.0);
  Au.assign((size_t)2 * X * px, 0.0);
  Az.assign((size_t)2 * Kk * 2 * pz, 0.0);
  for (int kx = 0; kx < X; ++kx)
    for (int xp = 0; xp < px; ++xp) {
      const int idx = (int)(((long long)kx * xp) % px);
      Au[(size_t)(2 * kx) * px + xp] = h.twx[2 * idx];           // cos
      Au[(size_t)(2 * kx + 1) * px + xp] = h.twx[2 * idx + 1];   // -sin
      Ax[(size_t)(2 * kx) * px + xp] = h.twx[2 * idx] * norm;
      Ax[(size_t)(2 * kx + 1) * px + xp] = h.twx[2 * idx + 1] * norm;
    }
  for (int kk = 0; kk < Kk; ++kk) {
    const int zo = kk < Nz / 2 ? kk : kk + 1 + Nz / 2;  // padded output row of kept index kk
    for (int zp = 0; zp < pz; ++zp) {
      const int idx = (int)(((long long)zo * zp) % pz);
      const double c = h.twz[2 * idx], ms = h.twz[2 * idx + 1];  // cos, -sin
      Az[(size_t)(2 * kk) * 2 * pz + 2 * zp] = c;
      Az[(size_t)(2 * kk) * 2 * pz + 2 * zp + 1] = -ms;
      Az[(size_t)(2 * kk + 1) * 2 * pz + 2 * zp] = ms;
      Az[(size_t)(2 * kk + 1) * 2 * pz + 2 * zp + 1] = c;
    }
  }
}

// the matrices as whole tables (c_setup_tc_table: they show what the split
// tables below take their rows from)
int build_fwd_tc_tables(const HostTables& h, std::vector<uint32_t>& xfrag, std::vector<int>& xex,
                        std::vector<uint32_t>& zfrag, std::vector<int>& zex, std::vector<uint32_t>& ufrag,
                        std::vector<int>& uex) {
  const int pz = h.pz, px = h.px, X = h.X, Kk = h.Nz - 1;
  std::vector<double> Ax, Au, Az;
  fwd_tc_matrices(h, Ax, Au, Az);
  xfrag.clear(); xex.clear(); zfrag.clear(); zex.clear(); ufrag.clear(); uex.clear();
  const int cx = append_digit_table(Ax.data(), 2 * X, px, (2 * X + 15) / 16, (px + 15) / 16, xfrag, xex);
  const int cu = append_digit_table(Au.data(), 2 * X, px, (2 * X + 15) / 16, (px + 15) / 16, ufrag, uex);
  const int cz = append_digit_table(Az.data(), 2 * Kk, 2 * pz, (2 * Kk + 15) / 16, (2 * pz + 15) / 16, zfrag, zex);
  return std::min(cx, std::min(cu, cz));
}

// The same stages split radix-2 (decimation in frequency) as the kernels run
// them: per class the rows 2 e + part of the e-th kept output of that parity
// over the first half of the inputs (the class's own sums or differences), the
// classes' row tiles and exponents one after another.  Returns the k-tiles per
// chunk the tables allow.
int build_fwd_split_tables(const HostTables& h, std::vector<uint32_t>& xfrag, std::vector<int>& xex,
                           std::vector<uint32_t>& zfrag, std::vector<int>& zex, std::vector<uint32_t>& ufrag,
                           std::vector<int>& uex, bool& long_rows) {
  const int pz = h.pz, px = h.px, Nz = h.Nz;
  long_rows = false;
  const FwdTcDims d = fwd_tc_dims_n(Nz, h.X, pz, px);
  std::vector<double> Ax, Au, Az, C;
  fwd_tc_matrices(h, Ax, Au, Az);
  xfrag.clear(); xex.clear(); zfrag.clear(); zex.clear(); ufrag.clear(); uex.clear();
  int chunk = kMaxChunkKT;
  // outputs (of M's row pairs of ld words) of one class over its first K words
  auto add = [&](const std::vector<double>& M, int ld, const std::vector<int>& out, int K, int KT, int top,
                 std::vector<uint32_t>& frag, std::vector<int>& ex) {
    const int rows = 2 * (int)out.size();
    C.resize((size_t)rows * K);
    for (int r = 0; r < rows; ++r)
      std::copy_n(&M[(size_t)(2 * out[r / 2] + r % 2) * ld], K, &C[(size_t)r * K]);
    chunk = std::min(chunk, append_digit_table(C.data(), rows, K, (rows + 15) / 16, KT, frag, ex, top, &long_rows));
  };
  for (int c = 0; c < 2; ++c) {
    std::vector<int> kx;
    for (int e = 0; e < (c ? d.nxO : d.nxE); ++e) kx.push_back(2 * e + c);
    add(Ax, px, kx, d.pxh, d.KTxc, 512, xfrag, xex);
    add(Au, px, kx, d.pxh, d.KTxc, 512, ufrag, uex);
  }
  for (int c = 0; c < d.Rz; ++c) {
    std::vector<int> kk;
    z_class_modes(Nz, pz, c, kk);
    if ((int)kk.size() != (c ? d.nzO : d.nzE)) return 0;
    // (an odd length's inputs are no sums: 56 bits)
    add(Az, 2 * pz, kk, 2 * d.pzh, d.KTzc, d.Rz == 2 ? 512 : 256, zfrag, zex);
  }
  return chunk;
}

// ---------------------------------------------------------------------------
// shared-memory plan
// ---------------------------------------------------------------------------

// the digits (z, then x of xch columns)
__host__ __device__ constexpr size_t phys_tc_dbuf(const PhysTcDims& d, int xch) {
  const size_t z = (size_t)kDig * ((d.NZ + 7) / 8 * 8) * d.KSz * 2, x = (size_t)kDig * xch * d.KSx * 2;
  return ((z > x ? z : x) + 15) / 16 * 16;
}
// the exponents of both stages' columns, and the Z intermediate
__host__ __device__ constexpr size_t phys_tc_rest(const PhysTcDims& d, int pz, int X, int fb) {
  return (size_t)((d.NZ + 3) / 4 * 4 + (d.NX + 3) / 4 * 4) * sizeof(int) + (size_t)fb * pz * X * sizeof(cpx);
}
__host__ __device__ constexpr int phys_tc_all_columns(const PhysTcDims& d) { return (d.NX + 7) / 8 * 8; }

size_t phys_tc_smem_bytes(const Grid& g, int fb, int xch) {
  const PhysTcDims d = phys_tc_dims(g, fb);
  return phys_tc_dbuf(d, xch) + phys_tc_rest(d, g.pz, g.X, fb);
}
static size_t phys_tc_smem_bytes(const Grid& g, int fb) {
  return phys_tc_smem_bytes(g, fb, phys_tc_all_columns(phys_tc_dims(g, fb)));
}

// The x stage takes its columns in chunks where all of them at once would
// leave fewer than minb blocks an SM (1 KB reserved and 3 KB declared per
// block): the largest chunk (a multiple of 8) that lets the most blocks, up to
// minb, share one.  48x97x48, one field: all 72 columns 101 KB, 2 blocks; 40
// and 32, 68 KB, 3 (12 instances 1.66 -> 1.23 ms: the kernel waits on latency,
// and 8 warps an SM did not cover it).
static size_t phys_tc_smem_chunked(const Grid& g, int fb, int minb) {
  const int all = phys_tc_all_columns(phys_tc_dims(g, fb));
  for (int nb = minb; nb > 1; --nb)
    for (int c = all; c >= 16; c -= 8)
      if (nb * (phys_tc_smem_bytes(g, fb, c) + 4096) <= 233472) return phys_tc_smem_bytes(g, fb, c);
  return phys_tc_smem_bytes(g, fb);
}
// the chunk that smem bytes of a launch hold for a grid (a launch of several
// grids is sized by the largest), the columns shared evenly
__device__ __forceinline__ int phys_tc_xch(const PhysTcDims& d, int pz, int X, int fb, size_t smem) {
  const int all = phys_tc_all_columns(d);
  const int fit = min(all, (int)((smem - phys_tc_rest(d, pz, X, fb)) / ((size_t)kDig * d.KSx * 2)) / 8 * 8);
  const int n = (all + fit - 1) / fit;
  return ((all + n - 1) / n + 7) / 8 * 8;
}

// ---------------------------------------------------------------------------
// kernel
// ---------------------------------------------------------------------------

// block maximum of the CFL field of plane y (channel/pass1.c:116-138), from
// the written velocity fields
template <int NTHR>
__device__ __forceinline__ void plane_cfl(const Grid& g, const PhysArgs& a, const double* P, int inst, int y, int Q,
                                          int plane) {
  __shared__ double red[NTHR];
  double mx = 0.0;
  const double* Pu = P + (size_t)y * plane;
  const size_t fs = (size_t)Q * plane;
  const double c2 = g.cfl2[y];
  for (int i = threadIdx.x; i < plane; i += NTHR)
    mx = fmax(mx, fabs(Pu[i]) * g.cfl1 + fabs(Pu[fs + i]) * c2 + fabs(Pu[2 * fs + i]) * g.cfl3);
  red[threadIdx.x] = mx;
  __syncthreads();
  constexpr int P2 = NTHR >= 256 ? 256 : (NTHR >= 128 ? 128 : 64);  // largest power of 2 <= NTHR
  if (P2 < NTHR && threadIdx.x < NTHR - P2) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + P2]);
  if (P2 < NTHR) __syncthreads();
  for (int w = P2 / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double c = red[0] * g.dt;
    if (a.cflmax)
      atomicMax(reinterpret_cast<unsigned long long*>(&a.cflmax[inst / a.sdiv]),
                (unsigned long long)__double_as_longlong(c));
    if (c >= 2.8) atomicOr(&a.status[inst / a.sdiv], ST_CFL);
  }
}

// The even modes' rests wait for the odd modes' tile packed in the run-time-size
// builds, whose registers are fewest (48x33x48, 192 threads at 3 blocks:
// 88 bytes spilled instead of 184); the compiled sizes lose by it (192 instances
// of 32x65x32 2.86 -> 2.90 ms)
template <class S>
static constexpr bool kPackRests = std::is_same<S, SizesRT>::value;

// FB fields per pass, NTHR threads, MINB blocks per SM (the register
// budget), S the sizes (SizesRT, or SizesCT for a specialised grid)
template <bool MULTI, int MINB, int FB, int NTHR, class S>
__global__ void __launch_bounds__(NTHR, MINB) k_phys_inverse_tc(const __grid_constant__ Grid g0, PhysArgs a) {
  const int inst = blockIdx.y, y = blockIdx.x;
  CHN_INSTANCE_GRID(g0, a.grids, inst);
  const S gsz(g);
  if (y >= gsz.Q()) return;
  if (a.skip_blocked && blocked(a.status, a.sdiv, inst)) return;
  const PhysTcDims d = phys_tc_dims_n(gsz.Nz(), gsz.pz(), gsz.px(), gsz.X(), FB);
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned char* p = smem;
  int* exz = reinterpret_cast<int*>(p); p += (size_t)((d.NZ + 3) / 4 * 4) * sizeof(int);
  int* exx = reinterpret_cast<int*>(p); p += (size_t)((d.NX + 3) / 4 * 4) * sizeof(int);
  // x-stage columns per chunk: all of them in the fixed-size builds
  int XCH = phys_tc_all_columns(d);
  if constexpr (std::is_same<S, SizesRT>::value) {
    uint32_t dyn;
    asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
    XCH = phys_tc_xch(d, gsz.pz(), gsz.X(), FB, dyn);
  }
  uint16_t* dig = reinterpret_cast<uint16_t*>(p); p += phys_tc_dbuf(d, XCH);
  cpx* Zb = reinterpret_cast<cpx*>(p);  // staged inputs, then [fl][m][x]: the z stage's folded sums
  longlong2* Zs = reinterpret_cast<longlong2*>(Zb);

  const cpx* __restrict__ U = a.U.at(inst);
  double* __restrict__ P = a.P.at(inst);
  if (a.pslot.stride) P += (long long)a.pslot.slot() * a.pslot.stride;
  const size_t plane = (size_t)gsz.pz() * gsz.px();
  const uint4* __restrict__ Az = reinterpret_cast<const uint4*>(g.tcZ);
  const uint4* __restrict__ Ax = reinterpret_cast<const uint4*>(g.tcX);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  constexpr int nwarp = NTHR >> 5;
  const int Kk = gsz.Nz() - 1;  // kept kz rows
  const int chunk = gsz.tcch();
  const auto fold = gsz.fold();
  bool nonfinite = false;
  // this block's fields: all of them, or one of gridDim.z groups
  const int fper = (a.nfields + gridDim.z - 1) / gridDim.z, fbeg = blockIdx.z * fper;
  const int fend = min(a.nfields, fbeg + fper);
  for (int i = threadIdx.x; i < d.NZ; i += NTHR) exz[i] = 0;
  __syncthreads();
  for (int f0 = fbeg; f0 < fend; f0 += FB) {
    const int nfb = min(FB, fend - f0);
    // ---- z stage: columns n = fl * X + x.  The inputs are staged in the Z
    // buffer (free until the z stage writes it: X (Nz - 1) <= pz X values per
    // field); each thread keeps one column (consecutive threads: consecutive
    // x, coalesced loads) and its exponent maximum.  The x stage's column
    // exponents are cleared here and gathered by the z stage's epilogue.
    cpx* Fin = Zb;  // [n][kk]
    for (int i = threadIdx.x; i < d.NX; i += NTHR) exx[i] = 0;
    {
      const int ncol = nfb * gsz.X(), per = NTHR / ncol;
      if ((int)threadIdx.x < per * ncol) {
        const int n = threadIdx.x % ncol, fl = n / gsz.X(), x = n - fl * gsz.X();
        int emax = 0;
        for (int kk = threadIdx.x / ncol; kk < Kk; kk += per) {
          const int z = kk < gsz.Nz() / 2 ? kk : kk + 1;
          const cpx v = field_value_qx(g, gsz.Q(), gsz.X(), U, f0 + fl, z, y, x);
          Fin[(size_t)n * Kk + kk] = v;
          emax = max(emax, max(exp_field(v.re), exp_field(v.im)));
        }
        if (emax) atomicMax(&exz[n], emax);
      }
    }
    __syncthreads();
    {
      // K words (Re, Im of one mode): the even-zp modes, then the odd ones
      const int KW = d.KTz * 8;
      const size_t zstride = (size_t)((d.NZ + 7) / 8 * 8) * d.KSz / 2;  // words between digits
      uint32_t* dw = reinterpret_cast<uint32_t*>(dig);
      FlatRC rc(threadIdx.x, NTHR, KW);
      for (int i = threadIdx.x; i < d.NZ * KW; i += NTHR, rc.next()) {
        const int n = rc.r, w = rc.c;
        const int kk = g.tcZM[w];
        cpx v = {0.0, 0.0};
        if (kk >= 0 && n < nfb * gsz.X()) v = Fin[n * Kk + kk];
        const int ex = exz[n] - 1022;
        digits_pair(scaled56(v.re, ex), scaled56(v.im, ex), dw + ((size_t)n * d.KSz) / 2 + w, zstride);
      }
    }
    __syncthreads();
    {
      // rows Re Z[m], Im Z[m] for m < pzh; E + O -> Z[m], E - O -> Z[m + pzh],
      // kept as 64-bit sums, rounded to their unit (scale 2^zsum_exp(column): the rows of
      // this table share one exponent) that the x stage takes its digits
      // from; the exponent of each value into its x-stage column (fl, m) (not
      // the imaginary part of the kx = 0 bin, which c2r ignores)
      const int NT = (nfb * gsz.X() + 7) / 8;
      const size_t dstride = (size_t)((d.NZ + 7) / 8 * 8) * d.KSz;  // fp16 between digits
      for (int item = warp; item < d.MTz * NT; item += nwarp) {
        const int mt = item / NT, nt = item - mt * NT;
        long long TE[4], TO[4];
        const uint32_t h = fold_half(fold);
        uint32_t RE[4] = {h, h, h, h}, RO[4] = {0, 0, 0, 0};
        tc_tile_range(fold, Az, mt, d.KTz, 0, d.KTzE, chunk, dig, d.KSz, dstride, nt * 8, lane, TE, RE);
        const Rests<kPackRests<S>, Fold> rE(RE);
        tc_tile_range(fold, Az, mt, d.KTz, d.KTzE, d.KTz, chunk, dig, d.KSz, dstride, nt * 8, lane, TO, RO);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int row = mt * 16 + gq + 8 * (r >> 1), col = nt * 8 + 2 * t + (r & 1);
          if (row >= 2 * d.pzh || col >= nfb * gsz.X()) continue;
          const int ce = exz[col];
          const bool im = row >= d.pzh;
          const int m = im ? row - d.pzh : row;
          int fl = 0, x = col;  // col = fl X + x, fl < FB
          while (x >= gsz.X()) { x -= gsz.X(); ++fl; }
          const bool counts = !(im && x == 0);
          long long t;
          uint32_t rest;
          sum_plus(TE[r], rE[r], TO[r], RO[r], t, rest);
          const long long tp = sum_whole(fold, t, rest);
          longlong2& zp = Zs[((size_t)fl * gsz.pz() + m) * gsz.X() + x];
          if (im) zp.y = tp;
          else zp.x = tp;
          const int ep = zsum_field(tp, ce, fold.shift());
          if (counts && ep > 0) atomicMax(&exx[fl * gsz.pz() + m], ep);
          if (d.Rz == 2) {
            sum_minus(fold, TE[r], rE[r], TO[r], RO[r], t, rest);
            const long long tm = sum_whole(fold, t, rest);
            longlong2& zm = Zs[((size_t)fl * gsz.pz() + m + d.pzh) * gsz.X() + x];
            if (im) zm.y = tm;
            else zm.x = tm;
            const int em = zsum_field(tm, ce, fold.shift());
            if (counts && em > 0) atomicMax(&exx[fl * gsz.pz() + m + d.pzh], em);
          }
        }
      }
    }
    __syncthreads();
    // ---- x stage, both fields: columns n = fl * pz + m, K words: Re, Im of
    // Z[m][j] for the even j, then the odd j (Im of j = 0 unused).
    const int ncx = nfb * gsz.pz();
    const size_t xstride = (size_t)XCH * d.KSx;
    for (int n0 = 0; n0 < ncx; n0 += XCH) {
      const int nch = min(XCH, (ncx - n0 + 7) / 8 * 8);
      {
        uint32_t* dw = reinterpret_cast<uint32_t*>(dig);
        const int KW = d.KTx * 8, WE = d.KTxE * 8;
        FlatRC rc(threadIdx.x, NTHR, KW);
        for (int i = threadIdx.x; i < nch * KW; i += NTHR, rc.next()) {
          const int n = n0 + rc.r, w = rc.c;
          const int j = w < WE ? (w < d.nxE ? d.Rx * w : -1) : (w - WE < d.nxO ? 2 * (w - WE) + 1 : -1);
          longlong2 v = make_longlong2(0, 0);
          if (j >= 0 && n < ncx) {
            v = Zs[(size_t)n * gsz.X() + j];
            if (j == 0) v.y = 0;
            int fl = 0, m = n;  // n = fl pz + m
            while (m >= gsz.pz()) { m -= gsz.pz(); ++fl; }
            const int s = exx[n] - 1078 - zsum_exp(exz[fl * gsz.X() + j], fold.shift());
            v.x = scaled_sum(v.x, s);
            v.y = scaled_sum(v.y, s);
          }
          digits_pair(v.x, v.y, dw + ((size_t)rc.r * d.KSx) / 2 + w, xstride / 2);
        }
      }
      __syncthreads();
      // the z stage's column exponents are cleared for the next pass
      if (n0 + XCH >= ncx)
        for (int i = threadIdx.x; i < d.NZ; i += NTHR) exz[i] = 0;
      {
        // rows xp < pxh; E + O -> P[xp], E - O -> P[xp + pxh]
        const int NT = nch / 8;
        for (int item = warp; item < d.MTx * NT; item += nwarp) {
          const int mt = item / NT, nt = item - mt * NT;
          long long TE[4], TO[4];
          uint32_t RE[4] = {0, 0, 0, 0}, RO[4] = {0, 0, 0, 0};
          tc_tile_range(fold, Ax, mt, d.KTx, 0, d.KTxE, chunk, dig, d.KSx, xstride, nt * 8, lane, TE, RE);
          const Rests<kPackRests<S>, Fold> rE(RE);
          tc_tile_range(fold, Ax, mt, d.KTx, d.KTxE, d.KTx, chunk, dig, d.KSx, xstride, nt * 8, lane, TO, RO);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int xp = mt * 16 + gq + 8 * (r >> 1), col = n0 + nt * 8 + 2 * t + (r & 1);
            if (xp >= d.pxh || col >= ncx) continue;
            int fl = 0, m = col;  // col = fl pz + m, fl < FB
            while (m >= gsz.pz()) { m -= gsz.pz(); ++fl; }
            const int e = g.tcXE[xp] + col_exp(exx[col]) - 64 + fold.shift();
            double* Pr = P + ((size_t)(f0 + fl) * gsz.Q() + y) * plane + (size_t)m * gsz.px();
            Pr[xp] = round_plus(fold, TE[r], rE[r], TO[r], RO[r], e, nonfinite);
            if (d.Rx == 2) Pr[xp + d.pxh] = round_minus(fold, TE[r], rE[r], TO[r], RO[r], e, nonfinite);
          }
        }
      }
      __syncthreads();
    }
  }
  if (nonfinite && a.status) atomicOr(&a.status[inst / a.sdiv], ST_NONFINITE);
  // (with the fields in groups, k_cfl follows)
  if (a.cfl_check && gridDim.z == 1) plane_cfl<NTHR>(g, a, P, inst, y, gsz.Q(), gsz.pz() * gsz.px());
}

// The CFL check of a launch whose fields ran in blocks of their own (or in
// split passes), one block per plane
__global__ void __launch_bounds__(kThreads) k_cfl(const __grid_constant__ Grid g, PhysArgs a) {
  const int inst = blockIdx.y, y = blockIdx.x;
  if (a.skip_blocked && blocked(a.status, a.sdiv, inst)) return;
  double* __restrict__ P = a.P.at(inst);
  if (a.pslot.stride) P += (long long)a.pslot.slot() * a.pslot.stride;
  plane_cfl<kThreads>(g, a, P, inst, y, g.Q, g.pz * g.px);
}

// ---------------------------------------------------------------------------
// products + forward transforms
// ---------------------------------------------------------------------------

static constexpr int kPB = 3;  // products computed per pass over the plane
// threads of the one-plane build with run-time sizes for batches of one grid,
// whose blocks are large and two to an SM: 24 warps instead of 16 cover more of
// the latency that binds it (12 instances at 48x97x48 forward 0.947 -> 0.893 ms,
// 4 adjoint 0.618 -> 0.592).  The other builds keep 256: one component a block
// is slower with 384 (8 of 16x33x16 30 -> 34 us), several grids no faster (the
// register limit spills more there).
static constexpr int kWideThreads = 384;

// shared memory of a products block: pb product planes, x-stage digits of
// xch columns (a chunk), z-stage digits, exponents (px is even: a plane is
// whole 16-byte words)
__host__ __device__ constexpr size_t fwd_tc_smem_n(int Nz, int X, int pz, int px, int pb, int xch) {
  const FwdTcDims d = fwd_tc_dims_n(Nz, X, pz, px);
  const size_t dx = (size_t)kDig * xch * d.KSx * 2, dz = (size_t)kDig * d.Xp * d.KSz * 2;
  return (size_t)(pb * ((pz + 3) / 4 * 4) + (X + 3) / 4 * 4) * sizeof(int) + ((dx > dz ? dx : dz) + 15) / 16 * 16 +
         (size_t)pb * pz * px * sizeof(double);
}

// the widest x-stage chunk (a multiple of 8 columns) with which minb blocks
// of pb planes share an SM's 228 KB (1 KB reserved per block); 8 if none
__host__ __device__ constexpr int fwd_tc_xch_n(int Nz, int X, int pz, int px, int pb, int minb) {
  const int pzp = (pz + 7) / 8 * 8;
  for (int c = pzp; c > 8; c -= 8)
    if ((size_t)minb * (fwd_tc_smem_n(Nz, X, pz, px, pb, c) + 1024 + 1024) <= 233472) return c;
  return 8;
}

// pb product planes per pass: kPB for the forward modes (0, 1); for the
// adjoint modes (2, 3, six products) Grid::adjpb: kPB (each field loaded
// once per three products) or one (a smaller footprint leaves L1 to the
// tables), as the autotuner finds faster
inline int products_per_pass(const Grid& g, int mode) {
  if (mode < 2) return g.fwdpb;
  return g.adjpb == kPB && g.fwdpb == kPB ? kPB : 1;
}

// xch: x-stage columns (padded zp rows) digitised per chunk
size_t fwd_tc_smem_bytes(const Grid& g, int pb, int xch) { return fwd_tc_smem_n(g.Nz, g.X, g.pz, g.px, pb, xch); }

// The products of one plane (mode 0 primal, 1 tangent, 2 adjoint S and T,
// 3 the exact transpose; split_product) and their forward transforms as
// digit GEMMs: the products of three components in one pass over the plane
// (each field loaded once), then the transforms one component at a time;
// modes 0/1 write H slots 0..2, modes 2/3 fold each component into the
// output slots (assemble_stage).  Same outputs as k_products_fwd /
// k_products_adj.
// S: the sizes (SizesRT, or SizesCT for a specialised grid); NTHR threads, MINB
// blocks per SM (the register budget; with MINB > 2 the x stage runs in the chunks
// that let MINB blocks share an SM)
template <bool MULTI, int PB, class S, int MINB = 2, int NTHR = kThreads>
__global__ void __launch_bounds__(NTHR, MINB) k_products_tc(const __grid_constant__ Grid g0, ProdArgs a, int mode) {
  const int inst = blockIdx.y, y = blockIdx.x;
  CHN_INSTANCE_GRID(g0, a.grids, inst);
  const S gsz(g);
  if (y >= gsz.Q()) return;
  if (blocked(a.status, a.sdiv, inst)) return;
  const FwdTcDims d = fwd_tc_dims_n(gsz.Nz(), gsz.X(), gsz.pz(), gsz.px());
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned char* p = smem;
  const int exs = (gsz.pz() + 3) / 4 * 4, pb = PB;
  int* exx3 = reinterpret_cast<int*>(p); p += (size_t)pb * exs * sizeof(int);  // [c][zp]
  int* exz = reinterpret_cast<int*>(p); p += (size_t)((gsz.X() + 3) / 4 * 4) * sizeof(int);
  uint16_t* dig = reinterpret_cast<uint16_t*>(p);
  // x-stage columns per chunk: all of them in the fixed-size builds, else
  // the plan's (Grid::fxch, a multiple of 8)
  int XCH = d.pzp;
  if constexpr (MINB > 2) XCH = fwd_tc_xch_n(gsz.Nz(), gsz.X(), gsz.pz(), gsz.px(), PB, MINB);
  else if constexpr (kRunTimeSizes<S>) XCH = min(g.fxch, d.pzp);
  {
    const size_t dx = (size_t)kDig * XCH * d.KSx * 2, dz = (size_t)kDig * d.Xp * d.KSz * 2;
    p += ((dx > dz ? dx : dz) + 15) / 16 * 16;
  }
  // [c][zp][xp] products; over plane c Y [zp][kx] (folded sums), then the z
  // stage's outputs Fb [kk][kx] (less than half a plane)
  double* stage3 = reinterpret_cast<double*>(p);
  const size_t plane = (size_t)gsz.pz() * gsz.px(), fs = (size_t)gsz.Q() * plane;
  const double* __restrict__ Pp = a.Pp.base + (long long)(inst / a.pdiv) * a.Pp.stride + (size_t)y * plane +
                                  (a.pslot.stride ? (long long)a.pslot.slot() * a.pslot.stride : 0LL);
  const double* __restrict__ Pt = a.Pt.base ? a.Pt.at(inst) + (size_t)y * plane : nullptr;
  cpx* __restrict__ H = a.H.at(inst);
  // the exact transpose's forward transforms carry no 1/(px pz)
  const uint4* __restrict__ Ax = reinterpret_cast<const uint4*>(mode == 3 ? g.tcFXU : g.tcFX);
  const int* __restrict__ AxE = mode == 3 ? g.tcFXUE : g.tcFXE;
  const uint4* __restrict__ Az = reinterpret_cast<const uint4*>(g.tcFZ);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  constexpr int nwarp = NTHR >> 5;
  const auto fold = gsz.fold();
  // this block's components: all of them, or one of gridDim.z groups
  const int nall = mode >= 2 ? 6 : 3, qper = (nall + gridDim.z - 1) / gridDim.z, qbeg = blockIdx.z * qper;
  const int ncomp = min(nall, qbeg + qper);
  const size_t xstride = (size_t)XCH * d.KSx, zstride = (size_t)d.Xp * d.KSz;  // 16-bit words between digits
  for (int q = qbeg; q < ncomp; ++q) {
    const int c = (q - qbeg) % pb;
    double* stage = stage3 + (size_t)c * plane;
    longlong2* Yb = reinterpret_cast<longlong2*>(stage);  // Re, Im of Y[zp][kx]: t 2^(AxE[2 kx (+ 1)] + ysum_exp(exx[zp]))
    cpx* Fb = reinterpret_cast<cpx*>(stage);
    int* exx = exx3 + c * exs;
    if (c == 0) {
      // ---- products of components q .. q+2 (each field loaded once per
      // point), row exponents (one column per zp)
      for (int i = threadIdx.x; i < pb * exs; i += NTHR) exx3[i] = 0;
      __syncthreads();
      const int nc = min(pb, ncomp - q);
      FlatRC rc(threadIdx.x, NTHR, gsz.px());
      auto point = [&](int i) {
        double v[PB];
#pragma unroll
        for (int cc = 0; cc < PB; ++cc) v[cc] = cc < nc ? split_product(mode, Pp, Pt, fs, i, q + cc) : 0.0;
        const int row = rc.r;
#pragma unroll
        for (int cc = 0; cc < PB; ++cc) {
          if (cc >= nc) break;
          stage3[(size_t)cc * plane + i] = v[cc];
          const int e = exp_field(v[cc]);
          if (e) atomicMax(&exx3[cc * exs + row], e);
        }
      };
      if constexpr (kRunTimeSizes<S>) {
        for (int i = threadIdx.x; i < gsz.pz() * gsz.px(); i += NTHR, rc.next()) point(i);
      } else {
#pragma unroll 3
        for (int i = threadIdx.x; i < gsz.pz() * gsz.px(); i += NTHR, rc.next()) point(i);
      }
      __syncthreads();
    }
    // ---- x stage: columns zp, in chunks of XCH columns; Y
    // into the staging region (Y row zp lies below stage row zp, 16 X < 8 px
    // bytes per row, so a chunk's outputs only cover rows already digitised)
    // (the z stage's column exponents are cleared for this component first)
    for (int i = threadIdx.x; i < gsz.X(); i += NTHR) exz[i] = 0;
    for (int zc = 0; zc < d.pzp; zc += XCH) {
      const int nch = min(XCH, d.pzp - zc);
      FlatRC rcx(threadIdx.x, NTHR, d.KTxc * 8);
      for (int i = threadIdx.x; i < nch * (d.KTxc * 8); i += NTHR, rcx.next()) {
        const int n = zc + rcx.r;
        fwd_x_digits(d, stage + (size_t)n * gsz.px(), 2 * rcx.c, n < gsz.pz(), exx[min(n, gsz.pz() - 1)] - 1022,
                     reinterpret_cast<uint32_t*>(dig + (size_t)rcx.r * d.KSx), xstride / 2);
      }
      __syncthreads();
      const int NT = nch / 8;
      for (int item = warp; item < d.MTx * NT; item += nwarp) {
        const int mt = item / NT, nt = item - mt * NT;
        long long T[4];
        const uint32_t h = fold_half(fold);
        uint32_t R[4] = {h, h, h, h};  // (kept as T alone)
        tc_tile(fold, Ax, mt, d.KTxc, kChunkKT, dig + (mt >= d.MTxE ? d.KTxc * 16 : 0), d.KSx, xstride, nt * 8, lane, T,
                R);
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
          FwdRow row;
          if (!fwd_row(mt, gq + 8 * rr, d.MTxE, d.nxE, d.nxO, row)) continue;
          const int kx = 2 * row.e + row.cls, er = AxE[2 * (row.cls * d.nxE + row.e) + row.part];
          int ef = 0;  // the exponent field of this row's values, for the z stage's column
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int zp = zc + nt * 8 + 2 * t + c;
            if (zp >= gsz.pz()) continue;
            const long long tv = T[2 * rr + c];
            longlong2& yv = Yb[(size_t)zp * gsz.X() + kx];
            if (row.part) yv.y = tv;
            else yv.x = tv;
            ef = max(ef, sum_field(tv, er + ysum_exp(exx[zp], fold.shift()), exx[zp]));
          }
          if (ef > 0) atomicMax(&exz[kx], ef);
        }
      }
      __syncthreads();
    }
    // ---- z stage inputs: columns kx (Re, Im of Y[zp][kx] interleaved)
    {
      uint32_t* dw = reinterpret_cast<uint32_t*>(dig);
      FlatRC rc(threadIdx.x, NTHR, d.KTzc * 8);
      for (int i = threadIdx.x; i < d.Xp * (d.KTzc * 8); i += NTHR, rc.next()) {
        const int n = rc.r, zp = rc.c;
        longlong2 u = make_longlong2(0, 0), v = u;
        if (n < gsz.X() && zp < d.pzh) {
          const int2 er = *reinterpret_cast<const int2*>(AxE + 2 * ((n & 1) * d.nxE + (n >> 1)));
          auto input = [&](int z) {
            longlong2 w = Yb[(size_t)z * gsz.X() + n];
            const int s = exz[n] - 1078 - ysum_exp(exx[z], fold.shift());
            w.x = scaled_sum(w.x, s - er.x);
            w.y = scaled_sum(w.y, s - er.y);
            return w;
          };
          u = input(zp);
          if (d.Rz == 2) v = input(zp + d.pzh);
        }
        fwd_z_digits(d, zp, u, v, dw + ((size_t)n * d.KSz) / 2, zstride / 2);
      }
    }
    __syncthreads();
    // ---- z stage: columns kx -> Fb
    {
      const int NT = d.Xp / 8;
      for (int item = warp; item < d.MTz * NT; item += nwarp) {
        const int mt = item / NT, nt = item - mt * NT;
        long long T[4];
        uint32_t R[4] = {0, 0, 0, 0};
        tc_tile(fold, Az, mt, d.KTzc, kChunkKT, dig + (mt >= d.MTzE ? d.KTzc * 16 : 0), d.KSz, zstride, nt * 8, lane, T,
                R);
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
          FwdRow row;
          if (!fwd_row(mt, gq + 8 * rr, d.MTzE, d.nzE, d.nzO, row)) continue;
          const int er = g.tcFZE[2 * (row.cls * d.nzE + row.e) + row.part] - 64 + fold.shift();
          const int kk = fwd_z_mode(gsz.Nz(), d.Rz, row.cls, row.e);
#pragma unroll
          for (int c2 = 0; c2 < 2; ++c2) {
            const int kx = nt * 8 + 2 * t + c2;
            if (kx >= gsz.X()) continue;
            reinterpret_cast<double*>(Fb + (size_t)kk * gsz.X() + kx)[row.part] =
                round_sum(fold, T[2 * rr + c2], R[2 * rr + c2], er + col_exp(exz[kx]));
          }
        }
      }
    }
    __syncthreads();
    // ---- outputs (the (kk, kx) -> thread map is the same for every q)
    FlatRC rco(threadIdx.x, NTHR, gsz.X());
    for (int i = threadIdx.x; i < d.Kk * gsz.X(); i += NTHR, rco.next()) {
      const int kk = rco.r, x = rco.c;
      const int z = kk < gsz.Nz() / 2 ? kk : kk + 1;
      if (mode < 2) H[(((size_t)z * 5 + q) * gsz.Q() + y) * gsz.X() + x] = Fb[i];
      else if (gridDim.z > 1) a.tmp[((((size_t)inst * 6 + q) * gsz.Q() + y) * gsz.pz() + kk) * gsz.X() + x] = Fb[i];
      else assemble_stage(g, mode == 3, H, z, y, x, q, Fb[i]);
    }
    __syncthreads();
  }
}

// the adjoint modes' output slots from the six components' spectra in the
// scratch array [local instance][6][Q][pz][X] (kept rows first): launches that
// ran the components in blocks of their own, and the split passes
__global__ void __launch_bounds__(kThreads) k_assemble(const __grid_constant__ Grid g, ProdArgs a, int exact, int inst0) {
  const int il = blockIdx.y, inst = inst0 + il, kk = blockIdx.z, z = kk < g.Nz / 2 ? kk : kk + 1;
  if (blocked(a.status, a.sdiv, inst)) return;
  cpx* __restrict__ H = a.H.at(inst);
  const int i = blockIdx.x * kThreads + threadIdx.x;
  if (i >= g.Q * g.X) return;
  const int y = i / g.X, x = i - y * g.X;
  cpx v[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) v[q] = a.tmp[((((size_t)il * 6 + q) * g.Q + y) * g.pz + kk) * g.X + x];
#pragma unroll
  for (int q = 0; q < 6; ++q) assemble_stage(g, exact != 0, H, z, y, x, q, v[q]);
}

void launch_assemble(const Grid& g, const ProdArgs& a, bool exact, int inst0, int n, cudaStream_t st) {
  k_assemble<<<dim3((g.Q * g.X + kThreads - 1) / kThreads, n, g.Nz - 1), kThreads, 0, st>>>(g, a, exact, inst0);
}

void launch_cfl(const Grid& g, const PhysArgs& a, cudaStream_t st) {
  k_cfl<<<dim3(g.Q, a.ninst), kThreads, 0, st>>>(g, a);
}

// The forward products' shared-memory plan: product planes per pass of the
// forward modes (kPB, else one) and x-stage columns per chunk (the widest
// multiple of 8), the first that lets two blocks share an SM; false if none
// does (the FFT kernels then run).  48x97x48: one plane per pass, chunks of
// 48 columns, 112 KB per block.
bool fwd_tc_plan(const Grid& g, int optin, int& pb, int& xch) {
  const FwdTcDims d = fwd_tc_dims(g);
  const int pbs[2] = {kPB, 1};
  for (int p : pbs)
    for (int c = d.pzp; c >= 8; c -= 8)
      if (2 * (fwd_tc_smem_bytes(g, p, c) + 4096) <= (size_t)optin + 4096) {
        pb = p;
        xch = c;
        return true;
      }
  return false;
}

bool fwd_tc_fits(const Grid& g, int optin) {
  int pb = 0, xch = 0;
  return fwd_tc_plan(g, optin, pb, xch);
}

bool phys_tc_covers(const Grid& gmax, const Grid& g) {
  if (gmax.tci)
    for (int fb = 1; fb <= kFB; ++fb)
      for (int minb = 2; minb <= 5; ++minb)
        if (phys_tc_smem_bytes(g, fb, 8) > phys_tc_smem_chunked(gmax, fb, minb)) return false;
  if (gmax.tcf)
    for (int pb : {1, gmax.fwdpb}) {
      auto bytes = [&](const Grid& a) { return fwd_tc_smem_bytes(a, pb, std::min(gmax.fxch, fwd_tc_dims(a).pzp)); };
      if (bytes(g) > bytes(gmax)) return false;
    }
  return true;
}

template <class S>
static void launch_products_sizes(const Grid& g, const ProdArgs& a, int mode, cudaStream_t st) {
  const FwdTcDims d = fwd_tc_dims(g);
  const int xch = kRunTimeSizes<S> ? (g.fxch < d.pzp ? g.fxch : d.pzp) : d.pzp;
  const size_t sm = fwd_tc_smem_bytes(g, products_per_pass(g, mode), xch);
  const dim3 grid(g.Q, a.ninst);
  constexpr bool M = kRunTimeSizes<S>;  // only the run-time sizes serve uneven batches
  using RunTime = std::conditional_t<M, S, SizesRT>;
  if (products_per_pass(g, mode) == kPB) {
    if (M && a.grids) k_products_tc<true, kPB, RunTime><<<grid, kThreads, sm, st>>>(g, a, mode);
    else k_products_tc<false, kPB, S><<<grid, kThreads, sm, st>>>(g, a, mode);
  } else {
    if (M && a.grids) k_products_tc<true, 1, RunTime><<<grid, kThreads, sm, st>>>(g, a, mode);
    else k_products_tc<false, 1, S, 2, M ? kWideThreads : kThreads><<<grid, M ? kWideThreads : kThreads, sm, st>>>(g, a, mode);
  }
}

// Grid::prodb's bit (single-grid batches): two product planes per pass at 3
// blocks per SM (80 registers), the x stage in the chunks that fit
template <class S>
static void launch_products_b3(const Grid& g, const ProdArgs& a, int mode, cudaStream_t st) {
  const dim3 grid(g.Q, a.ninst);
  const size_t sm = fwd_tc_smem_bytes(g, 2, fwd_tc_xch_n(g.Nz, g.X, g.pz, g.px, 2, 3));
  k_products_tc<false, 2, S, 3><<<grid, kThreads, sm, st>>>(g, a, mode);
}

// The products' launches of few planes likewise: one component per block, the
// adjoint modes through the scratch array and k_assemble (unless a switch asked
// for a build of the others).  Forward modes up to
// 3 planes per SM (one instance at 32x65x32 40 -> 25 us), adjoint modes up to 2
// (76 -> 41); alone they gain up to 4 and 3 (8 of 16x33x16 39 -> 31, 64 -> 53),
// but not beside the tangents' launches (the limits below: inverse_groups).
int products_groups(const Grid& g, const ProdArgs& a, int mode) {
  const long long planes = (long long)g.Q * a.ninst;
  if (a.grids || (g.pfixed & (mode < 2 ? 1 : 2))) return 1;
  if (mode < 2) return planes <= 3 * 152 ? 3 : 1;
  return planes <= 2 * 152 && a.tmp && a.ninst <= a.tmp_inst ? 6 : 1;
}

// Grid::fixed & FIXED_PRODUCTS: the build compiled for the grid's sizes
// (32x65x32, 16x33x16; single-grid batches), else the run-time sizes
cudaError_t launch_products_tc(const Grid& g, const ProdArgs& a, int mode, cudaStream_t st) {
  const int groups = products_groups(g, a, mode);
  if (groups > 1) {
    const FwdTcDims d = fwd_tc_dims(g);
    const dim3 grid(g.Q, a.ninst, groups);
    const int xch = g.fxch < d.pzp ? g.fxch : d.pzp;
    const size_t sm = fwd_tc_smem_bytes(g, 1, xch);
    const bool fx = (g.fixed & FIXED_PRODUCTS) && xch == d.pzp;
    if (fx && sizes_match<Sizes32>(g)) k_products_tc<false, 1, Sizes32><<<grid, kThreads, sm, st>>>(g, a, mode);
    else if (fx && sizes_match<Sizes16>(g)) k_products_tc<false, 1, Sizes16><<<grid, kThreads, sm, st>>>(g, a, mode);
    else if (g.tcfl) k_products_tc<false, 1, SizesLong><<<grid, kThreads, sm, st>>>(g, a, mode);
    else k_products_tc<false, 1, SizesRT><<<grid, kThreads, sm, st>>>(g, a, mode);
    if (mode >= 2) launch_assemble(g, a, mode == 3, 0, a.ninst, st);
    return cudaGetLastError();
  }
  if ((g.prodb & (mode < 2 ? 1 : 2)) && !a.grids) {
    const bool fx = (g.fixed & FIXED_PRODUCTS) != 0;
    if (fx && sizes_match<Sizes32>(g)) launch_products_b3<Sizes32>(g, a, mode, st);
    else if (fx && sizes_match<Sizes16>(g)) launch_products_b3<Sizes16>(g, a, mode, st);
    else if (g.tcfl) launch_products_b3<SizesLong>(g, a, mode, st);
    else launch_products_b3<SizesRT>(g, a, mode, st);
    return cudaGetLastError();
  }
  const bool fx = (g.fixed & FIXED_PRODUCTS) && !a.grids && g.fxch >= fwd_tc_dims(g).pzp;
  if (fx && sizes_match<Sizes32>(g)) launch_products_sizes<Sizes32>(g, a, mode, st);
  else if (fx && sizes_match<Sizes16>(g)) launch_products_sizes<Sizes16>(g, a, mode, st);
  else if (g.tcfl) launch_products_sizes<SizesLong>(g, a, mode, st);
  else launch_products_sizes<SizesRT>(g, a, mode, st);
  return cudaGetLastError();
}

bool phys_tc_fits(const Grid& g, int optin) {
  // the kernel's static shared memory (reduction, staged grid) is below 4 KB;
  // the input staging keeps one thread per z-stage column (the widest build's
  // plan; the one-field builds need less)
  return kFB * g.X <= kThreads && phys_tc_smem_bytes(g, kFB) + 4096 <= (size_t)optin;
}

// Launches of few planes run a plane's fields in blocks of their own, FB
// fields each, instead of one after another: up to kGroupPlanes planes (3 per
// SM).  One instance at 32x65x32: 49 -> 23 us in one-field blocks.  Launches of
// more planes share the chip with another stream's: with limits of 5, 4 and 3
// per SM (inverse, forward, adjoint products) eight segments' adjoint chain at
// 16x33x16 takes 5.01 ms, with 3, 3, 2 4.72, with 2, 2, 1 4.83; five of
// 28x43x18 8.83, 8.63, 8.97.
static constexpr long long kGroupPlanes = 3 * 152;
static int inverse_groups(const Grid& g, const PhysArgs& a, int fb) {
  return !a.grids && (long long)g.Q * a.ninst <= kGroupPlanes ? (a.nfields + fb - 1) / fb : 1;
}

// Builds of the kernel (Grid::tcminb; the autotuner times them, the results
// are identical): fields per pass, threads, blocks per SM (the register
// budget) and the sizes, run-time (RT) or compiled for the grid (CT):
//   2: 2 fields, 256 threads, 2 blocks, RT   3: the same at 3 blocks
//   4: 1 field, 128 threads, 4 blocks, RT    5: the same at 5 blocks
//   6: build 4, CT                           7: build 2, CT
//   8: 1 field, 192 threads, 3 blocks, RT    9: build 8, CT
//  10: 1 field, 128 threads, 5 blocks, CT   11: 192 threads, 4 blocks, CT
//  12: 1 field, 256 threads, 3 blocks, CT
// One field per pass halves the shared memory; 192 threads give the z
// stage's six output tiles of a field one warp each; the compiled sizes
// need fewer registers (96 at 5 blocks of 128 threads without spills).
template <bool MULTI>
static void launch_inverse_build(const Grid& g, const PhysArgs& a, cudaStream_t st) {
  const int fb = (g.tcminb == 4 || g.tcminb == 5 || g.tcminb == 8) ? 1 : 2;
  const dim3 grid(g.Q, a.ninst, inverse_groups(g, a, fb));
  auto s = [&](int fb, int minb) { return phys_tc_smem_chunked(g, fb, minb); };
  using RT = SizesRT;
  switch (g.tcminb) {
    case 3: k_phys_inverse_tc<MULTI, 3, 2, 256, RT><<<grid, 256, s(2, 3), st>>>(g, a); break;
    case 4: k_phys_inverse_tc<MULTI, 4, 1, 128, RT><<<grid, 128, s(1, 4), st>>>(g, a); break;
    case 5: k_phys_inverse_tc<MULTI, 5, 1, 128, RT><<<grid, 128, s(1, 5), st>>>(g, a); break;
    case 8: k_phys_inverse_tc<MULTI, 3, 1, 192, RT><<<grid, 192, s(1, 3), st>>>(g, a); break;
    default: k_phys_inverse_tc<MULTI, 2, 2, 256, RT><<<grid, 256, s(2, 2), st>>>(g, a); break;
  }
}

bool phys_tc_specialised(const Grid& g) { return sizes_match<Sizes32>(g) || sizes_match<Sizes16>(g); }

// the run-time-size build a compile-time one stands for
static int inverse_rt_build(int b) {
  switch (b) {
    case 6: return 4;
    case 7: return 2;
    case 9: case 11: case 12: return 8;
    case 10: return 5;
    default: return b;
  }
}
static bool inverse_ct_build(int b) { return b == 6 || b == 7 || b >= 9; }

template <class S>
static void launch_inverse_ct(const Grid& g, const PhysArgs& a, cudaStream_t st) {
  const dim3 grid(g.Q, a.ninst, inverse_groups(g, a, g.tcminb == 7 ? 2 : 1));
  const size_t s1 = phys_tc_smem_bytes(g, 1);
  switch (g.tcminb) {
    case 6: k_phys_inverse_tc<false, 4, 1, 128, S><<<grid, 128, s1, st>>>(g, a); break;
    case 9: k_phys_inverse_tc<false, 3, 1, 192, S><<<grid, 192, s1, st>>>(g, a); break;
    case 10: k_phys_inverse_tc<false, 5, 1, 128, S><<<grid, 128, s1, st>>>(g, a); break;
    case 11: k_phys_inverse_tc<false, 4, 1, 192, S><<<grid, 192, s1, st>>>(g, a); break;
    case 12: k_phys_inverse_tc<false, 3, 1, 256, S><<<grid, 256, s1, st>>>(g, a); break;
    default: k_phys_inverse_tc<false, 2, 2, 256, S><<<grid, 256, phys_tc_smem_bytes(g, 2), st>>>(g, a); break;
  }
}

cudaError_t launch_phys_inverse_tc(const Grid& g, const PhysArgs& a, cudaStream_t st) {
  const bool ct = inverse_ct_build(g.tcminb) && !a.grids;
  if (ct && sizes_match<Sizes32>(g)) {
    launch_inverse_ct<Sizes32>(g, a, st);
  } else if (ct && sizes_match<Sizes16>(g)) {
    launch_inverse_ct<Sizes16>(g, a, st);
  } else {
    Grid gr = g;
    gr.tcminb = inverse_rt_build(g.tcminb);
    if (a.grids) launch_inverse_build<true>(gr, a, st);
    else launch_inverse_build<false>(gr, a, st);
  }
  if (a.cfl_check && inverse_groups(g, a, 1) > 1) launch_cfl(g, a, st);
  return cudaGetLastError();
}

void prepare_phys_tc(int optin) {
  using RT = SizesRT;
  allow_max_smem(k_phys_inverse_tc<false, 2, 2, 256, RT>, optin);
  allow_max_smem(k_phys_inverse_tc<true, 2, 2, 256, RT>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 3, 2, 256, RT>, optin);
  allow_max_smem(k_phys_inverse_tc<true, 3, 2, 256, RT>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 4, 1, 128, RT>, optin);
  allow_max_smem(k_phys_inverse_tc<true, 4, 1, 128, RT>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 5, 1, 128, RT>, optin);
  allow_max_smem(k_phys_inverse_tc<true, 5, 1, 128, RT>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 4, 1, 128, Sizes32>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 2, 2, 256, Sizes32>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 4, 1, 128, Sizes16>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 3, 1, 192, RT>, optin);
  allow_max_smem(k_phys_inverse_tc<true, 3, 1, 192, RT>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 3, 1, 192, Sizes32>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 3, 1, 192, Sizes16>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 5, 1, 128, Sizes32>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 4, 1, 192, Sizes32>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 3, 1, 256, Sizes32>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 5, 1, 128, Sizes16>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 4, 1, 192, Sizes16>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 3, 1, 256, Sizes16>, optin);
  allow_max_smem(k_phys_inverse_tc<false, 2, 2, 256, Sizes16>, optin);
  allow_max_smem(k_products_tc<false, kPB, RT>, optin);
  allow_max_smem(k_products_tc<true, kPB, RT>, optin);
  allow_max_smem(k_products_tc<false, 1, RT>, optin);
  allow_max_smem(k_products_tc<false, 1, RT, 2, kWideThreads>, optin);
  allow_max_smem(k_products_tc<true, 1, RT>, optin);
  allow_max_smem(k_products_tc<false, kPB, SizesLong>, optin);
  allow_max_smem(k_products_tc<true, kPB, SizesLong>, optin);
  allow_max_smem(k_products_tc<false, 1, SizesLong>, optin);
  allow_max_smem(k_products_tc<false, 1, SizesLong, 2, kWideThreads>, optin);
  allow_max_smem(k_products_tc<true, 1, SizesLong>, optin);
  allow_max_smem(k_products_tc<false, 2, SizesLong, 3>, optin);
  allow_max_smem(k_products_tc<false, kPB, Sizes32>, optin);
  allow_max_smem(k_products_tc<false, 2, SizesRT, 3>, optin);
  allow_max_smem(k_products_tc<false, 2, Sizes32, 3>, optin);
  allow_max_smem(k_products_tc<false, 2, Sizes16, 3>, optin);
  allow_max_smem(k_products_tc<false, 1, Sizes32>, optin);
  allow_max_smem(k_products_tc<false, kPB, Sizes16>, optin);
  allow_max_smem(k_products_tc<false, 1, Sizes16>, optin);
}

}  // namespace chn
