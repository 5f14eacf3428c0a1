// Coefficients -> velocity (channel/initAlphaBeta2.c:12-240) on the tensor
// cores, exact to the FP64 rounding of its result.
//
// The reconstruction is five real contractions per (kz, kx) column,
//   v = Q alpha, Q' alpha, Q'' alpha, g = R beta, R' beta   (Q planes each),
// followed by the K-algebra that mixes them into u, w, du/dy, dw/dy.  On
// GB300 the FP64 pipe (1.2 TFLOP/s) bounds the direct form; here each
// contraction runs as an fp16 tensor-core GEMM on integer digits:
//   - every basis row (plane y) and every coefficient column is scaled by a
//     power of two into an integer of 56 significant bits, written as seven
//     balanced base-256 digits (the top digit in [-256, 256], the others in
//     [-128, 127]); digits are exact in fp16;
//   - digit products of level l = i + k accumulate in FP32 through
//     mma.sync m16n8k16 (fp16 inputs, FP32 accumulator), exactly, in chunks
//     of two k-tiles (append_digit_table checks each table);
//   - levels l < 7 are kept (the rest lie below 2^-56 of the operands'
//     scale), folded exactly (digit_sum.cuh) and rounded once to FP64.
// Only the rounding and the K-algebra use the FP64 pipe.  Results agree with the FP64
// contraction to its own rounding.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "chn_common.cuh"
#include "kernels.h"
#include "setup.h"
#include "tc_common.cuh"
#include "sizes.cuh"

namespace chn {

static constexpr int kThreads = 256;
static constexpr int kTile = 16;   // kx columns per block (32 real columns: re, im interleaved)
static constexpr int kReconRegs = 8;  // coefficient rows a thread keeps in registers per class (R <= 128)

// ---------------------------------------------------------------------------
// host: basis digit tables in mma A-fragment order
// ---------------------------------------------------------------------------

// the exponent of a row of K entries: |row| < 2^e, and the sum of the row's
// 56-bit integers at most kLongRowSum * 2^56, so that a folded sum over the whole
// row fits 64 bits (only rows of more than 506 entries can need the second);
// top: the largest top digit of the data, 256, or 512 for the sums and
// differences of two 56-bit integers (half the row's sum then)
int digit_row_exponent(const double* row, int K, int top) {
  double mx = 0.0, sum = 0.0;
  for (int j = 0; j < K; ++j) {
    mx = std::fmax(mx, std::fabs(row[j]));
    sum += std::fabs(row[j]);
  }
  int e = 0;
  std::frexp(mx, &e);
  while (std::ldexp(sum, -e) >= kLongRowSum * 256 / top) ++e;
  return e;
}

int append_digit_table(const double* M, int rows, int K, int MT, int KT, std::vector<uint32_t>& frag,
                        std::vector<int>& ex, int top, bool* long_rows) {
  const size_t base = frag.size();
  frag.resize(base + (size_t)MT * KT * kDig * 32 * 4, 0u);
  const size_t ebase = ex.size();
  ex.resize(ebase + rows, -1022);
  std::vector<int> dig((size_t)rows * (KT * 16) * kDig, 0);
  int chunk = kMaxChunkKT;
  for (int y = 0; y < rows; ++y) {
    double mx = 0.0;
    for (int j = 0; j < K; ++j) mx = std::fmax(mx, std::fabs(M[(size_t)y * K + j]));
    if (mx == 0.0) continue;
    int e = digit_row_exponent(&M[(size_t)y * K], K, top);  // |M[y][j]| < 2^e
    double sum = 0.0;
    for (int j = 0; j < K; ++j) sum += std::fabs(M[(size_t)y * K + j]);
    auto is_long = [&] { return std::ldexp(sum, -e) >= kRowSum * 256 / top; };
    // The largest level sum any data digits (|d_0| <= top, the others <= 128)
    // can reach over `chunk` consecutive k-tiles sets the chunk.  Equal entries
    // (the kx = 0 row) have equal digits, which can all be large: a long row
    // that would not allow kChunkKT gives up a bit and takes other digits (Nx = 100,
    // Nz = 20, which ran the FFTs otherwise, at half the speed).
    auto row_chunk = [&](int chunk) {
      for (int j = 0; j < K; ++j) {
        const long long x = std::llround(std::ldexp(M[(size_t)y * K + j], 56 - e));
        digits56(x, &dig[((size_t)y * (KT * 16) + j) * kDig]);
      }
      for (int kt = 0; kt < KT && chunk > 0; ++kt) {
        const int k1 = std::min(std::min(kt + chunk, KT) * 16, K);
        long long used = 0;  // sum |digit i| of the window, i ascending
        for (int l = 0; l < kDig; ++l) {
          long long last = 0;
          for (int j = kt * 16; j < k1; ++j) last += std::abs(dig[((size_t)y * (KT * 16) + j) * kDig + l]);
          if (used * 128 + last * top > kLevelMax) {
            --chunk;
            --kt;  // this window again, one k-tile narrower
            break;
          }
          used += last;
        }
      }
      return chunk;
    };
    int c = row_chunk(chunk);
    while (c < kChunkKT && chunk >= kChunkKT && is_long()) {
      ++e;
      c = row_chunk(chunk);
    }
    chunk = c;
    ex[ebase + y] = e;
    if (long_rows && is_long()) *long_rows = true;
  }
  auto at = [&](int y, int k, int i) -> uint16_t {
    if (y >= rows || k >= K) return 0;
    return bf16_bits_of_int(dig[((size_t)y * (KT * 16) + k) * kDig + i]);
  };
  for (int mt = 0; mt < MT; ++mt)
    for (int kt = 0; kt < KT; ++kt)
      for (int i = 0; i < kDig; ++i)
        for (int lane = 0; lane < 32; ++lane) {
          const int g = lane >> 2, t = lane & 3;
          const int r0 = mt * 16 + g, r1 = r0 + 8, k0 = kt * 16 + 2 * t;
          uint32_t* f = &frag[base + ((((size_t)mt * KT + kt) * kDig + i) * 32 + lane) * 4];
          f[0] = (uint32_t)at(r0, k0, i) | ((uint32_t)at(r0, k0 + 1, i) << 16);
          f[1] = (uint32_t)at(r1, k0, i) | ((uint32_t)at(r1, k0 + 1, i) << 16);
          f[2] = (uint32_t)at(r0, k0 + 8, i) | ((uint32_t)at(r0, k0 + 9, i) << 16);
          f[3] = (uint32_t)at(r1, k0 + 8, i) | ((uint32_t)at(r1, k0 + 9, i) << 16);
        }
  return chunk;
}

// the five bases [Q][D or R] (rows: planes) and the five weighted
// transposes [D or R][Q] (rows: basis index) as digit tables
bool build_recon_tc_tables(const HostTables& h, std::vector<uint32_t>& frag, std::vector<int>& ex,
                           std::vector<uint32_t>& wfrag, std::vector<int>& wex) {
  const int MT = (h.Q + 15) / 16, KT = (h.R + 15) / 16;
  const std::vector<double>* B[5] = {&h.Bq, &h.Bqp, &h.Bqpp, &h.Br, &h.Brp};
  bool ok = true;
  frag.clear();
  ex.clear();
  for (int b = 0; b < 5; ++b)
    ok &= append_digit_table(B[b]->data(), h.Q, b < 3 ? h.D : h.R, MT, KT, frag, ex) >= kChunkKT;
  const int MTw = (h.R + 15) / 16, KTw = (h.Q + 15) / 16;
  const std::vector<double>* W[5] = {&h.Wq, &h.Wqp, &h.Wqpp, &h.Wr, &h.Wrp};
  wfrag.clear();
  wex.clear();
  for (int b = 0; b < 5; ++b) {
    // rows padded to R so that every table has MTw row tiles and R exponents
    std::vector<double> m((size_t)h.R * h.Q, 0.0);
    const int rows = b < 3 ? h.D : h.R;
    std::copy(W[b]->begin(), W[b]->begin() + (size_t)rows * h.Q, m.begin());
    ok &= append_digit_table(m.data(), h.R, h.Q, MTw, KTw, wfrag, wex) >= kChunkKT;
  }
  return ok;
}

// the exact adjoint's tables: the bases transposed ([D or R][Q], rows
// padded to R) for Recon^T, and the weighted transposes of Qpw, Qw, Rw
// turned plane-major ([Q][D or R], columns padded to R) for Quad^T
bool build_adj_tc_tables(const HostTables& h, std::vector<uint32_t>& btfrag, std::vector<int>& btex,
                         std::vector<uint32_t>& wtfrag, std::vector<int>& wtex) {
  const int MTw = (h.R + 15) / 16, KTq = (h.Q + 15) / 16;
  const std::vector<double>* B[5] = {&h.Bq, &h.Bqp, &h.Bqpp, &h.Br, &h.Brp};
  bool ok = true;
  btfrag.clear();
  btex.clear();
  for (int b = 0; b < 5; ++b) {
    const int cols = b < 3 ? h.D : h.R;  // B[b] is [Q][cols]
    std::vector<double> m((size_t)h.R * h.Q, 0.0);
    for (int i = 0; i < cols; ++i)
      for (int y = 0; y < h.Q; ++y) m[(size_t)i * h.Q + y] = (*B[b])[(size_t)y * cols + i];
    ok &= append_digit_table(m.data(), h.R, h.Q, MTw, KTq, btfrag, btex) >= kChunkKT;
  }
  const std::vector<double>* W[3] = {&h.Wqp, &h.Wq, &h.Wr};  // [D or R][Q]
  wtfrag.clear();
  wtex.clear();
  for (int b = 0; b < 3; ++b) {
    const int rows = b < 2 ? h.D : h.R;
    std::vector<double> m((size_t)h.Q * h.R, 0.0);
    for (int y = 0; y < h.Q; ++y)
      for (int i = 0; i < rows; ++i) m[(size_t)y * h.R + i] = (*W[b])[(size_t)i * h.Q + y];
    ok &= append_digit_table(m.data(), h.Q, h.R, KTq, MTw, wtfrag, wtex) >= kChunkKT;
  }
  return ok;
}

// ---------------------------------------------------------------------------
// device
// ---------------------------------------------------------------------------

__host__ __device__ inline int recon_tc_kstride(int KT) { return KT * 16 + 8; }  // fp16 per digit row (padded)

// tile: kx columns per block (16 or 8)
size_t recon_tc_smem_bytes(const Grid& g, int tile) {
  const int KT = (g.R + 15) / 16;
  return (size_t)2 * kDig * (2 * tile) * recon_tc_kstride(KT) * sizeof(uint16_t) + (2 * tile + 1) * sizeof(int);
}

size_t recon_tc_smem_bytes(const Grid& g) { return recon_tc_smem_bytes(g, kTile); }

// The (kx, kz) = (0, 0) column (channel/initAlphaBeta2.c:25-68) is real: u = R a,
// du = R' a, v = 0, w = R b, dw = R' b with a, b the real parts of alpha and
// beta (a complex-to-real transform ignores the imaginary parts).  Its two
// systems are Re and Im of the beta class's column 0: the contractions with R
// and R' give (u, w) and (du, dw).  A non-finite imaginary part makes its
// system's column NaN.
__device__ __forceinline__ cpx mean_coefficients(const cpx& al, const cpx& be) {
  return cpx{exp_field(al.im) == 0x7FF ? al.im : al.re, exp_field(be.im) == 0x7FF ? be.im : be.re};
}

// u, w and du/dy, dw/dy of a column from f = -Q' alpha, g = R beta and Q''
// alpha, R' beta: u = (kx Im f + kz Im g)/K2 - i (kx Re f + kz Re g)/K2 etc.
__device__ __forceinline__ void recon_velocity(double ax, double az, const cpx& qp, const cpx& gg, cpx& u, cpx& w) {
  const cpx f = {-qp.re, -qp.im};
  u = cpx{fma(ax, f.im, az * gg.im), -fma(ax, f.re, az * gg.re)};
  w = cpx{fma(-ax, gg.im, az * f.im), fma(ax, gg.re, -az * f.re)};
}
__device__ __forceinline__ void recon_derivative(double ax, double az, const cpx& qpp, const cpx& rp, cpx& du, cpx& dw) {
  du = cpx{fma(-ax, qpp.im, az * rp.im), fma(ax, qpp.re, -az * rp.re)};
  dw = cpx{-fma(ax, rp.im, az * qpp.im), fma(ax, rp.re, az * qpp.re)};
}

// Block z ntx + tx: kx tile tx of line z.  S: the sizes (SizesRT, or SizesCT for a specialised grid); TILE kx
// columns per block (2 TILE real digit columns) in NTHR = 16 TILE threads
template <bool MULTI, class S, int TILE = kTile, int NTHR = kThreads, int MINB = 2>
__global__ void __launch_bounds__(NTHR, MINB) k_recon_tc(const __grid_constant__ Grid g0, ReconArgs a) {
  const int ntx = (g0.X + TILE - 1) / TILE;
  const int z = blockIdx.x / ntx, tx = blockIdx.x - z * ntx;
  const int inst = blockIdx.y;
  CHN_INSTANCE_GRID(g0, a.grids, inst);
  const S gsz(g);
  if (z >= gsz.Nz() || tx * TILE >= gsz.X()) return;
  if (z == gsz.Nz() / 2) return;  // never read (channel/pass1.c:51-85 skips it)
  if (a.status != nullptr && (a.status[inst / a.sdiv] & ST_CFL) != 0) return;
  const int x0 = tx * TILE;
  const int nx = min(TILE, gsz.X() - x0);
  const int KT = (gsz.R() + 15) / 16, KS = recon_tc_kstride(KT), MT = (gsz.Q() + 15) / 16;
  const bool meancol = (z == 0 && x0 == 0);  // column 0 of this tile is the mean mode
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* dig = reinterpret_cast<uint16_t*>(smem);  // [cls][digit][n 2 TILE][KS]
  int* exc = reinterpret_cast<int*>(smem + (size_t)2 * kDig * (2 * TILE) * KS * sizeof(uint16_t));  // [cls][TILE], mean's Im
  const cpx* __restrict__ C = a.C.at(inst);
  if (a.slot.stride) C += (long long)a.slot.slot() * a.slot.stride;
  auto mean_slot = [&](int cls, int col) { return meancol && cls == 1 && col == 0; };
  auto im_slot = [&](int cls, int col) { return mean_slot(cls, col) ? 2 * TILE : cls * TILE + col; };
  // coefficient (class, row, column), its exponent fields joined into e, eim
  auto cval = [&](int cls, int j, int col, int& e, int& eim) -> cpx {
    const int K = cls == 0 ? gsz.D() : gsz.R();
    if (j >= K || col >= nx) return cpx{0.0, 0.0};
    const cpx* p = C + (((size_t)z * 2 + cls) * gsz.R() + j) * gsz.X() + x0 + col;
    if (meancol && col == 0) {
      if (cls == 0) return cpx{0.0, 0.0};
      const cpx v = mean_coefficients(*(p - (size_t)gsz.R() * gsz.X()), *p);
      column_exponents(v, true, e, eim);
      return v;
    }
    column_exponents(*p, false, e, eim);
    return *p;
  };
  // column exponents: |c| < 2^exc over the column's real and imaginary parts
  for (int i = threadIdx.x; i < 2 * TILE + 1; i += NTHR) exc[i] = 0;
  __syncthreads();
  const int nent = 2 * (KT * 16) * TILE;
  if (KT <= kReconRegs && NTHR == 16 * TILE) {
    // thread t holds column t % TILE and the row pairs 2 (t / TILE) + 32 k,
    // + 1 of both classes (k < KT / 2; entry 2 k + p of vin): its coefficients
    // stay in registers from the exponent maxima to the digits, which pack two
    // rows a word
    const int col = threadIdx.x % TILE, j0 = 2 * (threadIdx.x / TILE);
    auto row = [&](int k) { return j0 + 32 * (k >> 1) + (k & 1); };
    cpx vin[2][kReconRegs];
    int emax[2] = {0, 0}, eim = 0;
#pragma unroll
    for (int cls = 0; cls < 2; ++cls)
#pragma unroll
      for (int k = 0; k < kReconRegs; ++k) {
        vin[cls][k] = k < (KT + 1) / 2 * 2 ? cval(cls, row(k), col, emax[cls], eim) : cpx{0.0, 0.0};
      }
#pragma unroll
    for (int cls = 0; cls < 2; ++cls)
      if (emax[cls]) atomicMax(&exc[cls * TILE + col], emax[cls]);
    if (eim) atomicMax(&exc[2 * TILE], eim);
    __syncthreads();
#pragma unroll
    for (int cls = 0; cls < 2; ++cls) {
      const int ex = exc[cls * TILE + col] - 1022, exi = exc[im_slot(cls, col)] - 1022;
#pragma unroll
      for (int k = 0; k < kReconRegs; k += 2) {
        if (k >= KT || row(k) >= KT * 16) break;
        // digit q of column n at dig[((cls * 7 + q) * 2 TILE + n) * KS + j]
        uint32_t* d = reinterpret_cast<uint32_t*>(dig + ((size_t)cls * kDig * (2 * TILE) + 2 * col) * KS + row(k));
        digits_pair(scaled56(vin[cls][k].re, ex), scaled56(vin[cls][k + 1].re, ex), d, (size_t)TILE * KS);
        digits_pair(scaled56(vin[cls][k].im, exi), scaled56(vin[cls][k + 1].im, exi), d + KS / 2, (size_t)TILE * KS);
      }
    }
  } else {
    for (int i = threadIdx.x; i < nent; i += NTHR) {
      const int cls = i / ((KT * 16) * TILE), r = i - cls * (KT * 16) * TILE, j = r / TILE, col = r - j * TILE;
      int e = 0, eim = 0;
      cval(cls, j, col, e, eim);
      if (e) atomicMax(&exc[cls * TILE + col], e);
      if (eim) atomicMax(&exc[2 * TILE], eim);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nent / 2; i += NTHR) {
      const int cls = i / ((KT * 8) * TILE), r = i - cls * (KT * 8) * TILE, j = 2 * (r / TILE), col = r % TILE;
      int e = 0, eim = 0;
      const cpx v0 = cval(cls, j, col, e, eim), v1 = cval(cls, j + 1, col, e, eim);
      const int ex = exc[cls * TILE + col] - 1022, exi = exc[im_slot(cls, col)] - 1022;
      // digit q of column n at dig[((cls * 7 + q) * 2 TILE + n) * KS + j]
      uint32_t* d = reinterpret_cast<uint32_t*>(dig + ((size_t)cls * kDig * (2 * TILE) + 2 * col) * KS + j);
      digits_pair(scaled56(v0.re, ex), scaled56(v1.re, ex), d, (size_t)TILE * KS);
      digits_pair(scaled56(v0.im, exi), scaled56(v1.im, exi), d + KS / 2, (size_t)TILE * KS);
    }
  }
  __syncthreads();

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  const int NT = (2 * nx + 7) / 8;  // n-tiles of 8 real columns (4 complex)
  const uint4* __restrict__ A = reinterpret_cast<const uint4*>(g.tcA);
  cpx* __restrict__ U = a.U.at(inst);
  const size_t cs = (size_t)gsz.Q() * gsz.X();
  const int order[5] = {0, 1, 3, 2, 4};
  for (int item = warp; item < MT * NT; item += NTHR >> 5) {
    const int mt = item / NT, nt = item - mt * NT;
    const int col = nt * 4 + t;  // this thread's complex column
    cpx held[2];                 // Q' alpha, then Q'' alpha, at rows gq and gq + 8
    for (int ob = 0; ob < 5; ++ob) {
      const int b = order[ob], cls = b < 3 ? 0 : 1;
      const int KTb = ((cls == 0 ? gsz.D() : gsz.R()) + 15) / 16;
      const int ecol = col_exp(exc[cls * TILE + col]) - 64 + LongFold().shift();
      const int ecoli = col_exp(exc[im_slot(cls, col)]) - 64 + LongFold().shift();
      long long T[4];
      uint32_t R[4] = {0, 0, 0, 0};
      tc_tile_range<(MINB <= 2)>(LongFold(), A + (size_t)b * MT * KT * kDig * 32, mt, KT, 0, KTb, kChunkKT,
                                 dig + (size_t)cls * kDig * (2 * TILE) * KS, KS, (size_t)(2 * TILE) * KS, nt * 8, lane,
                                 T, R);
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int y = mt * 16 + gq + 8 * rr;
        if (y >= gsz.Q() || col >= nx) continue;
        const bool mean = meancol && col == 0;
        const int e = g.tcE[(size_t)b * gsz.Q() + y];
        const cpx val = {round_sum(LongFold(), T[2 * rr], R[2 * rr], e + ecol),
                         round_sum(LongFold(), T[2 * rr + 1], R[2 * rr + 1], e + ecoli)};
        const int x = x0 + col;
        cpx* out = U + ((size_t)z * 5 * gsz.Q() + y) * gsz.X() + x;
        const double ax = g.kxK2[(size_t)z * gsz.X() + x], az = g.kzK2[(size_t)z * gsz.X() + x];
        if (b == 0) {
          out[cs] = val;  // v = Q alpha
        } else if (b == 1 || b == 2) {
          held[rr] = val;
        } else if (mean) {
          out[b == 3 ? 0 : 3 * cs] = cpx{val.re, 0.0};
          out[b == 3 ? 2 * cs : 4 * cs] = cpx{val.im, 0.0};
        } else if (b == 3) {
          recon_velocity(ax, az, held[rr], val, out[0], out[2 * cs]);
        } else {
          recon_derivative(ax, az, held[rr], val, out[3 * cs], out[4 * cs]);
        }
      }
    }
  }
}

// The reconstruction for launches with few blocks, where a block has its SM
// almost to itself: 4-column tiles (one 8-column digit tile), a warp per
// (16 planes, output group) -- u and w, du/dy and dw/dy, v -- whose tables'
// k-tiles run as one stream with two in flight.  KP: row pairs of a class a
// thread holds (R <= 64 KP).
template <class S, int KP>
__global__ void __launch_bounds__(256, 1) k_recon_few(const __grid_constant__ Grid g, ReconArgs a) {
  constexpr int TILE = 4, NTHR = 256, NC = 2 * TILE;
  const S gsz(g);
  const int ntx = (gsz.X() + TILE - 1) / TILE;
  const int z = blockIdx.x / ntx, tx = blockIdx.x - z * ntx;
  const int inst = blockIdx.y;
  if (z == gsz.Nz() / 2) return;  // never read (channel/pass1.c:51-85 skips it)
  if (a.status != nullptr && (a.status[inst / a.sdiv] & ST_CFL) != 0) return;
  const cpx* __restrict__ C = a.C.at(inst);
  if (a.slot.stride) C += (long long)a.slot.slot() * a.slot.stride;
  cpx* __restrict__ U = a.U.at(inst);
  const int x0 = tx * TILE, nx = min(TILE, gsz.X() - x0);
  const bool meancol = z == 0 && x0 == 0;
  const int KT = (gsz.R() + 15) / 16, KS = recon_tc_kstride(KT), MT = (gsz.Q() + 15) / 16;
  extern __shared__ __align__(16) unsigned char smem[];
  uint16_t* dig = reinterpret_cast<uint16_t*>(smem);  // [cls][digit][n 2 TILE][KS]
  int* exc = reinterpret_cast<int*>(smem + (size_t)2 * kDig * NC * KS * sizeof(uint16_t));  // [cls][TILE], mean's Im
  if (threadIdx.x < 2 * TILE + 1) exc[threadIdx.x] = 0;
  __syncthreads();
  {
    // threads [0, 128) the alpha rows, the rest the beta ones; row pairs 2 (t / TILE) + 64 k
    const int cls = threadIdx.x >> 7, col = threadIdx.x % TILE, j0 = 2 * ((threadIdx.x & 127) / TILE);
    const int K = cls == 0 ? gsz.D() : gsz.R();
    const bool mean = meancol && col == 0, on = col < nx && !(mean && cls == 0), own = mean && cls == 1;
    const cpx* src = C + ((size_t)(z * 2 + cls) * gsz.R()) * gsz.X() + x0 + col;
    cpx v[KP][2];
    int e = 0, eim = 0;
#pragma unroll
    for (int k = 0; k < KP; ++k)
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int j = j0 + p + 64 * k;
        v[k][p] = (on && j < K) ? src[(size_t)j * gsz.X()] : cpx{0.0, 0.0};
        if (mean && on && j < K) v[k][p] = mean_coefficients(src[((ptrdiff_t)j - gsz.R()) * gsz.X()], v[k][p]);
        column_exponents(v[k][p], own, e, eim);
      }
#pragma unroll
    for (int o = 16; o >= TILE; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
    if ((threadIdx.x & 31) < TILE) atomicMax(&exc[cls * TILE + col], e);
    if (eim) atomicMax(&exc[2 * TILE], eim);
    __syncthreads();
    const int ex = exc[cls * TILE + col] - 1022, exi = own ? exc[2 * TILE] - 1022 : ex;
#pragma unroll
    for (int k = 0; k < KP; ++k) {
      const int j = j0 + 64 * k;
      if (j >= KT * 16) break;
      uint32_t* d = reinterpret_cast<uint32_t*>(dig + ((size_t)cls * kDig * NC + 2 * col) * KS + j);
      digits_pair(scaled56(v[k][0].re, ex), scaled56(v[k][1].re, ex), d, (size_t)NC * KS / 2);
      digits_pair(scaled56(v[k][0].im, exi), scaled56(v[k][1].im, exi), d + KS / 2, (size_t)NC * KS / 2);
    }
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t = lane & 3;
  const uint4* __restrict__ A = reinterpret_cast<const uint4*>(g.tcA) + lane;
  const size_t cs = (size_t)gsz.Q() * gsz.X();
  const int x = x0 + min(t, nx - 1);
  const double ax = g.kxK2[(size_t)z * gsz.X() + x], az = g.kzK2[(size_t)z * gsz.X() + x];
  const uint32_t base0 = tc_row_addr(dig, KS, (size_t)NC * KS, 0, lane);
  const uint32_t cls_bytes = (uint32_t)(2 * kDig * NC * KS);
  // items: (Q', R) of every row tile, (Q'', R'), then Q
  const int nit = 3 * MT;
  auto table = [&](int item, int part) {
    const int grp = item / MT, mt = item - grp * MT, b = grp == 0 ? (part ? 3 : 1) : (grp == 1 ? (part ? 4 : 2) : 0);
    return A + ((size_t)b * MT + mt) * KT * kFragStep;
  };
  FragPair pf;
  if (warp < nit) tc_stream_start(pf, table(warp, 0));
  for (int item = warp; item < nit; item += NTHR / 32) {
    const int grp = item / MT, mt = item - grp * MT, nxt = item + NTHR / 32;
    const int nparts = grp < 2 ? 2 : 1;
    cpx val[2][2];
    for (int part = 0; part < nparts; ++part) {
      const int b = grp == 0 ? (part ? 3 : 1) : (grp == 1 ? (part ? 4 : 2) : 0), cls = b < 3 ? 0 : 1;
      const uint4* next = part + 1 < nparts ? table(item, 1) : (nxt < nit ? table(nxt, 0) : nullptr);
      long long T[4];
      uint32_t R[4] = {0, 0, 0, 0};
      tc_tile_stream(LongFold(), pf, table(item, part), next, KT, base0 + cls * cls_bytes, (uint32_t)(4 * NC * KS), T, R);
      const int ecol = col_exp(exc[cls * TILE + t]) - 64 + LongFold().shift();
      const int ecoli = meancol && cls == 1 && t == 0 ? col_exp(exc[2 * TILE]) - 64 + LongFold().shift() : ecol;
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const int e = g.tcE[(size_t)b * gsz.Q() + min(mt * 16 + gq + 8 * rr, gsz.Q() - 1)];
        const cpx v = {round_sum(LongFold(), T[2 * rr], R[2 * rr], e + ecol),
                       round_sum(LongFold(), T[2 * rr + 1], R[2 * rr + 1], e + ecoli)};
        if (part) val[1][rr] = v;
        else val[0][rr] = v;
      }
    }
#pragma unroll
    for (int rr = 0; rr < 2; ++rr) {
      const int y = mt * 16 + gq + 8 * rr;
      if (y >= gsz.Q() || t >= nx) continue;
      cpx* out = U + ((size_t)z * 5 * gsz.Q() + y) * gsz.X() + x;
      if (meancol && t == 0 && grp < 2) {
        out[grp == 0 ? 0 : 3 * cs] = cpx{val[1][rr].re, 0.0};
        out[grp == 0 ? 2 * cs : 4 * cs] = cpx{val[1][rr].im, 0.0};
      } else if (grp == 0) recon_velocity(ax, az, val[0][rr], val[1][rr], out[0], out[2 * cs]);
      else if (grp == 1) recon_derivative(ax, az, val[0][rr], val[1][rr], out[3 * cs], out[4 * cs]);
      else out[cs] = val[0][rr];
    }
  }
}

// Grid::rbuild (single-grid batches) 0: 16-column tiles in 256-thread
// blocks at 2 per SM; 1: 8-column tiles in 128-thread blocks at 4; 2:
// 16-column tiles at 3 per SM, the table fragments loaded without prefetch
// (80 registers)
template <class S>
static void launch_recon_sizes(const Grid& g, const ReconArgs& a, cudaStream_t st) {
  if (g.rbuild == 1 && !a.grids) {
    const int ntx = (g.X + 7) / 8;
    k_recon_tc<false, S, 8, 128, 4><<<dim3(g.Nz * ntx, a.ninst), 128, recon_tc_smem_bytes(g, 8), st>>>(g, a);
    return;
  }
  if (g.rbuild == 2 && !a.grids) {
    const int ntx = (g.X + kTile - 1) / kTile;
    k_recon_tc<false, S, 16, 256, 3><<<dim3(g.Nz * ntx, a.ninst), 256, recon_tc_smem_bytes(g), st>>>(g, a);
    return;
  }
  const int ntx = (g.X + kTile - 1) / kTile;
  const size_t sm = recon_tc_smem_bytes(g);
  if (a.grids) k_recon_tc<true, SizesRT><<<dim3(g.Nz * ntx, a.ninst), kThreads, sm, st>>>(g, a);
  else k_recon_tc<false, S><<<dim3(g.Nz * ntx, a.ninst), kThreads, sm, st>>>(g, a);
}

// Grid::fixed & FIXED_RECON: the build compiled for the grid's sizes; launches
// of at most kFewTiles 4-column tiles (two waves of one block per SM) take
// k_recon_few, unless CHN_RECON_BUILD asked for a build
cudaError_t launch_recon_tc(const Grid& g, const ReconArgs& a, cudaStream_t st) {
  const int ntf = g.Nz * ((g.X + 3) / 4);
  if (!a.grids && !g.rfixed && g.R > 16 && g.R <= 128 && (long long)ntf * a.ninst <= kFewTiles) {
    const dim3 grid(ntf, a.ninst);
    const size_t sm = recon_tc_smem_bytes(g, 4);
    const bool fx = (g.fixed & FIXED_RECON) != 0;
    if (fx && sizes_match<Sizes32>(g)) k_recon_few<Sizes32, 1><<<grid, 256, sm, st>>>(g, a);
    else if (fx && sizes_match<Sizes16>(g)) k_recon_few<Sizes16, 1><<<grid, 256, sm, st>>>(g, a);
    else if (g.R <= 64) k_recon_few<SizesRT, 1><<<grid, 256, sm, st>>>(g, a);
    else k_recon_few<SizesRT, 2><<<grid, 256, sm, st>>>(g, a);
    return cudaGetLastError();
  }
  const bool fx = (g.fixed & FIXED_RECON) && !a.grids;
  if (fx && sizes_match<Sizes32>(g)) launch_recon_sizes<Sizes32>(g, a, st);
  else if (fx && sizes_match<Sizes16>(g)) launch_recon_sizes<Sizes16>(g, a, st);
  else launch_recon_sizes<SizesRT>(g, a, st);
  return cudaGetLastError();
}

void prepare_recon_tc(int optin) {
  allow_max_smem(k_recon_few<Sizes32, 1>, optin);
  allow_max_smem(k_recon_few<Sizes16, 1>, optin);
  allow_max_smem(k_recon_few<SizesRT, 1>, optin);
  allow_max_smem(k_recon_few<SizesRT, 2>, optin);
  allow_max_smem(k_recon_tc<false, SizesRT>, optin);
  allow_max_smem(k_recon_tc<true, SizesRT>, optin);
  allow_max_smem(k_recon_tc<false, Sizes32>, optin);
  allow_max_smem(k_recon_tc<false, Sizes16>, optin);
  allow_max_smem(k_recon_tc<false, SizesRT, 16, 256, 3>, optin);
  allow_max_smem(k_recon_tc<false, Sizes32, 16, 256, 3>, optin);
  allow_max_smem(k_recon_tc<false, Sizes16, 16, 256, 3>, optin);
  allow_max_smem(k_recon_tc<false, SizesRT, 8, 128, 4>, optin);
  allow_max_smem(k_recon_tc<false, Sizes32, 8, 128, 4>, optin);
  allow_max_smem(k_recon_tc<false, Sizes16, 8, 128, 4>, optin);
}

}  // namespace chn
