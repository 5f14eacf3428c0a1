// Dimensions of the inverse transforms as digit GEMMs (the mma.sync kernel
// of phys_tc.cu and the tcgen05 kernel of phys_tc5.cu share them).
#pragma once

#include <vector>

#include "chn_common.cuh"
#include "setup.h"
#include "tc_common.cuh"

namespace chn {

static constexpr int kFB = 2;  // fields per pass of the mma.sync inverse (its widest build)

// kept kz modes of even / odd padded index zp (kk < Nz/2: zp = kk; else
// zp = kk + 1 + Nz/2, which runs over the odd Nz + 1 ... 3Nz/2 - 1); an odd
// pz keeps all modes in one class
__host__ __device__ constexpr void z_class_counts(int Nz, int pz, int& nE, int& nO) {
  if (pz % 2) {
    nE = Nz - 1;
    nO = 0;
    return;
  }
  const int h = Nz / 2;
  nE = (h + 1) / 2 + (h - 1) / 2;
  nO = h / 2 + h / 2;
}

struct PhysTcDims {
  int Rz, Rx, pzh, pxh;           // radix of each stage's split, output rows per half
  int nxE, nxO;                   // x modes of even / odd j
  int KTzE, KTz, KTxE, KTx;       // k-tiles of the even class, and in all
  int MTz, MTx, KSz, KSx, NZ, NX;  // NZ = columns of the z stage, NX = of the x stage
};

// from the sizes (a constant expression for compile-time sizes); fb: fields
// per pass (the x stage has one column per (field, m))
__host__ __device__ constexpr PhysTcDims phys_tc_dims_n(int Nz, int pz, int px, int X, int fb) {
  PhysTcDims d{};
  d.Rz = pz % 2 ? 1 : 2;
  d.Rx = px % 2 ? 1 : 2;
  d.pzh = pz / d.Rz;
  d.pxh = px / d.Rx;
  int nzE = 0, nzO = 0;
  z_class_counts(Nz, pz, nzE, nzO);
  d.nxE = (X + d.Rx - 1) / d.Rx;
  d.nxO = X - d.nxE;
  d.KTzE = (2 * nzE + 15) / 16;
  d.KTz = d.KTzE + (2 * nzO + 15) / 16;
  d.KTxE = (2 * d.nxE + 15) / 16;
  d.KTx = d.KTxE + (2 * d.nxO + 15) / 16;
  d.MTz = (2 * d.pzh + 15) / 16;
  d.MTx = (d.pxh + 15) / 16;
  d.KSz = d.KTz * 16 + 8;
  d.KSx = d.KTx * 16 + 8;
  d.NZ = fb * X;
  d.NX = fb * pz;
  return d;
}

__host__ __device__ inline PhysTcDims phys_tc_dims(const Grid& g, int fb = kFB) {
  return phys_tc_dims_n(g.Nz, g.pz, g.px, g.X, fb);
}

// the folded sums t (unit 2^fs) of the z stage (every row of its table has the
// exponent kZRowExp) of a column whose largest input exponent field is ce: the
// value is t 2^zsum_exp(ce); zsum_field: its exponent field (<= 0 for zeros; 0x7FF where
// the column held an infinity or a NaN)
static constexpr int kZRowExp = 1;
__device__ __forceinline__ int zsum_exp(int ce, int fs) { return kZRowExp + ce - 1022 - 64 + fs; }
__device__ __forceinline__ int zsum_field(long long t, int ce, int fs) { return sum_field(t, zsum_exp(ce, fs), ce); }
// of the forward x stage, without its row's exponent
__device__ __forceinline__ int ysum_exp(int ce, int fs) { return ce - 1022 - 64 + fs; }

// Dimensions of the forward transforms as digit GEMMs, the x stage (px is even)
// and for an even pz the z stage split radix-2 (decimation in frequency: the even outputs are the
// transform of a[n] + a[n + N/2], the odd ones of a[n] - a[n + N/2], exact on
// the 56-bit integers; half the digit products and table bytes: 32x65x32, 256
// products' instances 2.91 -> 2.78 ms over zero primal fields, 128x129x128, one, 1.21 -> 0.87).  Class c of a
// stage: its row tiles from MT?E on (c = 1), its digits KT?c k-tiles on.
struct FwdTcDims {
  int Rz, pxh, pzh;                     // radix of the z stage's split, inputs per class
  int nxE, nxO, nzE, nzO;               // kept outputs of even / odd index
  int KTxc, KTzc;                       // k-tiles of a class
  int MTxE, MTx, MTzE, MTz, KSx, KSz, pzp, Xp, Kk;
};

__host__ __device__ constexpr FwdTcDims fwd_tc_dims_n(int Nz, int X, int pz, int px) {
  FwdTcDims d{};
  d.Rz = pz % 2 ? 1 : 2;
  d.pxh = px / 2;
  d.pzh = pz / d.Rz;
  d.nxE = (X + 1) / 2;
  d.nxO = X - d.nxE;
  z_class_counts(Nz, pz, d.nzE, d.nzO);
  d.Kk = Nz - 1;
  d.KTxc = (d.pxh + 15) / 16;
  d.KTzc = (2 * d.pzh + 15) / 16;
  d.MTxE = (2 * d.nxE + 15) / 16;
  d.MTx = d.MTxE + (2 * d.nxO + 15) / 16;
  d.MTzE = (2 * d.nzE + 15) / 16;
  d.MTz = d.MTzE + (2 * d.nzO + 15) / 16;
  d.KSx = 2 * d.KTxc * 16 + 8;
  d.KSz = d.Rz * d.KTzc * 16 + 8;
  d.pzp = (pz + 7) / 8 * 8;
  d.Xp = (X + 7) / 8 * 8;
  return d;
}

__host__ __device__ inline FwdTcDims fwd_tc_dims(const Grid& g) { return fwd_tc_dims_n(g.Nz, g.X, g.pz, g.px); }

// the row of a stage's class (2 e + part) that row tile mt, row r (< 16) holds;
// false past the class
struct FwdRow {
  int cls, e, part;
};
__device__ __forceinline__ bool fwd_row(int mt, int r, int mtE, int nE, int nO, FwdRow& o) {
  o.cls = mt >= mtE ? 1 : 0;
  const int row = (mt - (o.cls ? mtE : 0)) * 16 + r;
  o.e = row >> 1;
  o.part = row & 1;
  return o.e < (o.cls ? nO : nE);
}
// the kept kz index of the e-th z output of a class (z_class_modes' order: kk <
// Nz/2 of that parity, then those whose padded index kk + 1 + Nz/2 has it)
__device__ __forceinline__ int fwd_z_mode(int Nz, int Rz, int cls, int e) {
  if (Rz == 1) return e;
  const int h = Nz / 2, low = (h + 1 - cls) / 2;  // kk = cls, cls + 2, ... < h
  if (e < low) return 2 * e + cls;
  // kk >= h with (kk + 1 + h) % 2 == cls: the first is h + ((h + 1 + h + cls) & 1)
  return h + ((1 + cls) & 1) + 2 * (e - low);
}
// digits of an x-stage column's two classes at inputs k, k + 1 (k even): the
// sums and differences with those pxh on
__device__ __forceinline__ void fwd_x_digits(const FwdTcDims& d, const double* src, int k, bool on, int ex, uint32_t* out,
                                             size_t stride) {
  const bool o0 = on && k < d.pxh, o1 = on && k + 1 < d.pxh;
  const long long a0 = scaled56(o0 ? src[k] : 0.0, ex), a1 = scaled56(o1 ? src[k + 1] : 0.0, ex);
  const long long b0 = scaled56(o0 ? src[k + d.pxh] : 0.0, ex), b1 = scaled56(o1 ? src[k + 1 + d.pxh] : 0.0, ex);
  digits_pair<true>(a0 + b0, a1 + b1, out + (k >> 1), stride);
  digits_pair<true>(a0 - b0, a1 - b1, out + d.KTxc * 8 + (k >> 1), stride);
}
// of a z-stage column's inputs zp (re, im) and zp + pzh, as 56-bit integers
__device__ __forceinline__ void fwd_z_digits(const FwdTcDims& d, int zp, longlong2 a, longlong2 b, uint32_t* out,
                                             size_t stride) {
  if (d.Rz == 1) {
    digits_pair<true>(a.x, a.y, out + zp, stride);
    return;
  }
  digits_pair<true>(a.x + b.x, a.y + b.y, out + zp, stride);
  digits_pair<true>(a.x - b.x, a.y - b.y, out + d.KTzc * 8 + zp, stride);
}

// the two stages' matrices (rows x K words of Re, Im) and the z stage's
// K-word -> kept kz map
bool phys_tc_matrices(const HostTables& h, std::vector<double>& Az, std::vector<double>& Ax,
                      std::vector<int>& zmap, int& zrows, int& Kz, int& xrows, int& Kx);

}  // namespace chn
