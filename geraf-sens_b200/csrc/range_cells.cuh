// Range cells: the sample sums of the MIXED form as piecewise polynomials of
// the path length.
//
// For one antenna the sum over samples is a trigonometric polynomial of the
// phase step d = k1 (D + 0.15) (cycles per sample), D the path length:
//   P(d) = sum_n s_n e^{-j 2 pi n d}.
// With the samples counted from their middle, n' = n - (S - 1)/2, the sum
//   P'(D) = sum_n s_n e^{-j 2 pi n' d(D)} = e^{+j 2 pi (S - 1)/2 d} P(d)
// varies slowly: over a cell of path length 1/kappa its fastest mode turns by
// pi S k1 / kappa rad.  In cell k, D = (k + x) / kappa with x in [-1/2, 1/2], each
// mode's e^{-j theta_n x}, theta_n = 2 pi n' k1 / kappa, is replaced by its
// interpolant of degree Q - 1 at the Q Chebyshev nodes, so P' is a polynomial
// of degree Q - 1 in x whose Q complex coefficients are sums over the samples
// formed once per (antenna, cell), and a (point, antenna) pair costs Q - 1
// multiply-adds instead of S.  The interpolation error of a mode is at most
// 2 J_Q(theta_n / 2) (Jacobi-Anger): see CellParams for the choices of kappa
// and Q, which keep it below the FP32 rounding of the sums.
// The phase of the middle sample joins the carrier's (K, b of PairPhase), so it
// costs nothing per pair.
#pragma once

#include "common.cuh"

namespace geraf {

// Cell width and coefficients.  Evaluation (gather): 4 S k1 cells per metre
// (18.7 mm at 4 GHz of swept bandwidth) with 6 coefficients: theta <= pi/4, error
// <= 1.6e-7 for the outermost sample, 3e-8 in the mean.  Accumulation (moments):
// 2 S k1 cells per metre (37 mm) with 8: theta <= pi/2, error <= 2.8e-8; wider cells are
// left less often but hold more moments (10 in 75 mm cells and 6 in 18.7 mm cells
// took the same time on 972 antennas x 50653 voxels, 6 in 18.7 mm cells 8% more on points
// along rays).
template <int OVERSAMPLE, int Q_>
struct CellParams {
  static constexpr int kOver = OVERSAMPLE;
  static constexpr int Q = Q_;
};
using GatherCells = CellParams<4, 6>;
using MomentCells = CellParams<2, 8>;

// Lengths of the pairs' legs are held in units of 2^-20 m (coordinates scaled by
// 2^20, exactly): a leg below 8 m is a whole number below 2^23 plus a rest, and
// the sum of two whole parts is exact in FP32.  Longer legs leave the cells to
// the direct kernels.
constexpr double kUnit = 1048576.0;  // per metre
constexpr double kMaxLeg = 7.9;      // metres
// Magic numbers of the rounding tricks.
constexpr float kWholeMagic = 8388608.0f;         // 2^23: fma(s, r, magic) rounds to a whole number
constexpr uint32_t kWholeMagicBits = 0x4B000000u;
constexpr float kRoundMagic = 12582912.0f;        // 1.5 * 2^23: also for negative numbers
constexpr uint32_t kRoundMagicBits = 0x4B400000u;
// s + kRestMagic holds s in steps of 2^4 square units; its low word is then the
// residual s - d^2 in those steps (|.| < 2^22 for legs below 8 m).
constexpr double kRestMagic = 1.5 * 72057594037927936.0;  // 1.5 * 2^56
constexpr float kRestStep = 16.0f;

__device__ __forceinline__ float rsqrt_fast(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// One leg of a path in units, |t - v| = d + (kRestStep / 2) l: d whole, the rest
// from one Newton step on the FP64 residual (total error ~1e-11 m at 0.5 m).
// s = |t - v|^2 = |t|^2 + |v|^2 - 2 t.v in FP64: 4 operations instead of 6, its
// cancellation (~1e-16 of the squared coordinates) far below what the phase
// needs (~1e-10 m^2).  tt carries a bias of that size so that s stays positive.
// Both hold only for coordinates that are small themselves, so t and v are taken from
// the centre of the scene's box (box_center), differences that FP64 forms exactly or
// nearly so: the centre is no further from an antenna than the box's far corner, so with legs
// below 8 m both stay below 8 m wherever the scene lies (about an origin 3 km away the
// phase would be off by 5e-4 rad, about one 1000 km away by cells).
// No conversion between FP32 and FP64 is issued: they share the 16-lane unit of the
// rsqrt, sine and cosine, which bounded the kernel with them (115 issue cycles
// per 32 pairs of the forward at 3072 x 110592 pairs); the words are shifted or
// read off magic sums instead.
struct Leg {
  float d, l;
};
__device__ __forceinline__ Leg leg_length(double m2x, double m2y, double m2z, double tt, double x, double y, double z,
                                          double vv) {
  const double s = fma(m2x, x, fma(m2y, y, fma(m2z, z, tt + vv)));
  // float(s), truncated: the exponent bias moves from 1023 to 127
  const float sf = __uint_as_float(
      __funnelshift_l(static_cast<uint32_t>(__double2loint(s)), static_cast<uint32_t>(__double2hiint(s)), 3) + 0x40000000u);
  const float r = rsqrt_fast(sf);
  const float w = fmaf(sf, r, kWholeMagic);
  Leg g;
  g.d = w - kWholeMagic;
  const double dd = __hiloint2double(0x43300000, static_cast<int>(__float_as_uint(w) - kWholeMagicBits)) -
                    4503599627370496.0;  // 2^52
  const double rest = fma(-dd, dd, s + kRestMagic);
  g.l = (__uint_as_float(static_cast<uint32_t>(__double2loint(rest)) + kRoundMagicBits) - kRoundMagic) * r;
  return g;
}

// Phase constants of a pair, in cycles: c = (d + (kRestStep / 2) l) K + b for the
// carrier plus the middle sample; kh + kl = K, b reduced to [-1/2, 1/2].
struct PairPhase {
  float kh, kl, k_rest, b;
  float kappa, kappa_rest;  // cells per unit
};

// kappa: cells per metre.
// Cells per metre for S samples, as the kernels round it.
inline double cells_per_metre(double k1, int64_t S, int over) {
  return static_cast<double>(static_cast<float>(over * static_cast<double>(S) * (k1 < 0.0 ? -k1 : k1)));
}

inline PairPhase pair_phase(double k0, double b0, double k1, double b1, int64_t S, double kappa) {
  const double mid = 0.5 * static_cast<double>(S - 1);
  const double K = (k0 + mid * k1) / kUnit;
  const double b = b0 + mid * b1;
  PairPhase p;
  p.kh = static_cast<float>(K);
  p.kl = static_cast<float>(K - static_cast<double>(p.kh));
  p.k_rest = 0.5f * kRestStep * p.kh;
  p.b = static_cast<float>(b - nearbyint(b));
  p.kappa = static_cast<float>(kappa / kUnit);
  p.kappa_rest = 0.5f * kRestStep * p.kappa;
  return p;
}

// Phase in cycles, within about [-1, 1], of the path hi + (kRestStep / 2) lo: each
// multiply-add rounds a number below 1, so the result is good to ~1e-7 cycles.
__device__ __forceinline__ float pair_cycles(const PairPhase& p, float hi, float lo) {
  const float k = fmaf(hi, p.kh, kRoundMagic) - kRoundMagic;
  return fmaf(hi, p.kh, -k) + fmaf(lo, p.k_rest, fmaf(hi, p.kl, p.b));
}

template <bool ACCURATE>
__device__ __forceinline__ float2 pair_phasor(float cycles) {
  return ACCURATE ? cis_cycles(cycles) : cis_cycles_fast(cycles);
}

// Cell of the path and the offset x in it; m is the cell index plus the magic.
struct CellPos {
  float m, x;
};
__device__ __forceinline__ CellPos pair_cell(const PairPhase& p, float hi, float lo) {
  CellPos c;
  c.m = fmaf(hi, p.kappa, kRoundMagic);
  const float k = c.m - kRoundMagic;
  c.x = fmaf(lo, p.kappa_rest, fmaf(hi, p.kappa, -k));
  return c;
}

// Middle of one side of the scene's box.
__device__ __forceinline__ double box_center(float lo, float hi) {
  return 0.5 * (static_cast<double>(lo) + static_cast<double>(hi));
}

// An antenna's coordinates for leg_length; bias bounds the voxels' |v|^2.
__device__ __forceinline__ void leg_antenna(const double* t, double bias, double* m) {
#pragma unroll
  for (int c = 0; c < 3; ++c) m[c] = -2.0 * kUnit * t[c];
  const double tt = fma(t[2], t[2], fma(t[1], t[1], t[0] * t[0]));
  m[3] = (tt + (4e-15 * (tt + bias) + 1e-18)) * (kUnit * kUnit);
}

// Range of |t - x| + |r - x| over the box [lo, hi] (lo xyz, hi xyz), and its longest leg.
template <typename F>
__device__ __forceinline__ void leg_range(const F* t, const F* box, F& near2, F& far2) {
  near2 = far2 = F(0);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const F a = box[c] - t[c], b = t[c] - box[3 + c];
    const F e = a > b ? (a > F(0) ? a : F(0)) : (b > F(0) ? b : F(0));
    const F fa = a < F(0) ? -a : a, fb = b < F(0) ? -b : b;
    const F g = fa > fb ? fa : fb;
    near2 += e * e;
    far2 += g * g;
  }
}

// Positive Chebyshev nodes on [-1/2, 1/2], cos((2 i + 1) pi / (2 Q)) / 2.
template <int Q>
__host__ __device__ constexpr double cell_node(int i) {
  static_assert(Q == 6 || Q == 8, "the numbers of coefficients in use");
  if (Q == 6) return i == 0 ? 0.48296291314453416 : i == 1 ? 0.3535533905932738 : 0.12940952255126037;
  return i == 0 ? 0.4903926402016152 : i == 1 ? 0.4157348061512726 : i == 2 ? 0.27778511650980114 : 0.09754516100806417;
}

// Interpolation of cos(theta x) and sin(theta x) on [-1/2, 1/2]: coefficients
// g[j] of x^j, even j for the cosine, odd j for the sine, from Newton's divided
// differences in x^2 at the positive nodes (FP64; every divisor is a compile-time constant).
template <int Q>
__device__ __forceinline__ void cell_basis(double theta, float* g) {
  constexpr int H = Q / 2;
  double c[H], s[H];
#pragma unroll
  for (int i = 0; i < H; ++i) {
    double sn, cs;
    sincos(theta * cell_node<Q>(i), &sn, &cs);
    c[i] = cs;
    s[i] = sn * (1.0 / cell_node<Q>(i));
  }
#pragma unroll
  for (int o = 1; o < H; ++o) {
#pragma unroll
    for (int i = H - 1; i >= o; --i) {
      const double d = 1.0 / (cell_node<Q>(i) * cell_node<Q>(i) - cell_node<Q>(i - o) * cell_node<Q>(i - o));
      c[i] = (c[i] - c[i - 1]) * d;
      s[i] = (s[i] - s[i - 1]) * d;
    }
  }
  // Newton form to monomials in x^2
  double mc[H] = {}, ms[H] = {};
#pragma unroll
  for (int i = H - 1; i >= 0; --i) {
    const double X = cell_node<Q>(i) * cell_node<Q>(i);
#pragma unroll
    for (int q = H - 1; q >= 1; --q) {
      mc[q] = mc[q - 1] - X * mc[q];
      ms[q] = ms[q - 1] - X * ms[q];
    }
    mc[0] = c[i] - X * mc[0];
    ms[0] = s[i] - X * ms[0];
  }
#pragma unroll
  for (int q = 0; q < H; ++q) {
    g[2 * q] = static_cast<float>(mc[q]);
    g[2 * q + 1] = static_cast<float>(ms[q]);
  }
}

}  // namespace geraf
