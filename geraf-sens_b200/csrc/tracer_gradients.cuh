// Gradients of one live (point, antenna) pair of the MIXED tracer adjoints, from the
// cell polynomial of the antenna's residual row (range_cells.cuh).  With P(x) =
// sum_n g_n e^{-j 2 pi n' d} (samples counted from their middle) and e the phasor of
// carrier and middle sample,
//   sum_n (g_r cos + g_i sin)       =  Re(e conj(P)),
//   sum_n w_n (g_i cos - g_r sin)   = -Im(e (w_mid conj(P) - j kappa c conj(P'))),
// so the phase-rate sum of the position gradient needs the derivative P' only for
// the sweep's share of the rate (a few percent of the carrier's), and the
// derivative's larger interpolation error stays below the FP32 rounding.
#pragma once

#include "range_cells.cuh"
#include "tracer_geometry.cuh"

namespace geraf {
namespace tracer {

struct AdjConsts {
  double K, b;   // phase of carrier and middle sample, cycles per metre and bias
  double k1, b1; // phase step per sample
  double kappa, theta_step;
  float w_mid, kappa_c;  // phase rate of carrier and middle sample; cells per unit delay
  int S;
};

inline AdjConsts adj_consts(double k0, double b0, double k1, double b1, float f0, float As, float fs, int64_t S) {
  AdjConsts c;
  const double mid = 0.5 * static_cast<double>(S - 1);
  c.K = k0 + mid * k1;
  c.b = b0 + mid * b1;
  c.k1 = k1;
  c.b1 = b1;
  // without a sweep every path is in one cell
  const double kappa = GatherCells::kOver * static_cast<double>(S) * (k1 < 0.0 ? -k1 : k1);
  c.kappa = kappa > 1e-6 ? kappa : 1e-6;
  c.theta_step = 2.0 * 3.14159265358979323846 * k1 / c.kappa;
  c.w_mid = static_cast<float>(2.0 * static_cast<double>(kPiF) * (static_cast<double>(f0) + static_cast<double>(As) / fs * mid));
  c.kappa_c = static_cast<float>(c.kappa * static_cast<double>(kSpeedOfLight));
  c.S = static_cast<int>(S);
  return c;
}

// Cell, offset and phasor of a pair's path, lengths in FP64.
struct PairPath {
  double cell;  // a whole number
  float x;
  float2 e;
};
__device__ __forceinline__ PairPath pair_path(const AdjConsts& c, const float* txp, const float* rxp, const float* pt) {
  double st = 0.0, sr = 0.0;
#pragma unroll
  for (int k = 2; k >= 0; --k) {
    const double dt = static_cast<double>(txp[k]) - static_cast<double>(pt[k]);
    const double dr = static_cast<double>(rxp[k]) - static_cast<double>(pt[k]);
    st = fma(dt, dt, st);
    sr = fma(dr, dr, sr);
  }
  const double d = sqrt_f64_fast(st) + sqrt_f64_fast(sr);
  const double u = d * c.kappa;
  const double ph = fma(d, c.K, c.b);
  PairPath p;
  p.cell = rint(u);
  p.x = static_cast<float>(u - p.cell);
  p.e = cis_cycles_fast(static_cast<float>(ph - rint(ph)));
  return p;
}

// Gradients before the division by the point count, from the pair's two sums
//   sum_re = sum_n (g_r cos + g_i sin),   f = -sum_n w_n (g_i cos - g_r sin):
// *g_sigma is set, gn and gp are added to.
template <bool WITH_POINTS>
__device__ __forceinline__ void pair_gradients(const PairGeom& g, float sum_re, float f, float sigma, const float* nrm,
                                               float* g_sigma, float* gn, float* gp) {
  const float atten = 1.0f / sq(g.dist);
  *g_sigma = atten * g.align * sum_re;
  const float scale = sigma * atten;
  const float nu = dot3(nrm, g.u);
#pragma unroll
  for (int k = 0; k < 3; ++k) gn[k] = fmaf(-2.0f * scale * sum_re, fmaf(nu, g.inc[k], g.idn * g.u[k]), gn[k]);
  if (WITH_POINTS) {
    const float amp = scale * g.align;
    const float d_dist = -2.0f * amp / g.dist * sum_re - amp * f / kSpeedOfLight;
    float v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = fmaf(-2.0f * nu, nrm[k], g.u[k]);
    const float iv = dot3(g.inc, v);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      // d rho / d p, and the change of the path length
      const float drho = (v[k] - g.inc[k] * iv) * g.inv_t - (g.refl[k] - g.ret[k] * g.align) * g.inv_r;
      gp[k] += fmaf(scale * sum_re, drho, d_dist * (g.inc[k] - g.ret[k]));
    }
  }
}

// The pair's two sums from the six coefficients c0, c1, c2 of its cell.
__device__ __forceinline__ float2 cell_sums(const AdjConsts& c, const PairPath& path, float4 c0, float4 c1, float4 c2) {
  const float2 xx = make_float2(path.x, path.x);
  const float2 e = path.e;
  // the polynomial and its derivative by Horner
  float2 pv = make_float2(c2.z, c2.w), dv = pv;
  pv = ffma2(pv, xx, make_float2(c2.x, c2.y));
  dv = ffma2(dv, xx, pv);
  pv = ffma2(pv, xx, make_float2(c1.z, c1.w));
  dv = ffma2(dv, xx, pv);
  pv = ffma2(pv, xx, make_float2(c1.x, c1.y));
  dv = ffma2(dv, xx, pv);
  pv = ffma2(pv, xx, make_float2(c0.z, c0.w));
  dv = ffma2(dv, xx, pv);
  pv = ffma2(pv, xx, make_float2(c0.x, c0.y));
  return make_float2(fmaf(e.x, pv.x, e.y * pv.y),
                     c.w_mid * fmaf(e.y, pv.x, -e.x * pv.y) - c.kappa_c * fmaf(e.x, dv.x, e.y * dv.y));
}

}  // namespace tracer
}  // namespace geraf
