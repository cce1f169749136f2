// Lensless specular signal tracer (RFSignalTracer) and along-ray resampler
// kernels for sm_100a.
//
// Forward  x[a,n] = (1/P) sum_p amp(a,p) exp(+j (w0 + w1 t_n) tau(a,p))          (sample-major)
// Adjoint  dL/dsigma[a,p], dL/dnormal[p], dL/dpoint[p]                             (point-major)
// amp = sigma[a,p] rho / D^2, rho = <normalize(rx-p), normalize(i - 2(i.n)n)>,
// i = normalize(p - tx), culled when rho < 1e-6 or i.n > 0, D = |tx-p| + |rx-p|,
// tau = (D + 0.15)/2.9979, w0 = 2 pi f0, w1 = 2 pi As
// (reference: geraf/ops/RFSignalTracer/csrc/signal_tracer/SignalTracer_cuda_kernel.cu:19-197, 351-587).
//
// The reference recomputes the specular geometry for every (point, antenna,
// sample) triple.  Here the geometry is formed once per (point, antenna) and the
// sample loop works on (amplitude, delay) only.  PLAIN forms keep the reference's
// FP32 order of operations, so that amplitudes and culling decisions are bit-identical, and
// evaluate its per-sample phase with accurate cosf/sinf in its summation order.  MIXED forms
// decide culling to the same bit (pair_geometry), reduce the carrier phase in FP64
// and sum the samples through range cells: the forward collects the points'
// moments per cell of path length (tracer_cells.cuh), the adjoint reads tables of
// the residual's sum (tracer_adjoint_cells.cu).  The adjoint of this file, a Horner
// recurrence over the samples, serves the calls that the tables do not; either also
// yields the position gradient the reference does not provide.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "tracer_cells.cuh"
#include "tracer_geometry.cuh"

namespace geraf {
namespace {

using namespace tracer;

// ---------------------------------------------------------------------------
template <typename T>
struct TrP {
  const T* normals;
  const T* sigmas;
  const T* points;
  const T* tx;
  const T* rx;
  const uint8_t* inb;
  T* out_r;
  T* out_i;
  const T* gr;
  const T* gi;
  T* g_normals;
  T* g_sigmas;
  T* g_points;
  float* partial;  // adjoint: [splits][P][6]
  int* status;
  int64_t A, S, P;
  float fs, f0, As;
  double k0, b0, k1, b1;
  int splits;
  int64_t per_split;  // antennas per split
  int rows, ld, bulk;  // adjoint: antenna stage
  size_t pos_off, buf_off;
  size_t cnt_off, list_off, contrib_off;  // MIXED adjoint: per-tile work lists
  // MIXED: the points left by the per-point pre-cull (tracer_precull.cu), in
  // ascending order, and their number (device); null: every point is visited
  const int* plist;
  const int* plist_count;
  const int* run_if;  // MIXED adjoint: when set, the kernel runs only if *run_if != 0
};

template <typename T>
__device__ __forceinline__ void load3(const T* base, int64_t i, float* out) {
  out[0] = ld_f(base, i * 3 + 0);
  out[1] = ld_f(base, i * 3 + 1);
  out[2] = ld_f(base, i * 3 + 2);
}

// PLAIN forward: block = (sample block, antenna).  Per point tile, the
// (amplitude, delay) of each point is formed once in shared memory; each
// thread then accumulates its sample over the tile in point order, with the
// reference's phase expression and accurate cosf/sinf
// (SignalTracer_cuda_kernel.cu:375-449).
template <typename T>
__global__ void __launch_bounds__(128) tracer_fwd_plain_kernel(const TrP<T> p) {
  constexpr int TILE = 256;
  __shared__ float s_amp[TILE], s_tau[TILE];
  __shared__ int s_valid[TILE];
  const int64_t a = blockIdx.x;
  const int64_t n = static_cast<int64_t>(blockIdx.y) * blockDim.x + threadIdx.x;
  const bool active = n < p.S;
  float txp[3], rxp[3];
  load3(p.tx, a, txp);
  load3(p.rx, a, rxp);
  const float sample_time = static_cast<float>(n) / p.fs;
  const float w = phase_rate(p.f0, p.As, sample_time);
  float acc_r = 0.0f, acc_i = 0.0f;
  for (int64_t p0 = 0; p0 < p.P; p0 += TILE) {
    const int count = static_cast<int>(min(static_cast<int64_t>(TILE), p.P - p0));
    for (int i = threadIdx.x; i < count; i += blockDim.x) {
      const int64_t pi = p0 + i;
      int valid = 0;
      float amp = 0.0f, tau = 0.0f;
      if (p.inb[pi]) {
        float nrm[3], pt[3];
        load3(p.normals, pi, nrm);
        load3(p.points, pi, pt);
        SpecGeom g;
        specular_geometry(txp, rxp, nrm, pt, g);
        if (!culled(g)) {
          float propagation_distance = path_distance(txp, rxp, pt);
          amp = ld_f(p.sigmas, a * p.P + pi) * g.align / sq(propagation_distance);
          propagation_distance += kPathBias;
          tau = propagation_distance / kSpeedOfLight;
          valid = 1;
        }
      }
      s_valid[i] = valid;
      s_amp[i] = amp;
      s_tau[i] = tau;
    }
    __syncthreads();
    if (active) {
      for (int i = 0; i < count; ++i) {
        if (!s_valid[i]) continue;
        const float phase = __fmul_rn(w, s_tau[i]);
        float c, sn;
        cos_sin(phase, &c, &sn);
        acc_r += s_amp[i] * c;
        acc_i += s_amp[i] * sn;
      }
    }
    __syncthreads();
  }
  if (active) {
    const int total_point_size = static_cast<int>(p.P);
    p.out_r[a * p.S + n] = from_f<T>(acc_r / total_point_size);
    p.out_i[a * p.S + n] = from_f<T>(acc_i / total_point_size);
  }
}

// MIXED forward.  Block = (antenna, point split): the points of the split (of the
// pre-cull's list) into the moments of their cells (tracer_cells.cuh).  64 antennas x
// 524288 points (10% listed, 8% of the pairs live) x 128 samples: 119 us against 181 us
// with a recurrence over the samples of every live pair.
template <typename T>
struct TrCellP {
  const T* normals;
  const T* sigmas;
  const T* points;
  const T* tx;
  const T* rx;
  const uint8_t* inb;
  T* out_r;
  T* out_i;
  const int* plist;
  const int* plist_count;
  TraceRecord* records;  // [A][splits]
  float2* rows;          // [A][splits][S]
  int64_t A, P;
  int splits;
  TraceConsts c;
};

// Positions [begin, end) of share b.
template <typename T>
__device__ __forceinline__ void share_range(const TrCellP<T>& p, int64_t b, int64_t& begin, int64_t& end) {
  const int64_t npts = p.plist != nullptr ? static_cast<int64_t>(*p.plist_count) : p.P;
  const int64_t per_split = (npts + p.splits - 1) / p.splits;
  begin = b % p.splits * per_split;
  end = min(npts, begin + per_split);
}

// Positions [begin, end) of share b (not inlined: it would take registers from the cells).
template <typename T>
static __device__ __noinline__ void share_direct(DirectSmem& sm, const TrCellP<T>& p, int64_t b, int64_t begin, int64_t end) {
  const int64_t a = b / p.splits;
  float txp[3], rxp[3];
  load3(p.tx, a, txp);
  load3(p.rx, a, rxp);
  const T* sigmas = p.sigmas + a * p.P;
  const int* plist = p.plist;
  const uint8_t* inb = p.inb;
  float2* row = p.rows + b * p.c.S;
  trace_direct<T>(
      sm, p.c, p.normals, p.points, txp, rxp, end - begin,
      [&](int64_t pos) -> int64_t { return plist != nullptr ? plist[begin + pos] : inb[begin + pos] ? begin + pos : -1; },
      [&](int64_t q) { return ld_f(sigmas, q); }, [&](int n, float2 y) { row[n] = y; });
}

template <typename T>
__global__ void __launch_bounds__(kTraceThreads, 5) tracer_fwd_cells_kernel(const __grid_constant__ TrCellP<T> p) {
  __shared__ union {
    TraceSmem cells;
    DirectSmem direct;
  } smem;
  TraceSmem& sm = smem.cells;
  const int64_t a = blockIdx.x / p.splits;
  int64_t begin, end;
  share_range(p, blockIdx.x, begin, end);
  float txp[3], rxp[3];
  load3(p.tx, a, txp);
  load3(p.rx, a, rxp);
  trace_begin(sm);
  const int64_t from = begin + trace_all<T>(
      sm, p.c, p.normals, p.points, txp, rxp, static_cast<int>(max(int64_t{0}, end - begin)),
      [&](int64_t pos) -> int64_t {
        return p.plist != nullptr ? p.plist[begin + pos] : p.inb[begin + pos] ? begin + pos : -1;
      },
      [&](int64_t q) { return ld_f(p.sigmas, a * p.P + q); });
  trace_store(sm, p.records + blockIdx.x, from < end);
  if (from < end) share_direct(smem.direct, p, blockIdx.x, from, end);
}

// Many antennas of up to kDirectPoints points: a block per antenna, without cells.
template <typename T>
__global__ void __launch_bounds__(kTraceThreads) tracer_fwd_short_kernel(const __grid_constant__ TrCellP<T> p) {
  __shared__ DirectSmem sm;
  const int64_t a = blockIdx.x;
  const int64_t count = p.plist != nullptr ? static_cast<int64_t>(*p.plist_count) : p.P;
  float txp[3], rxp[3];
  load3(p.tx, a, txp);
  load3(p.rx, a, rxp);
  const float divisor = static_cast<float>(p.P);
  trace_direct<T>(
      sm, p.c, p.normals, p.points, txp, rxp, count,
      [&](int64_t pos) -> int64_t { return p.plist != nullptr ? p.plist[pos] : p.inb[pos] ? pos : -1; },
      [&](int64_t q) { return ld_f(p.sigmas, a * p.P + q); },
      [&](int n, float2 y) {
        p.out_r[a * p.c.S + n] = from_f<T>(y.x / divisor);
        p.out_i[a * p.c.S + n] = from_f<T>(y.y / divisor);
      });
}

template <typename T>
__global__ void __launch_bounds__(kFinishThreads) tracer_fwd_finish_kernel(const TrCellP<T> p) {
  const int64_t a = blockIdx.x;
  const int n0 = blockIdx.y * kFinishSamples;
  trace_finish<T>(p.c, p.records + a * p.splits, p.rows + a * p.splits * p.c.S, p.splits, static_cast<float>(p.P), n0,
                  min(p.c.S, n0 + kFinishSamples), p.out_r + a * p.c.S, p.out_i + a * p.c.S);
}

template <typename T>
__global__ void __launch_bounds__(kFewThreads) tracer_fwd_finish_few_kernel(const TrCellP<T> p) {
  extern __shared__ __align__(16) unsigned char few_smem[];
  const FewTable f = few_table(p.c, few_smem);
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (kFewThreads / 32);
  for (int64_t a = blockIdx.x * static_cast<int64_t>(kFewThreads / 32) + (threadIdx.x >> 5); a < p.A; a += warps) {
    trace_finish_few<T>(p.c, f, p.records + a * p.splits, p.rows + a * p.splits * p.c.S, p.splits,
                        static_cast<float>(p.P), p.out_r + a * p.c.S, p.out_i + a * p.c.S);
  }
}

// ---------------------------------------------------------------------------
// Adjoint (point-major).  Block = point tile x antenna split; the residual
// rows g[a, :] stream through a double-buffered TMA ring.
struct AdjSmem {
  size_t pos_off, buf_off, total;
};

template <typename T>
AdjSmem adj_smem_layout(int rows, int ld) {
  AdjSmem s;
  s.pos_off = 128;
  size_t off = s.pos_off + 2 * static_cast<size_t>(rows) * 6 * sizeof(float);
  off = (off + 127) & ~static_cast<size_t>(127);
  s.buf_off = off;
  off += 4 * static_cast<size_t>(rows) * ld * sizeof(T);
  s.total = (off + 127) & ~static_cast<size_t>(127);
  return s;
}

// MIXED adjoint: the staged ring as above, then per-tile work lists -- live
// (point, antenna) counts [rows], their point slots [rows][threads] and the
// per-point gradient contributions [rows][nc][threads].
struct AdjMixedSmem {
  size_t pos_off, buf_off, cnt_off, list_off, contrib_off, total;
};

template <typename T>
AdjMixedSmem adj_mixed_smem_layout(int rows, int ld, int threads, int nc) {
  const AdjSmem base = adj_smem_layout<T>(rows, ld);
  AdjMixedSmem s;
  s.pos_off = base.pos_off;
  s.buf_off = base.buf_off;
  size_t off = base.total;
  s.cnt_off = off;
  off += (static_cast<size_t>(rows) * sizeof(int) + 127) & ~static_cast<size_t>(127);
  s.list_off = off;
  off += (static_cast<size_t>(rows) * threads * sizeof(int) + 127) & ~static_cast<size_t>(127);
  s.contrib_off = off;
  off += static_cast<size_t>(rows) * nc * threads * sizeof(float);
  s.total = (off + 127) & ~static_cast<size_t>(127);
  return s;
}

template <typename T>
__device__ __forceinline__ void stage_positions_f(float* pos, int stage, int rows_max, const T* tx,
                                                  const T* rx, int64_t a0, int rws) {
  for (int i = threadIdx.x; i < rws * 6; i += blockDim.x) {
    const int r = i / 6;
    const int c = i - r * 6;
    const T* src = c < 3 ? tx : rx;
    pos[(stage * rows_max + r) * 6 + c] = ld_f(src, (a0 + r) * 3 + (c % 3));
  }
}

// Writes one point's accumulated normal / position gradients (or partials).
template <typename T>
__device__ __forceinline__ void store_point_grads(const TrP<T>& p, int split, int64_t pi,
                                                  const float* gn, const float* gp, bool with_points) {
  if (p.splits == 1) {
    const int total_point_size = static_cast<int>(p.P);
#pragma unroll
    for (int k = 0; k < 3; ++k) p.g_normals[pi * 3 + k] = from_f<T>(gn[k] / total_point_size);
    if (with_points) {
#pragma unroll
      for (int k = 0; k < 3; ++k) p.g_points[pi * 3 + k] = from_f<T>(gp[k] / total_point_size);
    }
  } else {
    float* dst = p.partial + (split * p.P + pi) * 6;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      dst[k] = gn[k];
      dst[3 + k] = with_points ? gp[k] : 0.0f;
    }
  }
}

// PLAIN adjoint: thread = point, antennas and samples in the reference's order
// (SignalTracer_cuda_kernel.cu:491-586).  With grad_points requested, the delay
// derivative sum_n w_n (g_i cos - g_r sin) is accumulated alongside.
template <typename T, bool WITH_POINTS>
__global__ void __launch_bounds__(128) tracer_bwd_plain_kernel(const TrP<T> p) {
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
  float* pos = reinterpret_cast<float*>(smem + p.pos_off);
  PairStager<T> stg{reinterpret_cast<T*>(smem + p.buf_off), bar, p.ld, p.rows, p.bulk != 0};

  const int split = blockIdx.x % p.splits;
  const int64_t ptile = blockIdx.x / p.splits;
  const int64_t pi = ptile * blockDim.x + threadIdx.x;
  const int64_t a_begin = static_cast<int64_t>(split) * p.per_split;
  const int64_t a_end = min(p.A, a_begin + p.per_split);
  const int ntiles = a_end > a_begin ? ceil_div(a_end - a_begin, p.rows) : 0;
  const int S = static_cast<int>(p.S);
  const bool inside = pi < p.P;
  const bool active = inside && p.inb[pi];

  if (p.bulk && threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_barrier_init();
  }
  __syncthreads();

  float nrm[3] = {0.0f, 0.0f, 0.0f}, pt[3] = {0.0f, 0.0f, 0.0f};
  if (active) {
    load3(p.normals, pi, nrm);
    load3(p.points, pi, pt);
  }
  float accum_grad_normal[3] = {0.0f, 0.0f, 0.0f};
  float accum_grad_point[3] = {0.0f, 0.0f, 0.0f};

  auto issue = [&](int tile, int stage) {
    const int64_t a0 = a_begin + static_cast<int64_t>(tile) * p.rows;
    const int rws = static_cast<int>(min(static_cast<int64_t>(p.rows), a_end - a0));
    stg.issue(stage, p.gr, p.gi, a0, rws, S);
    stage_positions_f<T>(pos, stage, p.rows, p.tx, p.rx, a0, rws);
  };
  if (ntiles > 0) issue(0, 0);
  if (ntiles > 1) issue(1, 1);

  for (int t = 0; t < ntiles; ++t) {
    const int s = t & 1;
    if (!stg.wait(s, (t >> 1) & 1, p.status)) {
      if (t + 1 < ntiles) stg.drain(s ^ 1, ((t + 1) >> 1) & 1, p.status);
      return;
    }
    const int64_t a0 = a_begin + static_cast<int64_t>(t) * p.rows;
    const int rws = static_cast<int>(min(static_cast<int64_t>(p.rows), a_end - a0));
    for (int r = 0; r < rws && inside; ++r) {
      const int64_t a = a0 + r;
      if (!active) {
        p.g_sigmas[a * p.P + pi] = from_f<T>(0.0f);
        continue;
      }
      const float* ps = pos + (s * p.rows + r) * 6;
      const float txp[3] = {ps[0], ps[1], ps[2]};
      const float rxp[3] = {ps[3], ps[4], ps[5]};
      SpecGeom g;
      specular_geometry(txp, rxp, nrm, pt, g);
      if (culled(g)) {
        p.g_sigmas[a * p.P + pi] = from_f<T>(0.0f);
        continue;
      }
      float gsa[3];
      align_normal_gradient(g, nrm, gsa);
      float propagation_distance = path_distance(txp, rxp, pt);
      const float propagation_attenuation = 1.0f / sq(propagation_distance);
      const float sigma_value = ld_f(p.sigmas, a * p.P + pi);
      const float dist_path = propagation_distance;
      propagation_distance += kPathBias;
      const float tau = propagation_distance / kSpeedOfLight;
      const T* rowr = stg.stage_ptr(s, 0) + r * p.ld;
      const T* rowi = stg.stage_ptr(s, 1) + r * p.ld;
      float accum_grad_sigma = 0.0f;
      float accum_raw = 0.0f;
      float accum_tau = 0.0f;
      for (int n = 0; n < S; ++n) {
        const float sample_time = static_cast<float>(n) / p.fs;
        const float omega = adjoint_phase_rate<T>(p.f0, p.As, sample_time);
        const float phase = __fmul_rn(omega, tau);
        float phase_real, phase_imag;
        cos_sin(phase, &phase_real, &phase_imag);
        const float gro = static_cast<float>(rowr[n]);
        const float gio = static_cast<float>(rowi[n]);
        const float grad_real = gro * phase_real;
        const float grad_imag = gio * phase_imag;
        const float normal_scale = sigma_value * propagation_attenuation;
        accum_grad_normal[0] += normal_scale * gsa[0] * (grad_real + grad_imag);
        accum_grad_normal[1] += normal_scale * gsa[1] * (grad_real + grad_imag);
        accum_grad_normal[2] += normal_scale * gsa[2] * (grad_real + grad_imag);
        accum_grad_sigma += propagation_attenuation * g.align * (grad_real + grad_imag);
        if (WITH_POINTS) {
          accum_raw += grad_real + grad_imag;
          accum_tau += omega * (gio * phase_real - gro * phase_imag);
        }
      }
      p.g_sigmas[a * p.P + pi] = from_f<T>(accum_grad_sigma / static_cast<int>(p.P));
      if (WITH_POINTS) {
        // dL/dp = dL/damp * damp/dp + dL/dtau * dtau/dp (before the 1/P factor)
        const float amp = sigma_value * g.align * propagation_attenuation;
        const float d_amp = accum_raw;
        const float dist_t = sqrtf(sq(txp[0] - pt[0]) + sq(txp[1] - pt[1]) + sq(txp[2] - pt[2]));
        const float dist_r = sqrtf(sq(rxp[0] - pt[0]) + sq(rxp[1] - pt[1]) + sq(rxp[2] - pt[2]));
        float drho[3];
        align_point_gradient(g, nrm, dist_t, dist_r, drho);
        const float d_tau = amp * accum_tau;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float dD = g.inc[k] - g.ret[k];
          const float damp_dp =
              sigma_value * propagation_attenuation * drho[k] - 2.0f * amp / dist_path * dD;
          accum_grad_point[k] += d_amp * damp_dp + d_tau * dD / kSpeedOfLight;
        }
      }
    }
    __syncthreads();
    if (t + 2 < ntiles) issue(t + 2, s);
  }
  if (inside) store_point_grads(p, split, pi, accum_grad_normal, accum_grad_point, WITH_POINTS);
}

// MIXED adjoint: a block owns blockDim points (one per thread) and streams
// antenna rows of the residual through a TMA ring.  Per (point, antenna) the
// residual polynomial Q(zeta) = sum_n conj(g[a,n]) zeta^n is evaluated by
// Horner in zeta^2 on the even and odd samples in the two lanes of packed
// f32x2 operations (2 instructions per sample) and, for position gradients,
// Q1 = sum_n n conj(g) zeta^n alongside (2 more).
//
// Culled pairs (back-facing or grazing, rho < 1e-6) skip all of that, so per
// stage the block first lists the (point, antenna) pairs that the early test
// cannot cull and then deals them out evenly over all threads, which form each
// pair's exact geometry once: no lane idles beside a lane that works.
// Each pair's normal / position contributions land in shared memory, and the
// point's owner thread adds them up in antenna order -- the same sums, in the
// same order, as one thread walking its point's antennas.  Six blocks are kept
// resident per SM (80 registers): 1-6% faster than the five that 93
// registers allowed, measured on 64 antennas x 524288 points x 128 samples and
// 128 antennas x 262144 points x 256 samples.
template <typename T, bool WITH_POINTS>
__global__ void __launch_bounds__(128, sizeof(T) == 8 ? 4 : 6) tracer_bwd_mixed_kernel(const TrP<T> p) {
  constexpr int NC = WITH_POINTS ? 6 : 3;
  extern __shared__ __align__(128) unsigned char smem[];
  if (p.run_if != nullptr && *p.run_if == 0) return;
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem);
  float* pos = reinterpret_cast<float*>(smem + p.pos_off);
  int* cnt = reinterpret_cast<int*>(smem + p.cnt_off);           // [rows]
  int* list = reinterpret_cast<int*>(smem + p.list_off);         // [rows][TILE]
  float* contrib = reinterpret_cast<float*>(smem + p.contrib_off);  // [rows][NC][TILE]
  PairStager<T> stg{reinterpret_cast<T*>(smem + p.buf_off), bar, p.ld, p.rows, p.bulk != 0};

  const int TILE = blockDim.x;
  // The number of listed points is on the device only: the blocks take the tiles of
  // points (times splits) in turn.  Thread t owns point position k = ptile * TILE + t:
  // listed point list[k], or point k when every point is visited.
  const int64_t npts = p.plist != nullptr ? static_cast<int64_t>(*p.plist_count) : p.P;
  const int64_t tiles = (npts + TILE - 1) / TILE * p.splits;
  if (p.bulk && threadIdx.x == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_barrier_init();
  }
  __syncthreads();
  int used = 0;  // stages the ring has carried: the phases of its barriers go on from tile to tile
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int split = static_cast<int>(tile % p.splits);
    const int64_t p_base = tile / p.splits * TILE;
    const int64_t k_own = p_base + threadIdx.x;
    const bool inside = k_own < npts;
    const int64_t pi = !inside ? 0 : p.plist != nullptr ? static_cast<int64_t>(p.plist[k_own]) : k_own;
    const int64_t a_begin = static_cast<int64_t>(split) * p.per_split;
    const int64_t a_end = min(p.A, a_begin + p.per_split);
    const int ntiles = a_end > a_begin ? ceil_div(a_end - a_begin, p.rows) : 0;
    const bool active = inside && (p.plist != nullptr || p.inb[pi]);

    float own_nrm[3] = {0.0f, 0.0f, 1.0f}, own_pt[3] = {0.0f, 0.0f, 0.0f};
    if (active) {
      load3(p.normals, pi, own_nrm);
      load3(p.points, pi, own_pt);
    }
    // w0 and w1/fs in rad per unit delay, as exact FP64 products of the FP32 constants.
    const float w0 = static_cast<float>(2.0 * static_cast<double>(kPiF) * p.f0);
    const float w1s = static_cast<float>(2.0 * static_cast<double>(kPiF) * p.As / p.fs);
    float gnorm[3] = {0.0f, 0.0f, 0.0f};
    float gpt[3] = {0.0f, 0.0f, 0.0f};

    auto issue = [&](int tile, int stage) {
      const int64_t a0 = a_begin + static_cast<int64_t>(tile) * p.rows;
      const int rws = static_cast<int>(min(static_cast<int64_t>(p.rows), a_end - a0));
      stg.issue(stage, p.gr, p.gi, a0, rws, static_cast<int>(p.S));
      stage_positions_f<T>(pos, stage, p.rows, p.tx, p.rx, a0, rws);
    };
    if (ntiles > 0) issue(0, used & 1);
    if (ntiles > 1) issue(1, (used + 1) & 1);

    for (int t = 0; t < ntiles; ++t) {
      const int s = (used + t) & 1;
      for (int r = threadIdx.x; r < p.rows; r += TILE) cnt[r] = 0;
      if (!stg.wait(s, ((used + t) >> 1) & 1, p.status)) {  // (its barrier also publishes cnt)
        if (t + 1 < ntiles) stg.drain(s ^ 1, ((used + t + 1) >> 1) & 1, p.status);
        return;
      }
      const int64_t a0 = a_begin + static_cast<int64_t>(t) * p.rows;
      const int rws = static_cast<int>(min(static_cast<int64_t>(p.rows), a_end - a0));

      // 1. list the stage's candidate pairs, those the early test cannot cull (the
      //    exact geometry, formed once in step 2, decides them); the other pairs get
      //    zero gradients here
      for (int r = 0; r < rws; ++r) {
        if (!inside) break;
        const float* ps = pos + (s * p.rows + r) * 6;
        const float txp[3] = {ps[0], ps[1], ps[2]};
        const float rxp[3] = {ps[3], ps[4], ps[5]};
        const bool live = active && !surely_culled(txp, rxp, own_nrm, own_pt);
        if (live) {
          list[r * TILE + atomicAdd(&cnt[r], 1)] = threadIdx.x;
        } else {
          p.g_sigmas[(a0 + r) * p.P + pi] = from_f<T>(0.0f);
  #pragma unroll
          for (int k = 0; k < NC; ++k) contrib[(r * NC + k) * TILE + threadIdx.x] = 0.0f;
        }
      }
      __syncthreads();

      // 2. every thread takes candidate pairs k = tid, tid + TILE, ... in (row, list) order
      int total = 0;
      for (int r = 0; r < rws; ++r) total += cnt[r];
      int r_cur = 0, r_start = 0;
      for (int k = threadIdx.x; k < total; k += TILE) {
        while (k >= r_start + cnt[r_cur]) {
          r_start += cnt[r_cur];
          ++r_cur;
        }
        const int r = r_cur;
        const int slot = list[r * TILE + (k - r_start)];
        const int64_t pj = p.plist != nullptr ? static_cast<int64_t>(p.plist[p_base + slot]) : p_base + slot;
        const int64_t a = a0 + r;
        float nrm[3], pt[3];
        load3(p.normals, pj, nrm);
        load3(p.points, pj, pt);
        const float* ps = pos + (s * p.rows + r) * 6;
        const float txp[3] = {ps[0], ps[1], ps[2]};
        const float rxp[3] = {ps[3], ps[4], ps[5]};
        SpecGeom geo;
        specular_geometry(txp, rxp, nrm, pt, geo);
        if (culled(geo)) {
          p.g_sigmas[a * p.P + pj] = from_f<T>(0.0f);
  #pragma unroll
          for (int c = 0; c < NC; ++c) contrib[(r * NC + c) * TILE + slot] = 0.0f;
          continue;
        }
        const double px = pt[0], py = pt[1], pz = pt[2];
        const PhaseCycles pc = path_cycles(ps[0] - px, ps[1] - py, ps[2] - pz, ps[3] - px,
                                           ps[4] - py, ps[5] - pz, p.k0, p.b0, p.k1, p.b1);
        const float2 zt = cis_cycles(pc.dcyc);
        const T* rowr = stg.stage_ptr(s, 0) + r * p.ld;
        const T* rowi = stg.stage_ptr(s, 1) + r * p.ld;
        float2 qv, q1;  // Q and Q1 = zeta Q'(zeta): packed even/odd Horner in zeta^2
        residual_sums<WITH_POINTS>(rowr, rowi, p.ld, zt, qv, q1);
        const float qr = qv.x, qi = qv.y;
        const float2 e0 = cis_cycles_fast(pc.frac0);
        const float2 eq = cmul(e0, make_float2(qr, qi));
        // sum_n (g_r cos + g_i sin) = Re(exp(j phi0) Q)
        const float sum_re = eq.x;
        const float propagation_distance = path_distance(txp, rxp, pt);
        const float propagation_attenuation = 1.0f / sq(propagation_distance);
        const float sigma_value = ld_f(p.sigmas, a * p.P + pj);
        p.g_sigmas[a * p.P + pj] =
            from_f<T>(propagation_attenuation * geo.align * sum_re / static_cast<float>(p.P));
        float gsa[3];
        align_normal_gradient(geo, nrm, gsa);
        const float normal_scale = sigma_value * propagation_attenuation;
  #pragma unroll
        for (int c = 0; c < 3; ++c) contrib[(r * NC + c) * TILE + slot] = normal_scale * gsa[c] * sum_re;
        if (WITH_POINTS) {
          // sum_n w_n (g_i cos - g_r sin) = -Im(exp(j phi0) (w0 Q + w1s Q1))
          const float2 f = cmul(e0, make_float2(w0 * qr + w1s * q1.x, w0 * qi + w1s * q1.y));
          const float amp = sigma_value * geo.align * propagation_attenuation;
          const float d_tau = -amp * f.y;
          const float dist_t = sqrtf(sq(txp[0] - pt[0]) + sq(txp[1] - pt[1]) + sq(txp[2] - pt[2]));
          const float dist_r = sqrtf(sq(rxp[0] - pt[0]) + sq(rxp[1] - pt[1]) + sq(rxp[2] - pt[2]));
          float drho[3];
          align_point_gradient(geo, nrm, dist_t, dist_r, drho);
  #pragma unroll
          for (int c = 0; c < 3; ++c) {
            const float dD = geo.inc[c] - geo.ret[c];
            const float damp_dp =
                normal_scale * drho[c] - 2.0f * amp / propagation_distance * dD;
            contrib[(r * NC + 3 + c) * TILE + slot] = sum_re * damp_dp + d_tau * dD / kSpeedOfLight;
          }
        }
      }
      __syncthreads();

      // 3. each owner adds its point's contributions in antenna order
      if (inside) {
        for (int r = 0; r < rws; ++r) {
  #pragma unroll
          for (int c = 0; c < 3; ++c) gnorm[c] += contrib[(r * NC + c) * TILE + threadIdx.x];
          if (WITH_POINTS) {
  #pragma unroll
            for (int c = 0; c < 3; ++c) gpt[c] += contrib[(r * NC + 3 + c) * TILE + threadIdx.x];
          }
        }
      }
      __syncthreads();
      if (t + 2 < ntiles) issue(t + 2, s);
    }
    used += ntiles;
    if (inside) store_point_grads(p, split, pi, gnorm, gpt, WITH_POINTS);
  }
}

// With a point list, only the listed points' partials are summed (the others'
// gradients were zeroed by the pre-cull).
template <typename T>
__global__ void tracer_bwd_finalize_kernel(const float* __restrict__ partial, int splits, int64_t P,
                                           T* g_normals, T* g_points, const int* plist,
                                           const int* plist_count) {
  const int64_t count = plist != nullptr ? static_cast<int64_t>(*plist_count) : P;
  for (int64_t k = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; k < count;
       k += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t i = plist != nullptr ? static_cast<int64_t>(plist[k]) : k;
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int s = 0; s < splits; ++s) {
      const float* src = partial + (s * P + i) * 6;
      for (int k = 0; k < 6; ++k) acc[k] += src[k];
    }
    const float inv = static_cast<float>(P);
    for (int k = 0; k < 3; ++k) g_normals[i * 3 + k] = from_f<T>(static_cast<float>(acc[k]) / inv);
    if (g_points != nullptr) {
      for (int k = 0; k < 3; ++k) g_points[i * 3 + k] = from_f<T>(static_cast<float>(acc[3 + k]) / inv);
    }
  }
}

// ---------------------------------------------------------------------------
// Along-ray linear resampler (SignalTracer_cuda_kernel.cu:199-349).  One warp
// per ray: the bracketing index and weights of every target depth are found
// once per ray (binary search over the ray's coarse depths) and reused for all
// A sigma rows; arithmetic is in the element type, as in the reference.
template <typename T>
struct BiP {
  const T* normals;
  const T* sigmas;
  const T* z;
  const T* tz;
  T* out_n;
  T* out_s;
  uint8_t* out_inb;
  int64_t A, R, S, T_;
};

template <typename T>
__device__ __forceinline__ int bracket_lower(const T* z, int S, T target) {
  int lower_index = 0;
  int upper_index = S - 1;
  while (lower_index < upper_index - 1) {
    const int mid_index = (lower_index + upper_index) / 2;
    if (z[mid_index] <= target) lower_index = mid_index;
    else upper_index = mid_index;
  }
  return lower_index;
}

template <typename T>
__device__ __forceinline__ T tmax(T a, T b) { return a > b ? a : b; }

// acc + w * g with the product rounded before the sum (never fused), as an
// atomicAdd of a precomputed product does in the reference.
__device__ __forceinline__ float add_product(float acc, float w, float g) {
  return __fadd_rn(acc, __fmul_rn(w, g));
}
__device__ __forceinline__ double add_product(double acc, double w, double g) {
  return __dadd_rn(acc, __dmul_rn(w, g));
}

template <typename T>
__global__ void __launch_bounds__(256) bilinear_fwd_kernel(const BiP<T> p) {
  const int64_t ray = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (ray >= p.R) return;
  const int S = static_cast<int>(p.S);
  const T* z = p.z + ray * p.S;
  const T* nrm = p.normals + ray * p.S * 3;
  for (int64_t t = lane; t < p.T_; t += 32) {
    const T target = p.tz[ray * p.T_ + t];
    const int lo = bracket_lower(z, S, target);
    const T z0 = z[lo];
    const T z1 = z[lo + 1];
    const bool oob = (target < z0) || (target > z1);
    p.out_inb[ray * p.T_ + t] = oob ? 0 : 1;
    T* on = p.out_n + (ray * p.T_ + t) * 3;
    if (oob) {
      on[0] = T(0.0f);
      on[1] = T(0.0f);
      on[2] = T(0.0f);
      for (int64_t a = 0; a < p.A; ++a) p.out_s[(a * p.R + ray) * p.T_ + t] = T(0.0f);
      continue;
    }
    const T weight_upper = (target - z0) / tmax(z1 - z0, static_cast<T>(1.0e-6f));
    const T weight_lower = static_cast<T>(1) - weight_upper;
    for (int axis = 0; axis < 3; ++axis) {
      const T normal_lower = nrm[lo * 3 + axis];
      const T normal_upper = nrm[(lo + 1) * 3 + axis];
      on[axis] = weight_lower * normal_lower + weight_upper * normal_upper;
    }
    for (int64_t a = 0; a < p.A; ++a) {
      const T* sg = p.sigmas + (a * p.R + ray) * p.S;
      p.out_s[(a * p.R + ray) * p.T_ + t] = weight_lower * sg[lo] + weight_upper * sg[lo + 1];
    }
  }
}

// Adjoint, gather form: lane j of the ray's warp owns coarse sample j and adds
// the contributions of the targets bracketing it in target order -- the same
// per-element order as the reference's single-writer atomicAdd sequence --
// onto the existing gradient value.  The brackets and weights of the ray's targets
// are found once, into shared memory; where the targets ascend (the usual case),
// those of one coarse sample are a contiguous range, found by binary search, else every
// sample scans them all.  Bound by the latency of a ray's chain, not by its bytes:
// 4096 rays x 128 samples x 128 targets took 0.86 ms when every (sample, target)
// pair searched the bracket again.
constexpr int kTargetTile = 512;  // targets held at a time; longer rows take several passes

template <typename T>
__global__ void __launch_bounds__(256) bilinear_bwd_kernel(const BiP<T> p) {
  extern __shared__ __align__(16) unsigned char bi_smem[];
  constexpr int kOut = 1 << 30;  // set in a bracket index: the target lies outside
  const int warps = blockDim.x >> 5;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int64_t ray = blockIdx.x * static_cast<int64_t>(warps) + warp;
  if (ray >= p.R) return;
  const int S = static_cast<int>(p.S);
  const int tile = static_cast<int>(min(p.T_, static_cast<int64_t>(kTargetTile)));
  T* weight = reinterpret_cast<T*>(bi_smem) + warp * tile;  // of the upper sample
  int* lower = reinterpret_cast<int*>(reinterpret_cast<T*>(bi_smem) + warps * tile) + warp * tile;
  const T* z = p.z + ray * p.S;
  for (int64_t t0 = 0; t0 < p.T_; t0 += kTargetTile) {
    const int nt = static_cast<int>(min(p.T_ - t0, static_cast<int64_t>(kTargetTile)));
    __syncwarp();
    for (int t = lane; t < nt; t += 32) {
      const T target = p.tz[ray * p.T_ + t0 + t];
      const int lo = bracket_lower(z, S, target);
      const T z0 = z[lo];
      const T z1 = z[lo + 1];
      const bool out = target < z0 || target > z1;
      weight[t] = (target - z0) / tmax(z1 - z0, static_cast<T>(1.0e-6f));
      lower[t] = lo | (out ? kOut : 0);
    }
    __syncwarp();
    bool ascending = true;
    for (int t = lane; t + 1 < nt; t += 32) ascending = ascending && (lower[t] & ~kOut) <= (lower[t + 1] & ~kOut);
    ascending = __all_sync(0xffffffffu, ascending);
    auto first_from = [&](int j) {  // the first target whose bracket is j or higher
      int lo = 0, hi = nt;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if ((lower[mid] & ~kOut) >= j) hi = mid;
        else lo = mid + 1;
      }
      return lo;
    };
    // p.normals = grad_output_normals [R,T,3], p.sigmas = grad_output_sigmas [A,R,T]
    const T* gno = p.normals + (ray * p.T_ + t0) * 3;
    for (int j = lane; j < S; j += 32) {
      const int t_begin = ascending ? first_from(j - 1) : 0;
      const int t_end = ascending ? first_from(j + 1) : nt;
      T* gn = p.out_n + (ray * p.S + j) * 3;
      T acc[3] = {gn[0], gn[1], gn[2]};
      for (int t = t_begin; t < t_end; ++t) {
        const int lo = lower[t];
        if (lo != j && lo + 1 != j) continue;
        const T w = lo == j ? static_cast<T>(1) - weight[t] : weight[t];
#pragma unroll
        for (int axis = 0; axis < 3; ++axis) acc[axis] = add_product(acc[axis], w, gno[t * 3 + axis]);
      }
#pragma unroll
      for (int axis = 0; axis < 3; ++axis) gn[axis] = acc[axis];
      for (int64_t a = 0; a < p.A; ++a) {
        const T* gso = p.sigmas + (a * p.R + ray) * p.T_ + t0;
        T* gs = p.out_s + (a * p.R + ray) * p.S + j;
        T sum = *gs;
        for (int t = t_begin; t < t_end; ++t) {
          const int lo = lower[t];
          if (lo != j && lo + 1 != j) continue;
          sum = add_product(sum, lo == j ? static_cast<T>(1) - weight[t] : weight[t], gso[t]);
        }
        *gs = sum;
      }
    }
  }
}

// ---------------------------------------------------------------------------
bool aligned16(const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; }

template <typename T>
TrP<T> make_params(const TracerArgs& a) {
  TrP<T> p;
  p.normals = static_cast<const T*>(a.normals);
  p.sigmas = static_cast<const T*>(a.sigmas);
  p.points = static_cast<const T*>(a.points);
  p.tx = static_cast<const T*>(a.tx);
  p.rx = static_cast<const T*>(a.rx);
  p.inb = a.inbounds;
  p.out_r = static_cast<T*>(a.out_real);
  p.out_i = static_cast<T*>(a.out_imag);
  p.gr = static_cast<const T*>(a.grad_real_out);
  p.gi = static_cast<const T*>(a.grad_imag_out);
  p.g_normals = static_cast<T*>(a.grad_normals);
  p.g_sigmas = static_cast<T*>(a.grad_sigmas);
  p.g_points = static_cast<T*>(a.grad_points);
  p.partial = nullptr;
  p.status = device_status_ptr();
  p.A = a.A;
  p.S = a.S;
  p.P = a.P;
  p.fs = a.fs;
  p.f0 = a.f0;
  p.As = a.As;
  const PhaseConsts pc = phase_consts(a.f0, a.As, a.fs);
  p.k0 = pc.k0;
  p.b0 = pc.b0;
  p.k1 = pc.k1;
  p.b1 = pc.b1;
  p.splits = 1;
  p.per_split = 0;
  p.rows = 1;
  p.ld = 4;
  p.bulk = 0;
  p.pos_off = p.buf_off = 0;
  p.plist = nullptr;
  p.plist_count = nullptr;
  p.run_if = nullptr;
  return p;
}

// Workspace of the MIXED forward and adjoint: the split partials, then (when the
// pre-cull applies) the point list region.
size_t list_region_offset(size_t partial_bytes) { return (partial_bytes + 255) & ~static_cast<size_t>(255); }

// Workspace of the MIXED forward: the shares' records, their rows of samples, the point list.
struct FwdLayout {
  size_t rows, list;
};
FwdLayout fwd_layout(const TracerArgs& a, int splits) {
  const size_t shares = static_cast<size_t>(splits) * a.A;
  FwdLayout l;
  l.rows = list_region_offset(shares * sizeof(TraceRecord));
  l.list = l.rows + list_region_offset(shares * a.S * sizeof(float2));
  return l;
}

}  // namespace

bool finish_by_warps(int64_t A, int64_t S, double kappa) {
  return A >= 2 * static_cast<int64_t>(current_device_info().sm_count) && S <= kFewSamples && kappa > kTraceMinKappa;
}

cudaError_t launch_few(const void* fn, void* params, int64_t A, int64_t S, cudaStream_t st) {
  const size_t smem = few_smem_bytes(S);
  const DeviceInfo dev = current_device_info();
  // blocks that registers (3) and shared memory let stay: each forms the table once
  const int64_t resident = std::min<int64_t>(3, std::max<int64_t>(1, (dev.max_smem_optin + 1024) / (smem + 1024)));
  const int64_t blocks = std::min<int64_t>((A + kFewThreads / 32 - 1) / (kFewThreads / 32), resident * dev.sm_count);
  // one limit for all sizes: other threads may be launching the kernel at theirs
  const cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(few_smem_bytes(kFewSamples)));
  if (err != cudaSuccess) return err;
  void* args[] = {params};
  return cudaLaunchKernel(fn, dim3(static_cast<unsigned>(blocks)), dim3(kFewThreads), args, smem, st);
}

namespace {

// Forward calls that tracer_fwd_short_kernel takes: two blocks per SM or more.
bool short_antennas(const TracerArgs& a) {
  return a.P <= kDirectPoints && a.A >= 2 * static_cast<int64_t>(current_device_info().sm_count);
}

template <typename T>
cudaError_t launch_tracer_fwd(const TracerArgs& a, const Tuning& t, void* ws, cudaStream_t st) {
  TrP<T> p = make_params<T>(a);
  if (a.mode == kPlain) {
    const int threads = 128;
    dim3 grid(static_cast<unsigned>(a.A), static_cast<unsigned>((a.S + threads - 1) / threads));
    tracer_fwd_plain_kernel<T><<<grid, threads, 0, st>>>(p);
    return cudaGetLastError();
  }
  TrCellP<T> c;
  c.normals = p.normals;
  c.sigmas = p.sigmas;
  c.points = p.points;
  c.tx = p.tx;
  c.rx = p.rx;
  c.inb = p.inb;
  c.out_r = p.out_r;
  c.out_i = p.out_i;
  c.A = a.A;
  c.P = a.P;
  c.splits = t.splits;
  c.c = trace_consts(p.k0, p.b0, p.k1, p.b1, a.S);
  unsigned char* base = static_cast<unsigned char*>(ws);
  c.records = reinterpret_cast<TraceRecord*>(base);
  const FwdLayout l = fwd_layout(a, t.splits);
  c.rows = reinterpret_cast<float2*>(base + l.rows);
  c.plist = nullptr;
  c.plist_count = nullptr;
  if (tracer_point_list_applies(a)) {
    void* lws = base + l.list;
    const cudaError_t err = tracer_point_list(a, lws, false, st);
    if (err != cudaSuccess) return err;
    const PointList pl = tracer_point_list_view(lws, a.P);
    c.plist = pl.list;
    c.plist_count = pl.count;
  }
  if (a.A * t.splits > 0x7fffffff) return cudaErrorInvalidConfiguration;
  if (t.splits == 1 && short_antennas(a)) {
    tracer_fwd_short_kernel<T><<<static_cast<unsigned>(a.A), kTraceThreads, 0, st>>>(c);
    return cudaGetLastError();
  }
  tracer_fwd_cells_kernel<T><<<static_cast<unsigned>(a.A * t.splits), kTraceThreads, 0, st>>>(c);
  if (finish_by_warps(a.A, a.S, c.c.kappa) && t.splits <= kFewShares) {
    return launch_few(reinterpret_cast<const void*>(&tracer_fwd_finish_few_kernel<T>), &c, a.A, a.S, st);
  }
  const dim3 grid(static_cast<unsigned>(a.A), static_cast<unsigned>((a.S + kFinishSamples - 1) / kFinishSamples));
  tracer_fwd_finish_kernel<T><<<grid, kFinishThreads, 0, st>>>(c);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_tracer_bwd(const TracerArgs& a, const Tuning& t, void* ws, cudaStream_t st) {
  TrP<T> p = make_params<T>(a);
  // workspace: the range cells' (when they apply), the split partials, the point list
  const bool cells = tracer_adjoint_cells_apply(a);
  unsigned char* after_cells = static_cast<unsigned char*>(ws) + (cells ? tracer_adjoint_cells_workspace(a) : 0);
  p.partial = reinterpret_cast<float*>(after_cells);
  const int threads = t.threads;
  p.splits = t.splits;
  const int64_t rows_total = std::max<int64_t>(1, (a.A + t.stage_rows - 1) / t.stage_rows);
  p.per_split = ((rows_total + t.splits - 1) / t.splits) * t.stage_rows;
  p.ld = static_cast<int>(((std::max<int64_t>(a.S, 1) + 3) / 4) * 4);
  const size_t es = a.dtype == kF64 ? 8 : 4;
  p.bulk = (a.S > 0 && a.S % 4 == 0 && (a.S * es) % 16 == 0 && aligned16(a.grad_real_out) &&
            aligned16(a.grad_imag_out))
               ? 1
               : 0;
  int rows = t.stage_rows;
  const bool with_points = a.grad_points != nullptr;
  const int nc = with_points ? 6 : 3;
  auto layout = [&](int rw) {
    if (a.mode == kPlain) {
      const AdjSmem b = adj_smem_layout<T>(rw, p.ld);
      return AdjMixedSmem{b.pos_off, b.buf_off, 0, 0, 0, b.total};
    }
    return adj_mixed_smem_layout<T>(rw, p.ld, threads, nc);
  };
  AdjMixedSmem lay = layout(rows);
  const DeviceInfo dev = current_device_info();
  while (rows > 1 && lay.total > static_cast<size_t>(dev.max_smem_optin)) {
    rows /= 2;
    lay = layout(rows);
  }
  if (rows != t.stage_rows) {
    p.per_split = ((std::max<int64_t>(1, (a.A + rows - 1) / rows) + t.splits - 1) / t.splits) * rows;
  }
  p.rows = rows;
  p.pos_off = lay.pos_off;
  p.buf_off = lay.buf_off;
  p.cnt_off = lay.cnt_off;
  p.list_off = lay.list_off;
  p.contrib_off = lay.contrib_off;
  const void* fn;
  if (a.mode == kPlain) {
    fn = with_points ? reinterpret_cast<const void*>(&tracer_bwd_plain_kernel<T, true>)
                     : reinterpret_cast<const void*>(&tracer_bwd_plain_kernel<T, false>);
  } else {
    fn = with_points ? reinterpret_cast<const void*>(&tracer_bwd_mixed_kernel<T, true>)
                     : reinterpret_cast<const void*>(&tracer_bwd_mixed_kernel<T, false>);
  }
  cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(lay.total));
  if (err != cudaSuccess) return err;
  const int64_t ptiles = (a.P + threads - 1) / threads;
  int64_t blocks = ptiles * t.splits;
  // MIXED blocks take tiles in turn; a few waves of them
  if (a.mode == kMixed) blocks = std::min<int64_t>(blocks, static_cast<int64_t>(dev.sm_count) * 24);
  if (blocks > 0x7fffffff) return cudaErrorInvalidConfiguration;
  if (a.mode == kMixed && tracer_point_list_applies(a)) {
    // lists the points and zeroes the gradients of every point it leaves out
    const size_t partial_bytes = t.splits > 1 ? static_cast<size_t>(t.splits) * a.P * 6 * sizeof(float) : 0;
    void* lws = after_cells + list_region_offset(partial_bytes);
    err = tracer_point_list(a, lws, true, st, cells ? tracer_adjoint_cells_boxes(ws) : nullptr);
    if (err != cudaSuccess) return err;
    const PointList pl = tracer_point_list_view(lws, a.P);
    p.plist = pl.list;
    p.plist_count = pl.count;
    if (cells) {
      err = tracer_adjoint_cells(a, ws, pl, p.partial, t.splits, st, &p.run_if);
      if (err != cudaSuccess) return err;
    }
  }
  void* args[] = {&p};
  err = cudaLaunchKernel(fn, dim3(static_cast<unsigned>(blocks)), dim3(threads), args, lay.total, st);
  if (err != cudaSuccess) return err;
  if (t.splits > 1) {
    const int fin_blocks = static_cast<int>(std::min<int64_t>((a.P + 255) / 256, 148 * 16));
    tracer_bwd_finalize_kernel<T><<<std::max(fin_blocks, 1), 256, 0, st>>>(
        p.partial, t.splits, a.P, p.g_normals, with_points ? p.g_points : nullptr, p.plist, p.plist_count);
    err = cudaGetLastError();
  }
  return err;
}

template <typename T>
BiP<T> make_bi(const BilinearArgs& a) {
  BiP<T> p;
  p.normals = static_cast<const T*>(a.normals);
  p.sigmas = static_cast<const T*>(a.sigmas);
  p.z = static_cast<const T*>(a.z_vals);
  p.tz = static_cast<const T*>(a.tz_vals);
  p.out_n = static_cast<T*>(a.out_normals);
  p.out_s = static_cast<T*>(a.out_sigmas);
  p.out_inb = a.out_inbounds;
  p.A = a.A;
  p.R = a.R;
  p.S = a.S;
  p.T_ = a.T;
  return p;
}

}  // namespace

// ---------------------------------------------------------------------------
cudaError_t launch_tracer_bwd_finalize(int dtype, const float* partial, int splits, int64_t P, void* g_normals,
                                       void* g_points, cudaStream_t st, const int* plist,
                                       const int* plist_count) {
  const int blocks = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((P + 255) / 256, 148 * 16)));
  if (dtype == kF64) {
    tracer_bwd_finalize_kernel<double><<<blocks, 256, 0, st>>>(partial, splits, P, static_cast<double*>(g_normals),
                                                               static_cast<double*>(g_points), plist, plist_count);
  } else {
    tracer_bwd_finalize_kernel<float><<<blocks, 256, 0, st>>>(partial, splits, P, static_cast<float*>(g_normals),
                                                              static_cast<float*>(g_points), plist, plist_count);
  }
  return cudaGetLastError();
}

// The NUFFT form's interpolation width, and the same call in the MIXED form when that width
// is 8 or more: the range cells are then both the more accurate and the faster way (64-bit
// error 1.2e-6 by 8 taps, 9e-7 by the cells).  Fewer taps are a coarser form of their own.
int nufft_taps(const Tuning& t) { return t.taps == 4 || t.taps == 6 || t.taps == 10 || t.taps == 12 ? t.taps : 8; }

TracerArgs resolved_form(const TracerArgs& a, const Tuning& t) {
  TracerArgs b = a;
  if (a.mode == kNufft && nufft_taps(t) >= 8) b.mode = kMixed;
  return b;
}

Tuning tracer_forward_resolve(const TracerArgs& call, const Tuning& req) {
  const TracerArgs a = resolved_form(call, req);
  if (a.mode == kNufft) return tracer_nufft_forward_resolve(a, req);
  Tuning t = req;
  if (t.items <= 0) t.items = 1;
  if (t.stage_rows <= 0) t.stage_rows = 8;
  if (a.mode == kPlain) {
    t.splits = 1;
    return t;
  }
  // MIXED: one block per (antenna, split of the points).  Each share costs a record of its cells, so
  // one wave of blocks, or shares of 2048 points where those are more (632 antennas x 1774 points
  // x 200 samples: 87 us with one, 322 us with a share per batch of 128; 1000 x 20000 x 128: 711 us with one,
  // 493 us with 5); where the antennas fill the GPU, no more than the finish by warps adds up.
  const int64_t batches = std::max<int64_t>(1, (a.P + kTraceThreads - 1) / kTraceThreads);
  if (t.splits <= 0) {
    const int sms = current_device_info().sm_count;
    const int64_t antennas = std::max<int64_t>(1, a.A), wave = 5 * static_cast<int64_t>(sms);
    int64_t most = std::max(wave / antennas, (a.P + 2047) / 2048);
    if (antennas >= wave) most = std::min<int64_t>(most, kFewShares);
    if (short_antennas(a)) most = 1;
    t.splits = pick_splits(antennas, 5, sms, std::min(most, batches));
  }
  t.splits = static_cast<int>(std::min<int64_t>(std::max(t.splits, 1), batches));
  return t;
}

size_t tracer_forward_workspace(const TracerArgs& call, const Tuning& t) {
  const TracerArgs a = resolved_form(call, t);
  if (a.mode == kNufft) return tracer_nufft_forward_workspace(a, t);
  if (a.mode == kPlain) return 0;
  const size_t before_list = fwd_layout(a, t.splits).list;
  return tracer_point_list_applies(a) ? before_list + tracer_point_list_bytes(a.P) : before_list;
}

cudaError_t tracer_forward(const TracerArgs& call, const Tuning& t, void* ws, cudaStream_t st) {
  const TracerArgs a = resolved_form(call, t);
  if (a.mode == kNufft) return tracer_nufft_forward(a, t, ws, st);
  if (a.A == 0 || a.S == 0) return cudaSuccess;
  if (a.dtype == kF64) return launch_tracer_fwd<double>(a, t, ws, st);
  return launch_tracer_fwd<float>(a, t, ws, st);
}

Tuning tracer_backward_resolve(const TracerArgs& call, const Tuning& req) {
  const TracerArgs a = resolved_form(call, req);
  if (a.mode == kNufft) return tracer_nufft_backward_resolve(a, req);
  Tuning t = req;
  if (t.threads != 64 && t.threads != 128) t.threads = 128;
  if (t.items <= 0) t.items = 1;
  // MIXED: 4-antenna stages keep 6 blocks resident per SM (8 fit 4, by shared
  // memory); 5% faster on 64 antennas x 524288 points x 128 samples
  if (t.stage_rows <= 0) t.stage_rows = a.mode == kMixed ? 4 : 8;
  t.stage_rows = std::min(t.stage_rows, 64);
  if (t.chunk <= 0) t.chunk = 16;
  const int64_t rows_total = std::max<int64_t>(1, (a.A + t.stage_rows - 1) / t.stage_rows);
  if (t.splits <= 0) {
    int64_t ptiles = std::max<int64_t>(1, (a.P + t.threads - 1) / t.threads);
    // With the point pre-cull only the blocks of listed points have work; the
    // default assumes a quarter of the points are listed (14% on 64 antennas
    // looking at a 4096-ray SDF scene).
    if (a.mode == kMixed && tracer_point_list_applies(a)) ptiles = std::max<int64_t>(1, ptiles / 4);
    const DeviceInfo dev = current_device_info();
    const int per_sm = std::max(1, 1024 / t.threads);
    t.splits = a.mode == kPlain ? 1 : pick_splits(ptiles, per_sm, dev.sm_count, rows_total);
  }
  t.splits = static_cast<int>(std::min<int64_t>(std::max(t.splits, 1), rows_total));
  return t;
}

size_t tracer_backward_workspace(const TracerArgs& call, const Tuning& t) {
  const TracerArgs a = resolved_form(call, t);
  if (a.mode == kNufft) return tracer_nufft_backward_workspace(a, t);
  const size_t partial_bytes = t.splits > 1 && a.P > 0 ? static_cast<size_t>(t.splits) * a.P * 6 * sizeof(float) : 0;
  if (!tracer_point_list_applies(a)) return partial_bytes;
  const size_t cells = tracer_adjoint_cells_apply(a) ? tracer_adjoint_cells_workspace(a) : 0;
  return cells + list_region_offset(partial_bytes) + tracer_point_list_bytes(a.P);
}

cudaError_t tracer_backward(const TracerArgs& call, const Tuning& t, void* ws, cudaStream_t st) {
  const TracerArgs a = resolved_form(call, t);
  if (a.mode == kNufft) return tracer_nufft_backward(a, t, ws, st);
  if (a.P == 0) return cudaSuccess;
  if (a.dtype == kF64) return launch_tracer_bwd<double>(a, t, ws, st);
  return launch_tracer_bwd<float>(a, t, ws, st);
}

cudaError_t bilinear_forward(const BilinearArgs& a, cudaStream_t st) {
  if (a.R == 0 || a.T == 0) return cudaSuccess;
  const int64_t blocks = (a.R * 32 + 255) / 256;
  if (a.dtype == kF64) bilinear_fwd_kernel<double><<<static_cast<unsigned>(blocks), 256, 0, st>>>(make_bi<double>(a));
  else bilinear_fwd_kernel<float><<<static_cast<unsigned>(blocks), 256, 0, st>>>(make_bi<float>(a));
  return cudaGetLastError();
}

cudaError_t bilinear_backward(const BilinearArgs& a, cudaStream_t st) {
  if (a.R == 0 || a.S == 0) return cudaSuccess;
  constexpr int kRays = 8;  // per block
  const int64_t blocks = (a.R + kRays - 1) / kRays;
  const size_t tile = static_cast<size_t>(std::min<int64_t>(a.T, kTargetTile)) * kRays;
  if (a.dtype == kF64) {
    bilinear_bwd_kernel<double><<<static_cast<unsigned>(blocks), kRays * 32, tile * (sizeof(double) + sizeof(int)), st>>>(make_bi<double>(a));
  } else {
    bilinear_bwd_kernel<float><<<static_cast<unsigned>(blocks), kRays * 32, tile * (sizeof(float) + sizeof(int)), st>>>(make_bi<float>(a));
  }
  return cudaGetLastError();
}

}  // namespace geraf
