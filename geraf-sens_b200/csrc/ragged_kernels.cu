// Batched signal tracer over all antennas of a step, each antenna with its own
// uneven set of points (rays x samples surviving the filter-based culling),
// in the MIXED arithmetic form.
//
// Layout: points / normals [P, 3], sigmas [P] and inbounds [P] hold the points
// of antenna 0, then antenna 1, ... ; point_offsets [A + 1] (int64, CSR) gives
// antenna a the points [offsets[a], offsets[a+1]).  Per antenna the result is
// exactly the reference's tracer over that antenna's points:
//   x[a, n] = (1 / P_a) sum_{p of a} sigma[p] rho / D^2 exp(+j (w0 + w1 t_n) tau)
// (SignalTracer_cuda_kernel.cu:351-450 with total_point_size = P_a).
//
// Forward: one persistent launch.  A one-block prep pass validates the
// offsets and lays out work items (antenna, chunk of `chunk` points); resident
// blocks then take items from an atomic counter until none are left, so
// antennas with 512 rays and antennas with 8192 rays load-balance.  An item
// leaves the moments of its points in range cells (tracer_cells.cuh); a finish
// pass turns each antenna's moments into samples in item order (deterministic).
// Adjoint: a point belongs to one antenna, so its gradients need no reduction
// across antennas; blocks screen runs of points and deal the live ones out
// over their threads.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "tracer_cells.cuh"
#include "tracer_geometry.cuh"
#include "tracer_gradients.cuh"

namespace geraf {
namespace {

using namespace tracer;

constexpr int kStatusBadOffsets = 1;  // GERAF_ERR_INVALID_ARGUMENT

template <typename T>
struct RgP {
  const T* normals;
  const T* sigmas;
  const T* points;
  const int64_t* offsets;
  const T* tx;
  const T* rx;
  const uint8_t* inb;  // may be null: all points in bounds
  T* out_r;
  T* out_i;
  const T* gr;
  const T* gi;
  T* g_normals;
  T* g_sigmas;
  T* g_points;
  TraceRecord* records;   // [max_items]
  float2* rows;           // [max_items][S]
  int64_t* item_offsets;  // [A + 1]
  unsigned long long* counter;
  int* status;
  int64_t A, S, P, max_items;
  int chunk;
  float fs, f0, As;
  double k0, b0, k1, b1;
  TraceConsts c;
};

template <typename T>
__device__ __forceinline__ void ld3(const T* base, int64_t i, float* out) {
  out[0] = ld_f(base, i * 3 + 0);
  out[1] = ld_f(base, i * 3 + 1);
  out[2] = ld_f(base, i * 3 + 2);
}

// Validates the CSR offsets and writes item_offsets (prefix sums of
// ceil(P_a / chunk)); resets the work counter.  Malformed offsets give zero
// items and raise the status word, so nothing downstream reads a point.
template <typename T>
__global__ void __launch_bounds__(1024) ragged_prep_kernel(const RgP<T> p) {
  __shared__ int bad;
  __shared__ long long carry;
  if (threadIdx.x == 0) {
    bad = (p.offsets[0] != 0 || p.offsets[p.A] != p.P) ? 1 : 0;
    carry = 0;
    *p.counter = 0ull;
  }
  __syncthreads();
  for (int64_t a = threadIdx.x; a < p.A; a += blockDim.x) {
    if (p.offsets[a + 1] < p.offsets[a]) bad = 1;
  }
  __syncthreads();
  if (bad) {
    for (int64_t a = threadIdx.x; a <= p.A; a += blockDim.x) p.item_offsets[a] = 0;
    if (threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, kStatusBadOffsets);
    return;
  }
  // Block-wide exclusive scan of item counts, blockDim antennas at a time.
  __shared__ long long warp_sums[32];
  for (int64_t base = 0; base < p.A; base += blockDim.x) {
    const int64_t a = base + threadIdx.x;
    long long cnt = 0;
    if (a < p.A) cnt = (p.offsets[a + 1] - p.offsets[a] + p.chunk - 1) / p.chunk;
    long long incl = cnt;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int d = 1; d < 32; d <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += y;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const int nw = blockDim.x >> 5;
      long long v = lane < nw ? warp_sums[lane] : 0;
      for (int d = 1; d < 32; d <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += y;
      }
      if (lane < nw) warp_sums[lane] = v;
    }
    __syncthreads();
    const long long before = (warp > 0 ? warp_sums[warp - 1] : 0) + carry;
    if (a < p.A) p.item_offsets[a] = before + incl - cnt;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = before + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) p.item_offsets[p.A] = carry;
}

// Antenna owning work item `item`: the last a with item_offsets[a] <= item.
__device__ __forceinline__ int64_t item_antenna(const int64_t* item_offsets, int64_t A, int64_t item) {
  int64_t lo = 0, hi = A;  // invariant: item_offsets[lo] <= item < item_offsets[hi]
  while (hi - lo > 1) {
    const int64_t mid = (lo + hi) >> 1;
    if (item_offsets[mid] <= item) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Points [first, first + count) of antenna a.
template <typename T>
__device__ __forceinline__ void item_range(const RgP<T>& p, int64_t item, int64_t& a, int64_t& first, int64_t& count) {
  a = item_antenna(p.item_offsets, p.A, item);
  first = p.offsets[a] + (item - p.item_offsets[a]) * p.chunk;
  count = min(p.offsets[a + 1] - first, static_cast<int64_t>(p.chunk));
}

// Row of an item whose cells do not fit their slots.
template <typename T>
__device__ __forceinline__ void item_direct(DirectSmem& sm, const RgP<T>& p, int64_t item) {
  int64_t a, first, count;
  item_range(p, item, a, first, count);
  float txp[3], rxp[3];
  ld3(p.tx, a, txp);
  ld3(p.rx, a, rxp);
  trace_direct<T>(
      sm, p.c, p.normals, p.points, txp, rxp, count,
      [&](int64_t pos) -> int64_t { return p.inb == nullptr || p.inb[first + pos] ? first + pos : -1; },
      [&](int64_t q) { return ld_f(p.sigmas, q); }, [&](int n, float2 y) { p.rows[item * p.c.S + n] = y; });
}
// (Not inlined: it would take registers from the cells.)
template <typename T>
static __device__ __noinline__ void item_direct_call(DirectSmem& sm, const RgP<T>& p, int64_t item) {
  item_direct(sm, p, item);
}

// Each work item's points go into the moments of their cells (tracer_cells.cuh).
// 64 antennas x 295000 points each (10% live) x 256 samples: 173 us against 590 us with
// a recurrence over the samples of every live point and a compaction per 128 points.
// An item whose cells do not fit their slots leaves a row instead: by ROWS from here, else from
// ragged_fwd_direct_kernel.
template <typename T, bool ROWS>
__global__ void __launch_bounds__(kTraceThreads, 6) ragged_fwd_kernel(const __grid_constant__ RgP<T> p) {
  __shared__ union {
    TraceSmem cells;
    DirectSmem direct;
  } smem;
  __shared__ long long s_item;
  TraceSmem& sm = smem.cells;
  const int64_t total = p.item_offsets[p.A];
  for (;;) {
    if (threadIdx.x == 0) s_item = static_cast<long long>(atomicAdd(p.counter, 1ull));
    __syncthreads();
    const int64_t item = s_item;
    if (item >= total) break;
    int64_t a, first, count;
    item_range(p, item, a, first, count);
    float txp[3], rxp[3];
    ld3(p.tx, a, txp);
    ld3(p.rx, a, rxp);
    trace_begin(sm);
    const bool fits = trace_screened<T>(sm, p.c, p.normals + first * 3, p.points + first * 3, p.sigmas + first,
                                        p.inb != nullptr ? p.inb + first : nullptr, txp, rxp, static_cast<int>(count));
    if (!fits) {  // no cells
      for (int i = threadIdx.x; i < kTraceSlots; i += kTraceThreads) sm.tag[i] = kTraceEmpty;
    }
    trace_store(sm, p.records + item, !fits);
    if (ROWS && !fits) item_direct_call(smem.direct, p, item);
  }
}

// The rows of calls of many items; a launch without any reads their records' flags alone.  (Within the
// kernel above it takes registers from the cells: 64 antennas x 100000 points x 256 samples, forward and
// adjoint, 235 -> 272 us.  Calls of an item per block are bound by their launches, so one fewer counts for
// more there: 8 to 32 antennas x 19000 to 63000 points 157 -> 155 us.)
template <typename T>
__global__ void __launch_bounds__(kTraceThreads) ragged_fwd_direct_kernel(const RgP<T> p) {
  __shared__ DirectSmem sm;
  const int64_t total = p.item_offsets[p.A];
  for (int64_t item = blockIdx.x; item < total; item += gridDim.x) {
    if (p.records[item].has_row != 0) item_direct(sm, p, item);
  }
}

// x[a, n] = (sum of antenna a's items, in item order) / P_a.
template <typename T>
__device__ __forceinline__ void finish_antenna(const RgP<T>& p, int64_t a) {
  const int n0 = blockIdx.y * kFinishSamples;
  const int64_t it = p.item_offsets[a];
  trace_finish<T>(p.c, p.records + it, p.rows + it * p.c.S, p.item_offsets[a + 1] - it,
                  static_cast<float>(p.offsets[a + 1] - p.offsets[a]), n0, min(p.c.S, n0 + kFinishSamples),
                  p.out_r + a * p.c.S, p.out_i + a * p.c.S);
}

template <typename T>
__global__ void __launch_bounds__(kFinishThreads) ragged_finish_kernel(const RgP<T> p) {
  finish_antenna(p, blockIdx.x);
}

// Of many antennas, those of more than kFewShares items: a block looks at antennas a =
// blockIdx.x, + gridDim.x, ...
template <typename T>
__global__ void __launch_bounds__(kFinishThreads) ragged_finish_long_kernel(const RgP<T> p) {
  __shared__ int64_t todo[kFinishThreads];
  __shared__ int count;
  for (int64_t a0 = blockIdx.x; a0 < p.A; a0 += static_cast<int64_t>(gridDim.x) * kFinishThreads) {
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    const int64_t a = a0 + static_cast<int64_t>(threadIdx.x) * gridDim.x;
    if (a < p.A && p.item_offsets[a + 1] - p.item_offsets[a] > kFewShares) todo[atomicAdd(&count, 1)] = a;
    __syncthreads();
    for (int i = 0; i < count; ++i) {
      finish_antenna(p, todo[i]);
      __syncthreads();
    }
    __syncthreads();
  }
}

// The others.
template <typename T>
__global__ void __launch_bounds__(kFewThreads) ragged_finish_few_kernel(const RgP<T> p) {
  extern __shared__ __align__(16) unsigned char few_smem[];
  const FewTable f = few_table(p.c, few_smem);
  const int64_t warps = static_cast<int64_t>(gridDim.x) * (kFewThreads / 32);
  for (int64_t a = blockIdx.x * static_cast<int64_t>(kFewThreads / 32) + (threadIdx.x >> 5); a < p.A; a += warps) {
    const int64_t it = p.item_offsets[a], items = p.item_offsets[a + 1] - it;
    if (items > kFewShares) continue;
    trace_finish_few<T>(p.c, f, p.records + it, p.rows + it * p.c.S, static_cast<int>(items),
                        static_cast<float>(p.offsets[a + 1] - p.offsets[a]), p.out_r + a * p.c.S, p.out_i + a * p.c.S);
  }
}

// Antenna owning point pi: the last a with offsets[a] <= pi.  *owned is false
// when the offsets do not cover pi (malformed input).
__device__ __forceinline__ int64_t point_antenna(const int64_t* offsets, int64_t A, int64_t pi,
                                                 bool* owned) {
  int64_t lo = 0, hi = A;
  while (hi - lo > 1) {
    const int64_t mid = (lo + hi) >> 1;
    if (offsets[mid] <= pi) lo = mid;
    else hi = mid;
  }
  *owned = A > 0 && offsets[lo] <= pi && pi < offsets[lo + 1];
  return lo;
}

// Gradients of one point that the early test cannot cull; a point that the exact geometry culls
// keeps what it has.  sums(zeta, q, q1) is residual_sums over the antenna's row.
template <typename T, bool WITH_POINTS, typename Sums>
__device__ __forceinline__ void point_gradients(const RgP<T>& p, int64_t pi, const float* txp, const float* rxp,
                                                float inv_pa, Sums sums) {
  float nrm[3], pt[3];
  ld3(p.normals, pi, nrm);
  ld3(p.points, pi, pt);
  const float sigma = ld_f(p.sigmas, pi);
  PairGeom g;
  if (!pair_geometry(txp, rxp, nrm, pt, g)) return;
  const PhaseCycles pc =
      path_cycles(static_cast<double>(txp[0]) - pt[0], static_cast<double>(txp[1]) - pt[1],
                  static_cast<double>(txp[2]) - pt[2], static_cast<double>(rxp[0]) - pt[0],
                  static_cast<double>(rxp[1]) - pt[1], static_cast<double>(rxp[2]) - pt[2], p.k0, p.b0, p.k1, p.b1);
  float2 q, q1;
  sums(cis_cycles(pc.dcyc), q, q1);
  float gs, gn[3] = {0.0f, 0.0f, 0.0f}, gp[3] = {0.0f, 0.0f, 0.0f};
  const float2 e0 = cis_cycles_fast(pc.frac0);
  // sum_n w_n (g_i cos - g_r sin) = -Im(exp(j phi0) (w0 Q + w1 Q1))
  const float w0 = static_cast<float>(2.0 * static_cast<double>(kPiF) * p.f0);
  const float w1s = static_cast<float>(2.0 * static_cast<double>(kPiF) * p.As / p.fs);
  const float f = cmul(e0, make_float2(w0 * q.x + w1s * q1.x, w0 * q.y + w1s * q1.y)).y;
  pair_gradients<WITH_POINTS>(g, cmul(e0, q).x, f, sigma, nrm, &gs, gn, gp);
  p.g_sigmas[pi] = from_f<T>(gs * inv_pa);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    p.g_normals[pi * 3 + c] = from_f<T>(gn[c] * inv_pa);
    if (WITH_POINTS) p.g_points[pi * 3 + c] = from_f<T>(gp[c] * inv_pa);
  }
}

// Adjoint.  A point belongs to one antenna, so its gradients depend on nothing else.  A
// block takes a run of consecutive points, kBwdTile at a time: it writes zeros for
// all of them (whole lines), screens them with the early test while the next tile's
// points are on their way, lists those the test cannot cull and, a full block of
// them at a time, gives them the exact geometry and the residual sums (packed
// even/odd Horner over the antenna's row in shared memory).
// The sums stay a recurrence over the samples here, the less exact form: the cell polynomials
// of tracer_gradients.cuh err by up to 3.7e-5 in single gradients, the recurrence by up to 4.8e-4.  They
// need tables, for which this entry point has no workspace; formed per block in shared memory they took
// 309 us against 365 us here (64 antennas x 295000 points, 10% live, x 256 samples).  404 us with 1024-point blocks that each
// looked their antenna up first and stored zeros point by point.
constexpr int kBwdThreads = 128;
constexpr int kBwdPer = 4;
constexpr int kBwdTile = kBwdThreads * kBwdPer;

// Zeros for kBwdTile consecutive points' `width` elements each, 16-byte aligned.
template <typename T, int WIDTH>
__device__ __forceinline__ void zero_tile(T* p) {
  constexpr int kVecs = kBwdTile * WIDTH * sizeof(T) / 16;
#pragma unroll
  for (int i = 0; i < kVecs; i += kBwdThreads) reinterpret_cast<uint4*>(p)[i + threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
}

template <typename T, bool WITH_POINTS>
__global__ void __launch_bounds__(kBwdThreads, 6) ragged_bwd_kernel(const RgP<T> p, int64_t run, int ld, int aligned) {
  extern __shared__ __align__(16) float srow[];  // [2][ld]
  __shared__ int list[kBwdTile + kBwdThreads];   // offsets in the run
  __shared__ int s_listed;
  const int lane = threadIdx.x & 31;
  const int64_t begin = blockIdx.x * run;
  const int64_t end = min(p.P, begin + run);
  float* rowr = srow;
  float* rowi = srow + ld;
  if (threadIdx.x == 0) s_listed = 0;

  int64_t a = 0, seg_end = begin;  // the current antenna's points end at seg_end
  float txp[3] = {0.0f, 0.0f, 0.0f}, rxp[3] = {0.0f, 0.0f, 0.0f};
  float inv_pa = 0.0f;

  // Gradients of listed points [from, from + cnt) of the current antenna.
  auto batch = [&](int cnt, int from) {
    if (threadIdx.x >= cnt) return;
    point_gradients<T, WITH_POINTS>(p, begin + list[from + threadIdx.x], txp, rxp, inv_pa,
                                    [&](float2 zeta, float2& q, float2& q1) {
                                      residual_sums<WITH_POINTS>(rowr, rowi, ld, zeta, q, q1);
                                    });
  };
  // The full batches that the list holds; all of it when `drain`.  Between two barriers.
  auto serve = [&](bool drain) {
    __syncthreads();
    int listed = s_listed;
    while (listed >= kBwdThreads || (drain && listed > 0)) {
      const int cnt = min(listed, kBwdThreads);
      listed -= cnt;
      batch(cnt, listed);
    }
    __syncthreads();
    if (threadIdx.x == 0) s_listed = listed;
  };

  float nrm[kBwdPer][3], pt[kBwdPer][3];
  unsigned inb = 0;  // bit j: point j of the thread is in bounds
  auto load = [&](int64_t t0) {
    inb = 0;
    if (t0 >= end) return;
    const int rest = static_cast<int>(min(end - t0, static_cast<int64_t>(kBwdTile))) - static_cast<int>(threadIdx.x);
    const T* pn = p.normals + (t0 + threadIdx.x) * 3;
    const T* pp = p.points + (t0 + threadIdx.x) * 3;
    const uint8_t* pb = p.inb != nullptr ? p.inb + t0 + threadIdx.x : nullptr;
#pragma unroll
    for (int j = 0; j < kBwdPer; ++j) {
      if (j * kBwdThreads < rest && (pb == nullptr || pb[j * kBwdThreads])) {
        inb |= 1u << j;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          nrm[j][c] = ld_f(pn, j * kBwdThreads * 3 + c);
          pt[j][c] = ld_f(pp, j * kBwdThreads * 3 + c);
        }
      }
    }
  };
  load(begin);
  for (int64_t t0 = begin; t0 < end; t0 += kBwdTile) {
    const int64_t t1 = min(end, t0 + kBwdTile);
    if (aligned && t1 - t0 == kBwdTile) {
      zero_tile<T, 1>(p.g_sigmas + t0);
      zero_tile<T, 3>(p.g_normals + t0 * 3);
      if (WITH_POINTS) zero_tile<T, 3>(p.g_points + t0 * 3);
    } else {
      zero_range(p.g_sigmas, t0, t1);
      zero_range(p.g_normals, t0 * 3, t1 * 3);
      if (WITH_POINTS) zero_range(p.g_points, t0 * 3, t1 * 3);
    }
    // the antennas of the tile, usually one
    for (int64_t cur = t0; cur < t1;) {
      if (cur >= seg_end) {
        serve(true);  // the preceding antenna's points
        bool owned;
        a = point_antenna(p.offsets, p.A, cur, &owned);
        if (!owned) {  // malformed offsets: the point keeps its zeros
          if (threadIdx.x == 0 && p.status != nullptr) atomicExch(p.status, kStatusBadOffsets);
          ++cur;
          continue;
        }
        seg_end = p.offsets[a + 1];
        inv_pa = 1.0f / static_cast<float>(seg_end - p.offsets[a]);
        ld3(p.tx, a, txp);
        ld3(p.rx, a, rxp);
        for (int n = threadIdx.x; n < ld; n += kBwdThreads) {
          rowr[n] = n < p.S ? ld_f(p.gr, a * p.S + n) : 0.0f;
          rowi[n] = n < p.S ? ld_f(p.gi, a * p.S + n) : 0.0f;
        }
        __syncthreads();
      }
      const int64_t stop = min(t1, seg_end);
      const int lo = static_cast<int>(cur - t0) - static_cast<int>(threadIdx.x);
      const int hi = static_cast<int>(stop - t0) - static_cast<int>(threadIdx.x);
      const int at0 = static_cast<int>(t0 - begin) + static_cast<int>(threadIdx.x);
#pragma unroll
      for (int j = 0; j < kBwdPer; ++j) {
        const bool keep = ((inb >> j) & 1u) && j * kBwdThreads >= lo && j * kBwdThreads < hi &&
                          !surely_culled(txp, rxp, nrm[j], pt[j]);
        const unsigned mask = __ballot_sync(0xffffffffu, keep);
        if (mask == 0u) continue;
        int at = 0;
        if (lane == 0) at = atomicAdd(&s_listed, __popc(mask));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (keep) list[at + __popc(mask & ((1u << lane) - 1u))] = at0 + j * kBwdThreads;
      }
      cur = stop;
    }
    load(t0 + kBwdTile);
    serve(false);
    __syncthreads();
  }
  serve(true);
}

// The adjoint where antennas have few points each, which would have the kernel above change
// antennas (a row to stage, three barriers) every few points: a block screens 512 points,
// each with its own antenna, lists those that the early test cannot cull, and its threads
// read their antennas' rows from device memory.  Bound by those reads.  64 samples, 1000
// antennas of one point: 1.40 ms above, 30 us here; 256 samples, 49152 x 4: 779 and 86 us, 16384
// x 32: 199 and 130 us; above 48 points the rows in shared memory win (2000 x 64: 50 us above,
// 106 us by this form's forerunner).
constexpr int kShortPoints = 48;  // per antenna, on average

template <typename T, bool WITH_POINTS>
__global__ void __launch_bounds__(kBwdThreads, 6) ragged_bwd_short_kernel(const RgP<T> p, int ld, int vector_rows) {
  __shared__ int list[kBwdTile];
  __shared__ int s_listed;
  const int64_t begin = blockIdx.x * static_cast<int64_t>(kBwdTile);
  const int64_t end = min(p.P, begin + kBwdTile);
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) s_listed = 0;
  zero_range(p.g_sigmas, begin, end);
  zero_range(p.g_normals, begin * 3, end * 3);
  if (WITH_POINTS) zero_range(p.g_points, begin * 3, end * 3);
  __syncthreads();
#pragma unroll 1
  for (int j = 0; j < kBwdPer; ++j) {
    const int64_t pi = begin + j * kBwdThreads + threadIdx.x;
    bool keep = false;
    if (pi < end) {
      bool owned;
      const int64_t a = point_antenna(p.offsets, p.A, pi, &owned);
      if (!owned && p.status != nullptr) atomicExch(p.status, kStatusBadOffsets);
      if (owned && (p.inb == nullptr || p.inb[pi])) {
        float nrm[3], pt[3], txp[3], rxp[3];
        ld3(p.normals, pi, nrm);
        ld3(p.points, pi, pt);
        ld3(p.tx, a, txp);
        ld3(p.rx, a, rxp);
        keep = !surely_culled(txp, rxp, nrm, pt);
      }
    }
    const unsigned mask = __ballot_sync(0xffffffffu, keep);
    int at = 0;
    if (lane == 0 && mask != 0u) at = atomicAdd(&s_listed, __popc(mask));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (keep) list[at + __popc(mask & ((1u << lane) - 1u))] = j * kBwdThreads + static_cast<int>(threadIdx.x);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < s_listed; i += kBwdThreads) {
    const int64_t pi = begin + list[i];
    bool owned;
    const int64_t a = point_antenna(p.offsets, p.A, pi, &owned);
    float txp[3], rxp[3];
    ld3(p.tx, a, txp);
    ld3(p.rx, a, rxp);
    const float inv_pa = 1.0f / static_cast<float>(p.offsets[a + 1] - p.offsets[a]);
    const T* gr = p.gr + a * p.S;
    const T* gi = p.gi + a * p.S;
    const int S = static_cast<int>(p.S);
    point_gradients<T, WITH_POINTS>(p, pi, txp, rxp, inv_pa, [&](float2 zeta, float2& q, float2& q1) {
      residual_sums<WITH_POINTS>(
          [=](int n, float4& re, float4& im) {
            if (vector_rows) {
              re = lds4(gr + n);
              im = lds4(gi + n);
            } else {
              re = make_float4(ld_f(gr, n), n + 1 < S ? ld_f(gr, n + 1) : 0.0f, n + 2 < S ? ld_f(gr, n + 2) : 0.0f,
                               n + 3 < S ? ld_f(gr, n + 3) : 0.0f);
              im = make_float4(ld_f(gi, n), n + 1 < S ? ld_f(gi, n + 1) : 0.0f, n + 2 < S ? ld_f(gi, n + 2) : 0.0f,
                               n + 3 < S ? ld_f(gi, n + 3) : 0.0f);
            }
          },
          S > 0 ? ld : 0, zeta, q, q1);
    });
  }
}

// ---------------------------------------------------------------------------
struct RaggedLayout {
  int64_t max_items;
  size_t records_off, rows_off, items_off, counter_off, total;
  int chunk;
};

// Points per work item: items_per_thread x threads when tuned, else at least
// 2048 and more for large steps (fewer partial rows); a multiple of 256.
int ragged_chunk(int64_t P, const Tuning& t) {
  int64_t c = t.items > 0 ? static_cast<int64_t>(t.items) * t.threads
                          : std::max<int64_t>(2048, std::min<int64_t>(16384, P / (148 * 8 + 1)));
  c = std::max<int64_t>(256, std::min<int64_t>(c, 1 << 20));
  return static_cast<int>((c + 255) / 256 * 256);
}

RaggedLayout ragged_layout(int64_t A, int64_t S, int64_t P, const Tuning& t) {
  RaggedLayout l;
  l.chunk = ragged_chunk(P, t);
  l.max_items = P / l.chunk + A + 1;
  l.records_off = 0;
  size_t off = static_cast<size_t>(l.max_items) * sizeof(TraceRecord);
  off = (off + 255) & ~static_cast<size_t>(255);
  l.rows_off = off;
  off += static_cast<size_t>(l.max_items) * std::max<int64_t>(S, 1) * sizeof(float2);
  off = (off + 255) & ~static_cast<size_t>(255);
  l.items_off = off;
  off += static_cast<size_t>(A + 1) * sizeof(int64_t);
  off = (off + 255) & ~static_cast<size_t>(255);
  l.counter_off = off;
  off += 256;
  l.total = off;
  return l;
}

template <typename T>
RgP<T> make_rg(const RaggedArgs& a, const Tuning& t, void* ws) {
  RgP<T> p{};
  p.normals = static_cast<const T*>(a.normals);
  p.sigmas = static_cast<const T*>(a.sigmas);
  p.points = static_cast<const T*>(a.points);
  p.offsets = a.offsets;
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
  if (ws != nullptr) {
    const RaggedLayout l = ragged_layout(a.A, a.S, a.P, t);
    unsigned char* base = static_cast<unsigned char*>(ws);
    p.records = reinterpret_cast<TraceRecord*>(base + l.records_off);
    p.rows = reinterpret_cast<float2*>(base + l.rows_off);
    p.item_offsets = reinterpret_cast<int64_t*>(base + l.items_off);
    p.counter = reinterpret_cast<unsigned long long*>(base + l.counter_off);
    p.max_items = l.max_items;
    p.chunk = l.chunk;
  }
  p.c = trace_consts(pc.k0, pc.b0, pc.k1, pc.b1, a.S);
  return p;
}

template <typename T>
cudaError_t launch_ragged_fwd(const RaggedArgs& a, const Tuning& t, void* ws, cudaStream_t st) {
  RgP<T> p = make_rg<T>(a, t, ws);
  ragged_prep_kernel<T><<<1, 1024, 0, st>>>(p);
  const int per_sm = resident_blocks(reinterpret_cast<const void*>(&ragged_fwd_kernel<T, false>), kTraceThreads, 0);
  const int64_t resident = std::max<int64_t>(1, static_cast<int64_t>(per_sm) * current_device_info().sm_count);
  if (p.max_items <= resident) {
    ragged_fwd_kernel<T, true><<<static_cast<unsigned>(p.max_items), kTraceThreads, 0, st>>>(p);
  } else {
    ragged_fwd_kernel<T, false><<<static_cast<unsigned>(resident), kTraceThreads, 0, st>>>(p);
    ragged_fwd_direct_kernel<T><<<static_cast<unsigned>(resident), kTraceThreads, 0, st>>>(p);
  }
  const int64_t sms = current_device_info().sm_count;
  const unsigned parts = static_cast<unsigned>((a.S + kFinishSamples - 1) / kFinishSamples);
  if (!finish_by_warps(a.A, a.S, p.c.kappa)) {
    ragged_finish_kernel<T><<<dim3(static_cast<unsigned>(a.A), parts), kFinishThreads, 0, st>>>(p);
  } else {
    ragged_finish_long_kernel<T><<<dim3(static_cast<unsigned>(std::min<int64_t>(a.A, 2 * sms)), parts), kFinishThreads, 0, st>>>(p);
    const cudaError_t err = launch_few(reinterpret_cast<const void*>(&ragged_finish_few_kernel<T>), &p, a.A, a.S, st);
    if (err != cudaSuccess) return err;
  }
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_ragged_bwd(const RaggedArgs& a, cudaStream_t st) {
  RgP<T> p = make_rg<T>(a, Tuning{}, nullptr);
  const int ld = static_cast<int>(((std::max<int64_t>(a.S, 1) + 3) / 4) * 4);
  const size_t smem = static_cast<size_t>(2 * ld) * sizeof(float);
  const bool with_points = a.grad_points != nullptr;
  const void* fn = with_points ? reinterpret_cast<const void*>(&ragged_bwd_kernel<T, true>)
                               : reinterpret_cast<const void*>(&ragged_bwd_kernel<T, false>);
  auto aligned16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
  if (a.P < kShortPoints * a.A) {
    int vector_rows = a.S % 4 == 0 && aligned16(a.grad_real_out) && aligned16(a.grad_imag_out) ? 1 : 0;
    const int64_t tiles = (a.P + kBwdTile - 1) / kBwdTile;
    if (tiles > 0x7fffffff) return cudaErrorInvalidConfiguration;
    if (with_points) ragged_bwd_short_kernel<T, true><<<static_cast<unsigned>(tiles), kBwdThreads, 0, st>>>(p, ld, vector_rows);
    else ragged_bwd_short_kernel<T, false><<<static_cast<unsigned>(tiles), kBwdThreads, 0, st>>>(p, ld, vector_rows);
    return cudaGetLastError();
  }
  int aligned = aligned16(a.grad_sigmas) && aligned16(a.grad_normals) && aligned16(a.grad_points) ? 1 : 0;
  // Runs of consecutive points: a few per resident block, so that the last ones end together.
  const int64_t slots = static_cast<int64_t>(current_device_info().sm_count) * 6;
  int64_t run = (a.P + 4 * slots - 1) / (4 * slots);
  run = std::max<int64_t>(1, std::min<int64_t>((run + kBwdTile - 1) / kBwdTile, 64)) * kBwdTile;
  const int64_t blocks = (a.P + run - 1) / run;
  if (blocks > 0x7fffffff) return cudaErrorInvalidConfiguration;
  void* args[] = {&p, &run, const_cast<int*>(&ld), &aligned};
  return cudaLaunchKernel(fn, dim3(static_cast<unsigned>(blocks)), dim3(kBwdThreads), args, smem, st);
}

}  // namespace

Tuning tracer_ragged_forward_resolve(const RaggedArgs& a, const Tuning& req) {
  Tuning t = req;
  if (t.threads != 64 && t.threads != 128 && t.threads != 256) t.threads = kTraceThreads;
  if (t.items < 0) t.items = 0;
  t.items = std::min(t.items, 4096);
  return t;
}

size_t tracer_ragged_workspace(int64_t A, int64_t S, int64_t P, const Tuning& t) {
  return ragged_layout(A, S, P, t).total;
}

cudaError_t tracer_forward_ragged(const RaggedArgs& a, const Tuning& t, void* ws, cudaStream_t st) {
  if (a.A == 0 || a.S == 0) return cudaSuccess;
  if (a.dtype == kF64) return launch_ragged_fwd<double>(a, t, ws, st);
  return launch_ragged_fwd<float>(a, t, ws, st);
}

cudaError_t tracer_backward_ragged(const RaggedArgs& a, cudaStream_t st) {
  if (a.P == 0) return cudaSuccess;
  if (a.dtype == kF64) return launch_ragged_bwd<double>(a, st);
  return launch_ragged_bwd<float>(a, st);
}

}  // namespace geraf
