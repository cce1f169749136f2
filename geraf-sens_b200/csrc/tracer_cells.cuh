// MIXED tracer forward through range cells: the live points of one antenna enter
// its samples through the moments of their cells (range_cells.cuh, the adjoint of
// the matched filter),
//   x[a, n] = (1/P) sum_cells e^{+j 2 pi n' d_k} (sum_q even g_q(n) M_q + j sum_q odd g_q(n) M_q),
//   M_q = sum_p amp_p e^{+j 2 pi c_p} x_p^q,
// so a live point costs eight multiply-adds instead of S phasors.
//
// A block takes runs of one antenna's points.  Points are screened with the
// conservative early test as they stream in; those it cannot cull are listed, and
// 128 at a time get the exact geometry, one per thread, so no lane sits out the
// expensive part (on a typical scene one point in ten is live).  The 128 points'
// contributions are then sorted by cell in shared memory and added up by groups
// of eight lanes, one per moment, in list order: no floating-point atomics, and the
// same bits on every run.  (Sums by each
// warp alone, over the set bits of its match masks and without barriers, took as long for
// the pre-cull's lists and 40 us longer for 64 antennas x 295000 screened points.)
//
// Cells are kept in kTraceSlots slots, cell k in slot k mod kTraceSlots.  (128 slots took 10
// to 13% longer on scenes that need a dozen cells.)  Points whose cells share a slot are
// 2.4 m of path or more apart (at 4 GHz swept): the block then leaves the rest of its share
// (of a list; a screened share as a whole) to trace_direct, at the cost of a recurrence over
// the samples but whatever the scene's depth.  Measured on 64 antennas x 262144 points, 10% live,
// x 128 samples: 68 us through the cells in a scene 0.2 m deep, 106 us in one 3 m deep
// (several passes over the points, each with its own cells, took 197 us there and 851 us in
// one 30 m deep).
#pragma once

#include "range_cells.cuh"
#include "tracer_geometry.cuh"

namespace geraf {
namespace tracer {

constexpr int kTraceThreads = 128;
constexpr int kTraceWarps = kTraceThreads / 32;
constexpr int kTracePer = 4;  // points per thread and screening pass
constexpr int kTraceQ = MomentCells::Q;
constexpr int kTraceSlots = 64;
constexpr int kTraceEmpty = INT32_MIN + 1;  // no path has this cell
// Not for the cells, whose sums of powers would make a NaN of it: an infinite amplitude; or a
// path whose cell's number no int holds (4e7 m at 4 GHz swept).
constexpr int kTraceOut = INT32_MIN + 2;
constexpr int kTraceRow = kTraceQ + 2;      // float2 per contribution row: 80 bytes, conflict-free

constexpr double kTraceMinKappa = 1e-6;     // cells per metre

struct TraceConsts {
  double K, b;       // phase of carrier and middle sample, cycles per metre and bias
  double k1, b1;     // phase step per sample
  double kappa, inv_kappa;  // cells per metre
  double theta_step;
  int S;
};

inline TraceConsts trace_consts(double k0, double b0, double k1, double b1, int64_t S) {
  TraceConsts t;
  const double mid = 0.5 * static_cast<double>(S - 1);
  t.K = k0 + mid * k1;
  t.b = b0 + mid * b1;
  t.k1 = k1;
  t.b1 = b1;
  // without a sweep every path is in cell 0
  const double kappa = MomentCells::kOver * static_cast<double>(S) * (k1 < 0.0 ? -k1 : k1);
  t.kappa = kappa > kTraceMinKappa ? kappa : kTraceMinKappa;
  t.inv_kappa = 1.0 / t.kappa;
  t.theta_step = 2.0 * 3.14159265358979323846 * k1 / t.kappa;
  t.S = static_cast<int>(S);
  return t;
}

// A share's result: moments of the cells in its slots (tag kTraceEmpty: unused), and a
// row of S samples when has_row says so.
struct TraceRecord {
  float2 moments[kTraceSlots][kTraceQ];
  int tag[kTraceSlots];
  int has_row;
  int pad[15];
};

struct TraceSmem {
  float2 rows[kTraceThreads][kTraceRow];
  float2 moments[kTraceSlots][kTraceQ];
  int4 hist[kTraceSlots];  // per warp
  int start[kTraceSlots + 1];
  int tag[kTraceSlots];
  int list[kTraceThreads * (kTracePer + 1)];
  alignas(16) int counts[kTracePer * kTraceWarps];
};

// A cell's moments as sample n sees them.
__device__ __forceinline__ float2 cell_sample(const TraceConsts& c, int k, const float2* m, const float* g, int n) {
  const double ph = (n - 0.5 * (c.S - 1)) * fma(c.k1, k * c.inv_kappa, c.b1);
  const float2 e = cis_cycles(static_cast<float>(ph - rint(ph)));
  float2 ev = make_float2(0.0f, 0.0f), od = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int q = 0; q < kTraceQ; q += 2) {
    ev = ffma2(make_float2(g[q], g[q]), m[q], ev);
    od = ffma2(make_float2(g[q + 1], g[q + 1]), m[q + 1], od);
  }
  return cmul(e, make_float2(ev.x - od.y, ev.y + od.x));
}

__device__ __forceinline__ void trace_begin(TraceSmem& sm) {
  for (int i = threadIdx.x; i < kTraceSlots * kTraceQ; i += kTraceThreads) {
    (&sm.moments[0][0])[i] = make_float2(0.0f, 0.0f);
  }
  for (int i = threadIdx.x; i < kTraceSlots; i += kTraceThreads) {
    sm.tag[i] = kTraceEmpty;
    sm.hist[i] = make_int4(0, 0, 0, 0);
  }
  __syncthreads();
}

// One batch: thread t holds a live contribution w at cell k, offset x (or none).  False, on
// every thread, when two cells want one slot, whatever the order of the threads, or one is
// kTraceOut: nothing of the batch is then added, and with KEEP the slots are as they were.
template <bool KEEP>
__device__ __forceinline__ bool trace_batch(TraceSmem& sm, bool live, float2 w, int k, float x) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slot = k & (kTraceSlots - 1);
  int held = k;
  if (live) held = sm.tag[slot];
  if (held == kTraceEmpty) sm.tag[slot] = k;  // one of them stays
  const unsigned same = __match_any_sync(0xffffffffu, live ? slot : kTraceSlots);
  const int rank = __popc(same & ((1u << lane) - 1u));
  if (live && rank == 0) reinterpret_cast<int*>(&sm.hist[slot])[warp] = __popc(same);
  __syncthreads();
  if (warp == 0) {  // exclusive prefix over (slot, warp), two slots per lane
    const int4 a = sm.hist[2 * lane], b = sm.hist[2 * lane + 1];
    const int sa = a.x + a.y + a.z + a.w, sb = b.x + b.y + b.z + b.w;
    int run = sa + sb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += y;
    }
    const int e = run - sa - sb;
    sm.start[2 * lane] = e;
    sm.start[2 * lane + 1] = e + sa;
    sm.hist[2 * lane] = make_int4(e, e + a.x, e + a.x + a.y, e + a.x + a.y + a.z);
    const int f = e + sa;
    sm.hist[2 * lane + 1] = make_int4(f, f + b.x, f + b.x + b.y, f + b.x + b.y + b.z);
    if (lane == 31) sm.start[kTraceSlots] = run;
  }
  __syncthreads();
  const bool other = live && (sm.tag[slot] != k || k == kTraceOut);
  if (live) {  // the contribution row w x^q, at its place in cell order
    const int place = reinterpret_cast<const int*>(&sm.hist[slot])[warp] + rank;
    float4* dst = reinterpret_cast<float4*>(&sm.rows[place][0]);
    float2 v = w;
#pragma unroll
    for (int q = 0; q < kTraceQ; q += 2) {
      const float2 u = make_float2(v.x * x, v.y * x);
      dst[q / 2] = make_float4(v.x, v.y, u.x, u.y);
      v = make_float2(u.x * x, u.y * x);
    }
  }
  if (__syncthreads_or(other)) {
    if (KEEP && held == kTraceEmpty) sm.tag[slot] = kTraceEmpty;  // the slots that this batch took
    return false;
  }
  for (int i = threadIdx.x; i < kTraceSlots; i += kTraceThreads) sm.hist[i] = make_int4(0, 0, 0, 0);
  const int q = threadIdx.x & (kTraceQ - 1);
  for (int s = threadIdx.x / kTraceQ; s < kTraceSlots; s += kTraceThreads / kTraceQ) {
    const int i0 = sm.start[s], i1 = sm.start[s + 1];
    if (i0 == i1) continue;
    // the batch's sum first, then onto the cell's: two levels, so that a cell of hundreds of
    // thousands of points errs by the square root of its batches, not of its points
    float2 acc = sm.rows[i0][q];
#pragma unroll 4
    for (int i = i0 + 1; i < i1; ++i) acc = fadd2(acc, sm.rows[i][q]);
    sm.moments[s][q] = fadd2(sm.moments[s][q], acc);
  }
  __syncthreads();
  return true;
}

// A point and its contribution.
struct TracePoint {
  float nrm[3], pt[3], sigma;
};

template <typename T>
__device__ __forceinline__ void load_point(const T* normals, const T* points, int64_t q, float* nrm, float* pt) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    nrm[a] = ld_f(normals, q * 3 + a);
    pt[a] = ld_f(points, q * 3 + a);
  }
}

// Amplitude and path length of a live point.
__device__ __forceinline__ bool trace_path(const float* txp, const float* rxp, const TracePoint& t, float& amp, double& d) {
  PairGeom g;
  if (!pair_geometry(txp, rxp, t.nrm, t.pt, g)) return false;
  amp = t.sigma * g.align / sq(g.dist);
  double st = 0.0, sr = 0.0;
#pragma unroll
  for (int a = 2; a >= 0; --a) {
    const double dt = static_cast<double>(txp[a]) - static_cast<double>(t.pt[a]);
    const double dr = static_cast<double>(rxp[a]) - static_cast<double>(t.pt[a]);
    st = fma(dt, dt, st);
    sr = fma(dr, dr, sr);
  }
  d = sqrt_f64_fast(st) + sqrt_f64_fast(sr);
  return true;
}

__device__ __forceinline__ bool trace_point(const TraceConsts& c, const float* txp, const float* rxp, const TracePoint& t,
                                            float2& w, int& cell, float& x) {
  float amp;
  double d;
  if (!trace_path(txp, rxp, t, amp, d)) return false;
  const double ph = fma(d, c.K, c.b);
  const double u = d * c.kappa, ku = rint(u);
  if (fabs(ku) < 1073741824.0 && fabsf(amp) < INFINITY) cell = static_cast<int>(ku);
  else cell = ku != ku || amp != amp ? 0 : kTraceOut;  // a NaN may go anywhere
  x = static_cast<float>(u - ku);
  const float2 e = cis_cycles_fast(static_cast<float>(ph - rint(ph)));
  w = make_float2(amp * e.x, amp * e.y);
  return true;
}

// `count` positions in batches of consecutive ones: for points of
// which most are live (the pre-cull's list).  index_of gives the point at a position, or -1 when
// it is out of bounds.  The next batch's points are loaded while one is summed.  Returns how
// many positions are in the moments: all, or those before the first batch that is not.
template <typename T, typename IndexOf, typename SigmaOf>
__device__ __forceinline__ int trace_all(TraceSmem& sm, const TraceConsts& c, const T* normals, const T* points,
                                          const float* txp, const float* rxp, int count, IndexOf index_of,
                                          SigmaOf sigma_of) {
  TracePoint next;
  int64_t next_q = -1;
  auto load = [&](int pos) {
    next_q = pos < count ? index_of(pos) : -1;
    if (next_q >= 0) {
      load_point(normals, points, next_q, next.nrm, next.pt);
      next.sigma = sigma_of(next_q);
    }
  };
  load(threadIdx.x);
  for (int p0 = 0; p0 < count; p0 += kTraceThreads) {
    float2 w = make_float2(0.0f, 0.0f);
    float x = 0.0f;
    int cell = 0;
    const bool live = next_q >= 0 && trace_point(c, txp, rxp, next, w, cell, x);
    load(p0 + kTraceThreads + threadIdx.x);
    if (!trace_batch<true>(sm, live, w, cell, x)) return p0;
  }
  return count;
}

// `count` consecutive points (their arrays from the first one on; inb may be null), screened first: those that the early test cannot cull are listed, 512
// positions at a time, and served in batches of 128.  False when a batch was not added.
template <typename T>
__device__ __forceinline__ bool trace_screened(TraceSmem& sm, const TraceConsts& c, const T* normals, const T* points,
                                               const T* sigmas, const uint8_t* inb, const float* txp, const float* rxp,
                                               int count) {
  static_assert(kTracePer == 4, "one 16-byte load per warp's counts");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int listed = 0;
  float nrm[kTracePer][3], pt[kTracePer][3];
  unsigned in = 0;  // bit j: point j of the thread is in bounds
  auto load = [&](int p0) {  // of the next pass, in flight while batches are summed
    in = 0;
    const int rest = count - p0 - static_cast<int>(threadIdx.x);
    const T* pn = normals + (static_cast<int64_t>(p0) + threadIdx.x) * 3;
    const T* pp = points + (static_cast<int64_t>(p0) + threadIdx.x) * 3;
    const uint8_t* pb = inb != nullptr ? inb + p0 + threadIdx.x : nullptr;
#pragma unroll
    for (int j = 0; j < kTracePer; ++j) {
      if (j * kTraceThreads < rest && (pb == nullptr || pb[j * kTraceThreads])) {
        in |= 1u << j;
        load_point(pn, pp, j * kTraceThreads, nrm[j], pt[j]);
      }
    }
  };
  load(0);
  for (int p0 = 0; p0 < count; p0 += kTraceThreads * kTracePer) {
    // Lane l of warp w keeps position p0 + 128 j + 32 w + l where bit l of its mask[j] is set.
    // The list's order is that of (warp, j, lane): the same on every run.
    unsigned mask[kTracePer];
#pragma unroll
    for (int j = 0; j < kTracePer; ++j) {
      mask[j] = __ballot_sync(0xffffffffu, ((in >> j) & 1u) && !surely_culled(txp, rxp, nrm[j], pt[j]));
    }
    if (lane == 0) {
      *reinterpret_cast<int4*>(&sm.counts[warp * kTracePer]) =
          make_int4(__popc(mask[0]), __popc(mask[1]), __popc(mask[2]), __popc(mask[3]));
    }
    __syncthreads();
    int before = listed;
#pragma unroll
    for (int w = 0; w < kTraceWarps; ++w) {
      const int4 n = *reinterpret_cast<const int4*>(&sm.counts[w * kTracePer]);
      if (w == warp) {
        const int at[kTracePer] = {before, before + n.x, before + n.x + n.y, before + n.x + n.y + n.z};
#pragma unroll
        for (int j = 0; j < kTracePer; ++j) {
          if ((mask[j] >> lane) & 1u) {
            sm.list[at[j] + __popc(mask[j] & ((1u << lane) - 1u))] = p0 + j * kTraceThreads + static_cast<int>(threadIdx.x);
          }
        }
      }
      before += n.x + n.y + n.z + n.w;
    }
    listed = before;
    load(p0 + kTraceThreads * kTracePer);
    __syncthreads();
    const bool drain = p0 + kTraceThreads * kTracePer >= count;
    while (listed >= kTraceThreads || (drain && listed > 0)) {
      const int cnt = min(listed, kTraceThreads);
      listed -= cnt;
      bool live = false;
      float2 w = make_float2(0.0f, 0.0f);
      float x = 0.0f;
      int cell = 0;
      if (threadIdx.x < cnt) {
        const int q = sm.list[listed + threadIdx.x];
        TracePoint t;
        load_point(normals, points, q, t.nrm, t.pt);
        t.sigma = ld_f(sigmas, q);
        live = trace_point(c, txp, rxp, t, w, cell, x);
      }
      if (!trace_batch<false>(sm, live, w, cell, x)) return false;
    }
  }
  return true;
}

// trace_direct: samples of a thread, and groups of them that one sweep over the points covers.
constexpr int kDirectK = 16;
constexpr int kDirectGroups = 16;

// Antennas of so few points take it as a whole where there are many of them: a point costs at most 2 S
// slots there, a cell about 35 S when the moments become samples, and the record between the two
// kernels goes.  Forward of 8853 antennas x 39 points x 128 samples, 10 m deep, 128 us through
// the cells and 60 so, 3072 x 384 x 128 64 and 58 us; past that the cells win (3072 x 384 x 512, all live: 100 and 143 us,
// but 68 and 45 with a tenth of 256 points live).  The batched tracer keeps its short antennas in the cells (13347 of 9
// points x 512: 219 us, 310 so).
constexpr int kDirectPoints = 384;

struct DirectSmem {
  union {
    struct {
      float2 seeds[kDirectGroups][kTraceThreads];
      float2 zeta[kTraceThreads];
    };
    float2 red[kDirectK * (kTraceThreads + kDirectGroups)];  // [G K][L + 1], off each other's banks
  };
  int counts[kTraceWarps];
};


// Samples without cells: store(n, sum over the live points of positions [0, count)).  A tile of
// 128 points leaves each group of 16 samples its start phasors, and thread (group, lane) runs its
// lane's points through its samples by the recurrence of rotate_accumulate, in two levels of
// sums (a tile's, the share's).  A sweep over the points covers 256 samples.  About 2 issue slots
// per live (point, sample): 64 antennas x 262144 live points x 128 samples take 634 us,
// whatever their paths.
template <typename T, typename IndexOf, typename SigmaOf, typename Store>
__device__ __forceinline__ void trace_direct(DirectSmem& sm, const TraceConsts& c, const T* normals, const T* points,
                                             const float* txp, const float* rxp, int64_t count, IndexOf index_of,
                                             SigmaOf sigma_of, Store store) {
  constexpr int K = kDirectK;
  int G = 1;
  while (G < kDirectGroups && G * K < c.S) G *= 2;
  const int L = kTraceThreads / G;
  const int group = threadIdx.x / L, in_group = threadIdx.x % L;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double mid = 0.5 * (c.S - 1);
  for (int n0 = 0; n0 < c.S; n0 += G * K) {
    float2 acc[K], sum[K];
#pragma unroll
    for (int m = 0; m < K; ++m) acc[m] = sum[m] = make_float2(0.0f, 0.0f);
    for (int64_t p0 = 0; p0 < count; p0 += kTraceThreads) {
      TracePoint t;
      const int64_t q = p0 + threadIdx.x < count ? index_of(p0 + threadIdx.x) : -1;
      if (q >= 0) {
        load_point(normals, points, q, t.nrm, t.pt);
        t.sigma = sigma_of(q);
      }
      float2 w = make_float2(0.0f, 0.0f), zt = w, zk = w;
      float amp;
      double d;
      const bool live = q >= 0 && !surely_culled(txp, rxp, t.nrm, t.pt) && trace_path(txp, rxp, t, amp, d);
      if (live) {
        const double step = fma(d, c.k1, c.b1), kc = step * K;
        const double start = fma(d, c.K, c.b) + (n0 - mid) * step;
        const float2 e = cis_cycles_fast(static_cast<float>(start - rint(start)));
        w = make_float2(amp * e.x, amp * e.y);
        zt = cis_cycles(static_cast<float>(step - rint(step)));
        zk = cis_cycles(static_cast<float>(kc - rint(kc)));
      }
      const unsigned ballot = __ballot_sync(0xffffffffu, live);
      if (lane == 0) sm.counts[warp] = __popc(ballot);
      __syncthreads();
      int slot = __popc(ballot & ((1u << lane) - 1u)), total = 0;
#pragma unroll
      for (int k = 0; k < kTraceWarps; ++k) {
        if (k < warp) slot += sm.counts[k];
        total += sm.counts[k];
      }
      if (live) {
        sm.zeta[slot] = zt;
        for (int k = 0; k < G; ++k) {
          sm.seeds[k][slot] = w;
          w = cmul(w, zk);
        }
      }
      __syncthreads();
      rotate_tile<K>(sm.seeds[group], sm.zeta, in_group, L, total, acc);
#pragma unroll
      for (int m = 0; m < K; ++m) sum[m] = fadd2(sum[m], acc[m]);
      __syncthreads();
    }
#pragma unroll
    for (int m = 0; m < K; ++m) sm.red[(group * K + m) * (L + 1) + in_group] = sum[m];
    __syncthreads();
    // few samples: several lanes of a warp to a sum (one pass over the sums then)
    const int per = max(1, kTraceThreads / (G * K));
    for (int i = threadIdx.x / per; i < G * K; i += kTraceThreads / per) {
      double2 x = make_double2(0.0, 0.0);
      for (int k = threadIdx.x % per; k < L; k += per) {
        const float2 y = sm.red[i * (L + 1) + k];
        x.x += y.x;
        x.y += y.y;
      }
      for (int o = per / 2; o > 0; o >>= 1) {
        x.x += __shfl_xor_sync(0xffffffffu, x.x, o);
        x.y += __shfl_xor_sync(0xffffffffu, x.y, o);
      }
      if (n0 + i < c.S && threadIdx.x % per == 0) {
        store(n0 + i, make_float2(static_cast<float>(x.x), static_cast<float>(x.y)));
      }
    }
    __syncthreads();
  }
}

__device__ __forceinline__ void trace_store(const TraceSmem& sm, TraceRecord* rec, bool has_row) {
  __syncthreads();
  for (int i = threadIdx.x; i < kTraceSlots * kTraceQ; i += kTraceThreads) {
    if (sm.tag[i / kTraceQ] != kTraceEmpty) (&rec->moments[0][0])[i] = (&sm.moments[0][0])[i];
  }
  for (int i = threadIdx.x; i < kTraceSlots; i += kTraceThreads) rec->tag[i] = sm.tag[i];
  if (threadIdx.x == 0) rec->has_row = has_row ? 1 : 0;
  __syncthreads();
}

// Samples [n_begin, n_begin + kFinishSamples) of one antenna from its runs' records, by
// kFinishThreads threads.  Per slot the cells are taken in ascending order, one per round
// (one round, unless runs of the antenna lie more than kTraceSlots cells apart).
//
// A call has few such blocks (one per antenna), so each is bound by latency: four
// groups of threads take every fourth run's moments, then every fourth slot's cells, and
// add up in a fixed order, in FP64 as the partial sums of the other forms are.  13 antennas x 78 runs: 44 us with one group, 14 us with four;
// 64 antennas x 23 runs: 19.5 and 10.9 us.
constexpr int kFinishSamples = 256;
constexpr int kFinishGroups = 4;
constexpr int kFinishThreads = kFinishSamples * kFinishGroups;

struct FinishSmem {
  union {
    double4 part[kFinishGroups][kTraceSlots][kTraceQ / 2];
    double2 acc[kFinishGroups][kFinishSamples];
  };
  float2 mom[kTraceSlots][kTraceQ];
  int next[kFinishGroups][kTraceSlots], top[kFinishGroups][kTraceSlots];
  int tag[kTraceSlots];
};

template <typename T>
__device__ __forceinline__ void trace_finish(const TraceConsts& c, const TraceRecord* rec, const float2* rows,
                                             int64_t runs, float divisor, int n_begin, int n_end, T* out_r, T* out_i) {
  __shared__ FinishSmem sm;
  static_assert(kFinishSamples == kTraceSlots * kTraceQ / 2, "a thread of a group per slot and pair of moments");
  const int group = threadIdx.x / kFinishSamples, in_group = threadIdx.x % kFinishSamples;
  const int slot = in_group / (kTraceQ / 2), pair = in_group % (kTraceQ / 2);
  const int n = n_begin + in_group;
  const bool mine = n < n_end;
  double2 acc = make_double2(0.0, 0.0);
  auto add = [](double2& s, float2 x) {
    s.x += x.x;
    s.y += x.y;
  };
  float g[kTraceQ];
  bool rowed = false;
  for (int64_t r = threadIdx.x; r < runs; r += kFinishThreads) rowed = rowed || rec[r].has_row != 0;
  if (__syncthreads_or(rowed) && mine) {
    for (int64_t r = group; r < runs; r += kFinishGroups) {
      if (rec[r].has_row) add(acc, rows[r * c.S + n]);
    }
  }
  if (mine) cell_basis<kTraceQ>(c.theta_step * (n - 0.5 * (c.S - 1)), g);
  int done = INT32_MIN;
  for (;;) {
    // the slot's lowest cell above the one done, and whether higher ones follow
    int next = INT32_MAX, top = INT32_MIN;
#pragma unroll 4
    for (int64_t r = group + pair * kFinishGroups; r < runs; r += kFinishGroups * kTraceQ / 2) {
      const int t = rec[r].tag[slot];
      if (t != kTraceEmpty && t > done) {
        next = min(next, t);
        top = max(top, t);
      }
    }
#pragma unroll
    for (int o = 1; o < kTraceQ / 2; o <<= 1) {
      next = min(next, __shfl_xor_sync(0xffffffffu, next, o));
      top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    }
    if (pair == 0) {
      sm.next[group][slot] = next;
      sm.top[group][slot] = top;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kFinishGroups; ++k) {
      next = min(next, sm.next[k][slot]);
      top = max(top, sm.top[k][slot]);
    }
    double4 m = make_double4(0.0, 0.0, 0.0, 0.0);
    if (next != INT32_MAX) {
#pragma unroll 8
      for (int64_t r = group; r < runs; r += kFinishGroups) {
        const int t = rec[r].tag[slot];
        const float4 y = reinterpret_cast<const float4*>(&rec[r].moments[slot][0])[pair];
        const bool take = t == next;  // unused slots hold no moments
        m.x += take ? y.x : 0.0f;
        m.y += take ? y.y : 0.0f;
        m.z += take ? y.z : 0.0f;
        m.w += take ? y.w : 0.0f;
      }
    }
    sm.part[group][slot][pair] = m;
    const bool more = next != INT32_MAX && top > next;
    done = next;
    const bool again = __syncthreads_or(more) != 0;
    if (group == 0) {
#pragma unroll
      for (int k = 1; k < kFinishGroups; ++k) {
        const double4 y = sm.part[k][slot][pair];
        m.x += y.x;
        m.y += y.y;
        m.z += y.z;
        m.w += y.w;
      }
      reinterpret_cast<float4*>(&sm.mom[slot][0])[pair] =
          make_float4(static_cast<float>(m.x), static_cast<float>(m.y), static_cast<float>(m.z), static_cast<float>(m.w));
      if (pair == 0) sm.tag[slot] = next;  // INT32_MAX: none
    }
    __syncthreads();
    if (mine) {
      for (int k = group; k < kTraceSlots; k += kFinishGroups) {
        if (sm.tag[k] != INT32_MAX) add(acc, cell_sample(c, sm.tag[k], sm.mom[k], g, n));
      }
    }
    if (!again) break;
    __syncthreads();
  }
  sm.acc[group][in_group] = acc;  // over part, last read before the last barrier
  __syncthreads();
  if (group == 0 && mine) {
#pragma unroll
    for (int k = 1; k < kFinishGroups; ++k) {
      acc.x += sm.acc[k][in_group].x;
      acc.y += sm.acc[k][in_group].y;
    }
    out_r[n] = from_f<T>(static_cast<float>(acc.x) / divisor);
    out_i[n] = from_f<T>(static_cast<float>(acc.y) / divisor);
  }
}

// The same for many antennas of few shares each, where a block per antenna mostly waits: a warp
// per antenna brings the used slots of its shares together in shared memory and walks them
// for 64 samples at a time.  What depends on the sample alone is in shared memory too: its
// basis, its phasor e^{j 2 pi n' b1}, and the cells' phasors, which are roots of unity: with
// kappa = 2 S |k1|, cell k turns sample n by (2 n - S + 1) k / (4 S) cycles.  49152 antennas x 300
// points x 64 samples: 1755 us by blocks of 1024 threads, 104 us so; 5739 x 1396 x 512, forward: 485 and
// 125 us, 13347 x 9 x 512 in one batch: 1032 and 216 us (137 and 310 us with one sample per lane and 128 threads).
constexpr int kFewThreads = 256;  // (128: 12 warps per SM at 512 samples, twice that so)
constexpr int kFewSamples = 1024;  // 112 KB of shared memory; the product of a turn and a cell stays below 2^24
constexpr int kFewShares = 16;
static_assert(MomentCells::kOver == 2, "cells of 1 / (2 S k1)");

struct FewWarp {
  float4 moments[kTraceSlots][kTraceQ / 2];  // of the used slots
  int slot[kTraceSlots], cell[kTraceSlots];  // cells mod 4 S
};
struct FewTable {
  FewWarp* warp;   // the calling warp's
  float* basis;    // [S][kTraceQ]
  float2* offset;  // [S]
  float2* root;    // [4 S], root i at root_at(i)
};
// Lanes read roots at a stride of twice their cell: spread so that they miss each other's banks.
__device__ __forceinline__ int root_at(int i) { return i + (i >> 4); }

inline size_t few_smem_bytes(int64_t S) {
  return kFewThreads / 32 * sizeof(FewWarp) + static_cast<size_t>(S) * (kTraceQ * sizeof(float) + 5 * sizeof(float2)) +
         static_cast<size_t>(S / 4 + 1) * sizeof(float2);
}

__device__ __forceinline__ FewTable few_table(const TraceConsts& c, unsigned char* smem) {
  FewTable f;
  f.warp = reinterpret_cast<FewWarp*>(smem) + (threadIdx.x >> 5);
  f.basis = reinterpret_cast<float*>(smem + kFewThreads / 32 * sizeof(FewWarp));
  f.offset = reinterpret_cast<float2*>(f.basis + c.S * kTraceQ);
  f.root = f.offset + c.S;
  for (int n = threadIdx.x; n < c.S; n += kFewThreads) {
    const double mid = n - 0.5 * (c.S - 1);
    float g[kTraceQ];
    cell_basis<kTraceQ>(c.theta_step * mid, g);
#pragma unroll
    for (int q = 0; q < kTraceQ; ++q) f.basis[n * kTraceQ + q] = g[q];
    const double ph = mid * c.b1;
    f.offset[n] = cis_cycles(static_cast<float>(ph - rint(ph)));
  }
  for (int i = threadIdx.x; i < 4 * c.S; i += kFewThreads) {
    const double ph = copysign(static_cast<double>(i) / (4 * c.S), c.k1);
    f.root[root_at(i)] = cis_cycles(static_cast<float>(ph - rint(ph)));
  }
  __syncthreads();
  return f;
}

// Used slots of `shares` shares into w, their moments added up; returns their number, or -1
// where two shares have other cells in a slot.
__device__ __forceinline__ int few_slots(const TraceRecord* rec, int shares, int M, FewWarp& w) {
  const int lane = threadIdx.x & 31;
  int tag[kTraceSlots / 32], used = 0;
  bool clash = false;
  __syncwarp();
#pragma unroll
  for (int h = 0; h < kTraceSlots / 32; ++h) tag[h] = rec[0].tag[h * 32 + lane];
#pragma unroll 2
  for (int r = 1; r < shares; ++r) {
#pragma unroll
    for (int h = 0; h < kTraceSlots / 32; ++h) {
      const int t = rec[r].tag[h * 32 + lane];
      if (t == kTraceEmpty) continue;
      clash = clash || (tag[h] != kTraceEmpty && tag[h] != t);
      tag[h] = t;
    }
  }
  if (__any_sync(0xffffffffu, clash)) return -1;
#pragma unroll
  for (int h = 0; h < kTraceSlots / 32; ++h) {
    const unsigned set = __ballot_sync(0xffffffffu, tag[h] != kTraceEmpty);
    if (tag[h] != kTraceEmpty) {
      const int e = used + __popc(set & ((1u << lane) - 1u));
      w.slot[e] = h * 32 + lane;
      w.cell[e] = (tag[h] % M + M) % M;
    }
    used += __popc(set);
  }
  __syncwarp();
  constexpr int kParts = kTraceQ / 2;
#pragma unroll 2
  for (int i = lane; i < used * kParts; i += 32) {
    const int slot = w.slot[i / kParts];
    const float4 first = reinterpret_cast<const float4*>(&rec[0].moments[slot][0])[i % kParts];
    if (shares == 1) {
      w.moments[i / kParts][i % kParts] = first;
      continue;
    }
    double4 m = make_double4(0.0, 0.0, 0.0, 0.0);
#pragma unroll 4
    for (int r = 0; r < shares; ++r) {
      const float4 y = reinterpret_cast<const float4*>(&rec[r].moments[slot][0])[i % kParts];
      const bool take = rec[r].tag[slot] != kTraceEmpty;  // unused slots hold no moments
      m.x += take ? y.x : 0.0f;
      m.y += take ? y.y : 0.0f;
      m.z += take ? y.z : 0.0f;
      m.w += take ? y.w : 0.0f;
    }
    w.moments[i / kParts][i % kParts] =
        make_float4(static_cast<float>(m.x), static_cast<float>(m.y), static_cast<float>(m.z), static_cast<float>(m.w));
  }
  __syncwarp();
  return used;
}

// kPer samples per lane share the reads of the moments.
template <int kPer, typename T>
__device__ __forceinline__ void finish_few_samples(const TraceConsts& c, const FewTable& f, const TraceRecord* rec,
                                                 const float2* rows, int shares, float divisor, T* out_r, T* out_i) {
  const int lane = threadIdx.x & 31;
  const int M = 4 * c.S;
  const float inv_m = 1.0f / static_cast<float>(M);
  FewWarp& w = *f.warp;
  // the shares as one where their cells agree, as in all but deep scenes they do, else one by one
  int used = shares > 0 ? few_slots(rec, shares, M, w) : 0;
  const bool together = used >= 0;
  for (int n0 = 0; n0 < c.S; n0 += 32 * kPer) {
    int n[kPer], turn[kPer];
    float g[kPer][kTraceQ];
    double2 acc[kPer];
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      n[u] = min(n0 + 32 * u + lane, c.S - 1);
      turn[u] = 2 * n[u] - c.S + 1 + (2 * n[u] < c.S - 1 ? M : 0);
      acc[u] = make_double2(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < kTraceQ; q += 4) {
        const float4 y = *reinterpret_cast<const float4*>(&f.basis[n[u] * kTraceQ + q]);
        g[u][q] = y.x;
        g[u][q + 1] = y.y;
        g[u][q + 2] = y.z;
        g[u][q + 3] = y.w;
      }
    }
    for (int r = 0; r < (together ? 1 : shares); ++r) {
      if (!together) used = few_slots(rec + r, 1, M, w);
      float2 sum[kPer];
#pragma unroll
      for (int u = 0; u < kPer; ++u) sum[u] = make_float2(0.0f, 0.0f);
      for (int e = 0; e < used; ++e) {
        float4 y[kTraceQ / 2];
#pragma unroll
        for (int q = 0; q < kTraceQ / 2; ++q) y[q] = w.moments[e][q];
        const int cell = w.cell[e];
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
          // turn * cell mod M: a product below 2^24, its quotient off by one at most
          const int product = turn[u] * cell;
          int i = product - static_cast<int>(static_cast<float>(product) * inv_m) * M;
          i += i < 0 ? M : 0;
          i -= i >= M ? M : 0;
          float2 ev = make_float2(0.0f, 0.0f), od = make_float2(0.0f, 0.0f);
#pragma unroll
          for (int q = 0; q < kTraceQ; q += 2) {
            ev = ffma2(make_float2(g[u][q], g[u][q]), make_float2(y[q / 2].x, y[q / 2].y), ev);
            od = ffma2(make_float2(g[u][q + 1], g[u][q + 1]), make_float2(y[q / 2].z, y[q / 2].w), od);
          }
          sum[u] = fadd2(sum[u], cmul(f.root[root_at(i)], make_float2(ev.x - od.y, ev.y + od.x)));
        }
      }
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        sum[u] = cmul(sum[u], f.offset[n[u]]);
        acc[u].x += sum[u].x;
        acc[u].y += sum[u].y;
      }
    }
    for (int r = 0; r < shares; ++r) {
      if (rec[r].has_row == 0) continue;
#pragma unroll
      for (int u = 0; u < kPer; ++u) {
        const float2 y = rows[static_cast<int64_t>(r) * c.S + n[u]];
        acc[u].x += y.x;
        acc[u].y += y.y;
      }
    }
#pragma unroll
    for (int u = 0; u < kPer; ++u) {
      if (n0 + 32 * u + lane >= c.S) continue;
      out_r[n[u]] = from_f<T>(static_cast<float>(acc[u].x) / divisor);
      out_i[n[u]] = from_f<T>(static_cast<float>(acc[u].y) / divisor);
    }
  }
}

template <typename T>
__device__ __forceinline__ void trace_finish_few(const TraceConsts& c, const FewTable& f, const TraceRecord* rec,
                                                 const float2* rows, int shares, float divisor, T* out_r, T* out_i) {
  if (c.S > 32) finish_few_samples<2>(c, f, rec, rows, shares, divisor, out_r, out_i);
  else finish_few_samples<1>(c, f, rec, rows, shares, divisor, out_r, out_i);
}

}  // namespace tracer
}  // namespace geraf
