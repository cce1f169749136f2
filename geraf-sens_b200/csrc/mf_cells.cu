// MIXED matched filter through range cells (range_cells.cuh): the forward
// evaluates each pair's sample sum as a polynomial of the path length in the
// pair's cell, from a per-antenna table of cell coefficients.
//
// Launches of the forward:
//   1. cell_prep_kernel: the voxels' bounding box (per-block partials) and the
//      interpolation basis of every sample;
//   2. mf_cell_table_kernel: per antenna, the cells its path lengths to the box
//      can reach, and their coefficients;
//   3. mf_cell_gather_kernel: the pairs;
//   4. the direct kernel (mf_kernels.cu), which returns at once unless step 2
//      found an antenna whose cells do not fit (more than kMaxCells, a leg beyond
//      kMaxLeg, non-finite positions): its band is only known on the device.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "kernels.h"
#include "range_cells.cuh"

namespace geraf {
namespace {

constexpr int kMaxCells = 96;    // cells per antenna: 1.8 m of path at 4 GHz swept
constexpr int kPrepBlocks = 256;
constexpr int kTableThreads = 128;
constexpr int kTableTile = 256;  // samples staged at a time by the table kernel

struct CellHead {
  int bad;  // set when some antenna's cells do not fit: the direct kernel runs instead
  int pad[3];
  double center[3];  // of the voxels' box: the origin of AntMeta and of the pairs' legs
};

struct AntMeta {
  double t[4];  // -2 t, |t|^2 from the centre, in units of 2^-20 m (biased, see leg_length)
  double r[4];
  int c0, cells;  // first cell (absolute) and number of cells
  int same_tx;    // the transmitter equals the preceding antenna's
  int pad;
};
static_assert(sizeof(AntMeta) == 80, "copied in 16-byte units");

size_t up256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

struct CellLayout {
  size_t head, bbox, basis, meta, table, partial, total;
};

CellLayout cell_layout(int64_t A, int64_t S, int64_t partial_bytes) {
  CellLayout l;
  l.head = 0;
  l.bbox = 256;
  l.basis = up256(l.bbox + kPrepBlocks * 6 * sizeof(float));
  l.meta = up256(l.basis + static_cast<size_t>(S) * GatherCells::Q * sizeof(float));
  l.table = up256(l.meta + static_cast<size_t>(A) * sizeof(AntMeta));
  l.partial = up256(l.table + static_cast<size_t>(A) * kMaxCells * GatherCells::Q * sizeof(float2));
  l.total = l.partial + up256(static_cast<size_t>(partial_bytes));
  return l;
}

// ---------------------------------------------------------------------------
template <typename T>
struct PrepP {
  const T* voxel;  // [3, N]
  int64_t N;
  int S;
  double theta_step;  // theta of one sample, 2 pi k1 / kappa
  float* bbox;        // [blocks][6]
  float* basis;       // [S][Q]
  CellHead* head;
};

template <typename T, int Q>
__global__ void __launch_bounds__(256) cell_prep_kernel(const PrepP<T> p) {
  __shared__ float red[8][6];
  const int64_t gid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  if (gid == 0) p.head->bad = 0;
  for (int64_t n = gid; n < p.S; n += step) {
    float g[Q];
    cell_basis<Q>(p.theta_step * (static_cast<double>(n) - 0.5 * (p.S - 1)), g);
#pragma unroll
    for (int q = 0; q < Q; ++q) p.basis[n * Q + q] = g[q];
  }
  float b[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  for (int64_t v = gid; v < p.N; v += step) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float x = ld_f(p.voxel, c * p.N + v);  // fminf / fmaxf drop a NaN coordinate
      b[c] = fminf(b[c], x);
      b[3 + c] = fmaxf(b[3 + c], x);
    }
  }
#pragma unroll
  for (int c = 0; c < 6; ++c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float y = __shfl_xor_sync(0xffffffffu, b[c], o);
      b[c] = c < 3 ? fminf(b[c], y) : fmaxf(b[c], y);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][c] = b[c];
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    float r = red[0][threadIdx.x];
    for (int w = 1; w < 8; ++w) r = threadIdx.x < 3 ? fminf(r, red[w][threadIdx.x]) : fmaxf(r, red[w][threadIdx.x]);
    p.bbox[blockIdx.x * 6 + threadIdx.x] = r;
  }
}

// The box over all partials, by one warp; lane c < 6 returns component c.
__device__ __forceinline__ float warp_bbox(const float* partial, int blocks, int lane) {
  float b[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  for (int i = lane; i < blocks; i += 32) {
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const float y = partial[i * 6 + c];
      b[c] = c < 3 ? fminf(b[c], y) : fmaxf(b[c], y);
    }
  }
  float out = 0.0f;
#pragma unroll
  for (int c = 0; c < 6; ++c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float y = __shfl_xor_sync(0xffffffffu, b[c], o);
      b[c] = c < 3 ? fminf(b[c], y) : fmaxf(b[c], y);
    }
    if (lane == c) out = b[c];
  }
  return out;
}

// ---------------------------------------------------------------------------
template <typename T>
struct TableP {
  const T* real;
  const T* imag;
  const T* tx;
  const T* rx;
  const float* bbox;
  const float* basis;
  AntMeta* meta;
  float2* table;  // [A][kMaxCells][Q]
  CellHead* head;
  int S, blocks;
  double k1, b1, kappa;  // kappa as rounded to FP32
};

// One block per antenna; thread (cell k, slice) sums its slice of the samples
// into the cell's Q coefficients: the sample turned by the exact phase of the
// cell's centre (FP64, reduced in cycles), times its basis.  About 45
// instructions per (cell, sample): 0.6 ms for 49152 antennas x 256 samples x 40 cells.
template <typename T>
__global__ void __launch_bounds__(kTableThreads) mf_cell_table_kernel(const TableP<T> p) {
  constexpr int Q = GatherCells::Q;
  __shared__ float box_s[6];
  __shared__ int band_s[2], skip_s;
  __shared__ float2 smp[kTableTile];
  __shared__ float bas[kTableTile * Q];
  __shared__ float2 red[kTableThreads * Q];
  const int64_t a = blockIdx.x;
  if (threadIdx.x < 32) {
    const float b = warp_bbox(p.bbox, p.blocks, threadIdx.x);
    if (threadIdx.x < 6) box_s[threadIdx.x] = b;
  } else if (threadIdx.x == 32) {
    skip_s = *reinterpret_cast<const volatile int*>(&p.head->bad);  // one answer for the whole block
  }
  __syncthreads();
  if (skip_s) return;  // an earlier antenna's cells did not fit
  if (threadIdx.x == 0) {
    double t[3], r[3], box[6];
    AntMeta m;
    double vv = 0.0;
    bool same = a > 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      t[c] = ld_f(p.tx, a * 3 + c);
      r[c] = ld_f(p.rx, a * 3 + c);
      if (a > 0) same = same && t[c] == static_cast<double>(ld_f(p.tx, (a - 1) * 3 + c));
      const double center = box_center(box_s[c], box_s[3 + c]);
      if (a == 0) p.head->center[c] = center;
      box[c] = box_s[c] - center;
      box[3 + c] = box_s[3 + c] - center;
      t[c] -= center;
      r[c] -= center;
      const double e = fmax(fabs(box[c]), fabs(box[3 + c]));
      vv = fma(e, e, vv);
    }
    leg_antenna(t, vv, m.t);
    leg_antenna(r, vv, m.r);
    double tn, tf, rn, rf;
    leg_range(t, box, tn, tf);
    leg_range(r, box, rn, rf);
    tn = sqrt(tn);
    tf = sqrt(tf);
    rn = sqrt(rn);
    rf = sqrt(rf);
    const double lo = floor((tn + rn) * p.kappa) - 2.0, hi = ceil((tf + rf) * p.kappa) + 2.0;
    const bool fits = tf < kMaxLeg && rf < kMaxLeg && hi - lo + 1.0 <= kMaxCells;  // false for NaN
    if (!fits) p.head->bad = 1;
    m.c0 = fits ? static_cast<int>(lo) : 0;
    m.cells = fits ? static_cast<int>(hi - lo) + 1 : 0;
    m.same_tx = same ? 1 : 0;
    m.pad = 0;
    p.meta[a] = m;
    band_s[0] = m.c0;
    band_s[1] = m.cells;
  }
  __syncthreads();
  const int c0 = band_s[0], nc = band_s[1];
  if (nc == 0) return;
  const int slices = kTableThreads / nc;
  const int slice = threadIdx.x / nc;
  const int k = threadIdx.x - slice * nc;
  const bool on = slice < slices;
  const double dk = fma(p.k1, static_cast<double>(c0 + k) / p.kappa, p.b1);
  const double mid = 0.5 * (p.S - 1);
  float2 acc[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) acc[q] = make_float2(0.0f, 0.0f);
  for (int n0 = 0; n0 < p.S; n0 += kTableTile) {
    const int cnt = min(kTableTile, p.S - n0);
    __syncthreads();
    for (int i = threadIdx.x; i < cnt; i += kTableThreads) {
      smp[i] = make_float2(ld_f(p.real, a * p.S + n0 + i), ld_f(p.imag, a * p.S + n0 + i));
    }
    for (int i = threadIdx.x; i < cnt * Q; i += kTableThreads) bas[i] = p.basis[n0 * Q + i];
    __syncthreads();
    if (on) {
      for (int i = slice; i < cnt; i += slices) {
        const double c = (static_cast<double>(n0 + i) - mid) * dk;
        const float2 e = cis_cycles(static_cast<float>(c - rint(c)));
        const float2 x = smp[i];
        // v = x e^{-j phase}; odd powers carry -j v
        const float2 v = make_float2(fmaf(x.x, e.x, x.y * e.y), fmaf(x.y, e.x, -x.x * e.y));
        const float2 w = make_float2(v.y, -v.x);
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const float g = bas[i * Q + q];
          acc[q] = ffma2(make_float2(g, g), (q & 1) ? w : v, acc[q]);
        }
      }
    }
  }
  if (on) {
#pragma unroll
    for (int q = 0; q < Q; ++q) red[(slice * nc + k) * Q + q] = acc[q];
  }
  __syncthreads();
  float2* out = p.table + a * kMaxCells * Q;
  for (int i = threadIdx.x; i < nc * Q; i += kTableThreads) {
    float2 s = red[i];
    for (int sl = 1; sl < slices; ++sl) s = fadd2(s, red[sl * nc * Q + i]);
    out[i] = s;
  }
}

// ---------------------------------------------------------------------------
template <typename T>
struct GatherCellsP {
  const T* voxel;
  T* out_r;
  T* out_i;
  const AntMeta* meta;
  const float2* table;
  float2* partial;
  const CellHead* head;
  int* status;
  int64_t A, N;
  int splits;
  int64_t ant_per_split;
  float kappa;  // cells per metre
  PairPhase ph;
};

constexpr int kCellBytes = GatherCells::Q * sizeof(float2);  // 48
constexpr int kRowBytes = kMaxCells * kCellBytes;            // 4608
// Launch shape of the gather.  Measured on 49152 antennas x 512000 voxels: 52.7 ms; 2 voxels
// per thread with 5 blocks per SM 65.2, 6 voxels with 2 blocks 59.0; stages of 4 antennas 75.1,
// of up to 16 antennas (8 KB pool) 53.9.
constexpr int kGatherVpt = 4;         // voxels per thread
constexpr int kGatherThreads = 128;   // consumer threads; one more warp copies
constexpr int kGatherBlocks = 3;      // resident per SM (128 registers)
constexpr int kGatherRows = 32;       // antennas per stage, at most
constexpr int kGatherStages = 3;
constexpr int kGatherPool = 16384;    // bytes of cells per stage
static_assert(kGatherPool >= kRowBytes, "any one antenna's cells fit");

struct GatherSmem {
  uint64_t full[kGatherStages];
  uint64_t empty[kGatherStages];
  int base[kGatherStages][kGatherRows];  // byte offset of the row's absolute cell 0, magic bits subtracted
  int count[kGatherStages];              // antennas in the stage
  float box[8];
  float red[4][8];
  alignas(16) AntMeta meta[kGatherStages][kGatherRows];
  alignas(16) unsigned char pool[kGatherStages][kGatherPool];
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// VPT voxels per thread; stages of up to kGatherRows antennas stream through a ring filled
// by a warp of its own.  Of each antenna's cells a stage holds those that the
// block's voxels can reach (their own bounding box): one bulk copy per antenna
// row.  A pair is two legs (the transmitter's only where it differs from the
// preceding antenna's: the virtual channels of one transmitter follow one
// another), the phase, one sincos, three 16-byte shared loads and five packed
// multiply-adds.  Terms are summed plainly within a stage and compensated across
// stages.
//
// About 61 instructions per 32 pairs, of which the FP64 ones take 21 issue cycles
// of their pipe, the rsqrt, sine and cosine 26 of theirs and the 16-byte loads (four
// wavefronts each whatever the addresses) 48 of a scheduler's 78 cycles per 32
// pairs (ncu, 3072 x 110592 pairs): shared-memory bandwidth comes first, then the
// latency of the FP64 chains, which is why 4 voxels per thread with few warps beat
// more warps with fewer.  49152 antennas x 256 samples x 512000 voxels: 950 ms by
// the direct kernel, 52.7 ms through the cells (478 G pairs/s); 3072 x 128 x
// 110592: 7.53 ms against 0.79 ms.
// ACCURATE: the phasor of a pair by sincospif (the NUFFT form's, ~1 ulp) instead
// of the hardware sine and cosine (4e-7).
template <typename T, bool ACCURATE>
__global__ void __launch_bounds__(kGatherThreads + 32, kGatherBlocks) mf_cell_gather_kernel(const GatherCellsP<T> p) {
  constexpr int VPT = kGatherVpt;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  GatherSmem& sm = *reinterpret_cast<GatherSmem*>(smem_raw);
  if (p.head->bad) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool producer = warp == kGatherThreads / 32;
  // split-major blocks: those resident together stream the same antennas' rows
  const int64_t vtiles = gridDim.x / p.splits;
  const int split = static_cast<int>(blockIdx.x / vtiles);
  const int64_t vtile = blockIdx.x - static_cast<int64_t>(split) * vtiles;
  const int64_t a_begin = static_cast<int64_t>(split) * p.ant_per_split;
  const int64_t a_end = min(p.A, a_begin + p.ant_per_split);
  const int num_ant = static_cast<int>(max(int64_t{0}, a_end - a_begin));

  float fx[VPT], fy[VPT], fz[VPT];
  int64_t vid[VPT];
  unsigned nan_voxel = 0;  // bit j: a NaN coordinate, whose result is NaN
  {
    float b[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      vid[j] = vtile * (kGatherThreads * VPT) + threadIdx.x + j * kGatherThreads;
      const int64_t v = min(vid[j], p.N - 1);
      fx[j] = fy[j] = fz[j] = 0.0f;
      if (producer) continue;
      fx[j] = ld_f(p.voxel, v);
      fy[j] = ld_f(p.voxel, p.N + v);
      fz[j] = ld_f(p.voxel, 2 * p.N + v);
      if (fx[j] != fx[j] || fy[j] != fy[j] || fz[j] != fz[j]) {
        nan_voxel |= 1u << j;
      } else {
        b[0] = fminf(b[0], fx[j]);
        b[1] = fminf(b[1], fy[j]);
        b[2] = fminf(b[2], fz[j]);
        b[3] = fmaxf(b[3], fx[j]);
        b[4] = fmaxf(b[4], fy[j]);
        b[5] = fmaxf(b[5], fz[j]);
      }
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float y = __shfl_xor_sync(0xffffffffu, b[c], o);
        b[c] = c < 3 ? fminf(b[c], y) : fmaxf(b[c], y);
      }
      if (lane == 0 && !producer) sm.red[warp][c] = b[c];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
      float r = sm.red[0][threadIdx.x];
#pragma unroll
      for (int w = 1; w < kGatherThreads / 32; ++w) {
        r = threadIdx.x < 3 ? fminf(r, sm.red[w][threadIdx.x]) : fmaxf(r, sm.red[w][threadIdx.x]);
      }
      // from the centre, as the antennas' positions are; all NaN voxels leave an empty box
      sm.box[threadIdx.x] = static_cast<float>(static_cast<double>(r) - p.head->center[threadIdx.x % 3]);
    }
    if (threadIdx.x == 32) {
      for (int s = 0; s < kGatherStages; ++s) {
        mbar_init(&sm.full[s], 32);  // every lane of the copying warp arrives, with its bytes
        mbar_init(&sm.empty[s], kGatherThreads / 32);
      }
      fence_barrier_init();
    }
    __syncthreads();
  }
  const bool any_valid = sm.box[0] <= sm.box[3];  // else every voxel of the block is NaN

  if (producer) {
    if (!any_valid) return;
    for (int t = 0, done = 0; done < num_ant; ++t) {
      const int s = t % kGatherStages, use = t / kGatherStages;
      const int64_t a0 = a_begin + done;
      uint32_t bytes = 0;
      int lo = 0, c0 = 0;
      if (lane < kGatherRows && lane < num_ant - done) {
        const AntMeta& m = p.meta[a0 + lane];
        float tp[3], rp[3], tn, tf, rn, rf;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          tp[c] = static_cast<float>(-0.5 / kUnit * m.t[c]);
          rp[c] = static_cast<float>(-0.5 / kUnit * m.r[c]);
        }
        c0 = m.c0;
        leg_range(tp, sm.box, tn, tf);
        leg_range(rp, sm.box, rn, rf);
        // One cell of margin on either side covers the FP32 rounding: positions from the centre
        // are below 8 m and paths below 16 m (kMaxLeg), good to 3e-6 m in all, a third of a
        // cell at the narrowest cells taken (1e5 per metre, mf_cells_scale_ok).  The pairs'
        // cells therefore stay in the row without a check per pair.
        lo = static_cast<int>(floorf((sqrtf(tn) + sqrtf(rn)) * p.kappa)) - 1 - c0;
        int hi = static_cast<int>(ceilf((sqrtf(tf) + sqrtf(rf)) * p.kappa)) + 1 - c0;
        lo = min(max(lo, 0), m.cells - 1);
        hi = min(max(hi, lo), m.cells - 1);
        bytes = static_cast<uint32_t>(hi - lo + 1) * kCellBytes;
      }
      uint32_t end = bytes;  // of the antenna's cells in the stage's pool
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += y;
      }
      const bool in = bytes != 0 && end <= kGatherPool;
      const int count = __popc(__ballot_sync(0xffffffffu, in));  // the first ones: `end` grows with the lane
      if (use > 0 && !__all_sync(0xffffffffu, mbar_wait_bounded(&sm.empty[s], (use - 1) & 1, p.status))) {
        // the consumers gave up: wait for the copies still in flight
        for (int u = max(0, t - kGatherStages); u < t; ++u) {
          mbar_wait_bounded(&sm.full[u % kGatherStages], (u / kGatherStages) & 1, p.status);
        }
        return;
      }
      if (in) {
        // byte offset of absolute cell k: base + (bits of k + magic) * 48, modulo 2^32
        sm.base[s][lane] = static_cast<int>(static_cast<uint32_t>(s * kGatherPool) + end - bytes -
                                            (static_cast<uint32_t>(c0 + lo) + kRoundMagicBits) * kCellBytes);
      }
      if (lane == 0) sm.count[s] = count;
      const uint32_t meta_bytes = lane == 0 ? count * static_cast<uint32_t>(sizeof(AntMeta)) : 0;
      mbar_arrive_expect_tx(&sm.full[s], (in ? bytes : 0) + meta_bytes);  // releases sm.base and sm.count too
      if (lane == 0) bulk_g2s(&sm.meta[s][0], p.meta + a0, meta_bytes, &sm.full[s]);
      if (in) {
        bulk_g2s(&sm.pool[s][end - bytes],
                 reinterpret_cast<const unsigned char*>(p.table) + (a0 + lane) * kRowBytes + lo * kCellBytes, bytes,
                 &sm.full[s]);
      }
      done += count;
    }
    return;
  }

  // NaN voxels take the corner of the box, so that their cells stay in the rows
  double vx[VPT], vy[VPT], vz[VPT], vv[VPT];
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const bool nan = (nan_voxel >> j) & 1u;
    vx[j] = (nan ? sm.box[0] : fx[j] - p.head->center[0]) * kUnit;
    vy[j] = (nan ? sm.box[1] : fy[j] - p.head->center[1]) * kUnit;
    vz[j] = (nan ? sm.box[2] : fz[j] - p.head->center[2]) * kUnit;
    vv[j] = fma(vx[j], vx[j], fma(vy[j], vy[j], vz[j] * vz[j]));
  }
  float yr[VPT], yi[VPT], cr[VPT], ci[VPT];
  float dt[VPT], lt[VPT];  // the transmitter's legs
#pragma unroll
  for (int j = 0; j < VPT; ++j) yr[j] = yi[j] = cr[j] = ci[j] = dt[j] = lt[j] = 0.0f;

  for (int t = 0, done = 0; any_valid && done < num_ant; ++t) {
    const int s = t % kGatherStages;
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&sm.full[s], (t / kGatherStages) & 1, p.status))) return;
    const int rws = sm.count[s];
    done += rws;
    float tr[VPT], ti[VPT];
#pragma unroll
    for (int j = 0; j < VPT; ++j) tr[j] = ti[j] = 0.0f;
    for (int r = 0; r < rws; ++r) {
      const AntMeta& m = sm.meta[s][r];
      if (!m.same_tx || (t == 0 && r == 0)) {
        const double2 t0 = *reinterpret_cast<const double2*>(&m.t[0]);
        const double2 t1 = *reinterpret_cast<const double2*>(&m.t[2]);
#pragma unroll
        for (int j = 0; j < VPT; ++j) {
          const Leg g = leg_length(t0.x, t0.y, t1.x, t1.y, vx[j], vy[j], vz[j], vv[j]);
          dt[j] = g.d;
          lt[j] = g.l;
        }
      }
      const double2 r0 = *reinterpret_cast<const double2*>(&m.r[0]);
      const double2 r1 = *reinterpret_cast<const double2*>(&m.r[2]);
      const unsigned char* rows = &sm.pool[0][0];
      const uint32_t base = static_cast<uint32_t>(sm.base[s][r]);
#pragma unroll
      for (int j = 0; j < VPT; ++j) {
        const Leg g = leg_length(r0.x, r0.y, r1.x, r1.y, vx[j], vy[j], vz[j], vv[j]);
        const float hi = dt[j] + g.d, lo = lt[j] + g.l;
        const CellPos c = pair_cell(p.ph, hi, lo);
        const float4* q = reinterpret_cast<const float4*>(
            rows + static_cast<uint32_t>(__float_as_uint(c.m) * static_cast<uint32_t>(kCellBytes) + base));
        const float4 q2 = q[2], q1 = q[1], q0 = q[0];
        const float2 xx = make_float2(c.x, c.x);
        float2 acc = ffma2(make_float2(q2.z, q2.w), xx, make_float2(q2.x, q2.y));
        acc = ffma2(acc, xx, make_float2(q1.z, q1.w));
        acc = ffma2(acc, xx, make_float2(q1.x, q1.y));
        acc = ffma2(acc, xx, make_float2(q0.z, q0.w));
        acc = ffma2(acc, xx, make_float2(q0.x, q0.y));
        const float2 e = pair_phasor<ACCURATE>(pair_cycles(p.ph, hi, lo));
        tr[j] = fmaf(e.x, acc.x, fmaf(e.y, acc.y, tr[j]));
        ti[j] = fmaf(e.x, acc.y, fmaf(-e.y, acc.x, ti[j]));
      }
    }
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      kahan_add(yr[j], cr[j], tr[j]);
      kahan_add(yi[j], ci[j], ti[j]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&sm.empty[s]);
  }

#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    if (vid[j] >= p.N) continue;
    if ((nan_voxel >> j) & 1u) yr[j] = yi[j] = NAN;
    if (p.splits == 1) {
      p.out_r[vid[j]] = from_f<T>(yr[j] / static_cast<float>(p.A));
      p.out_i[vid[j]] = from_f<T>(yi[j] / static_cast<float>(p.A));
    } else {
      p.partial[split * p.N + vid[j]] = make_float2(yr[j], yi[j]);
    }
  }
}

int gather_splits(int64_t A, int64_t N) {
  const int64_t vtiles = (N + kGatherThreads * kGatherVpt - 1) / (kGatherThreads * kGatherVpt);
  const int64_t stages = std::max<int64_t>(1, (A + kGatherRows - 1) / kGatherRows);
  return std::max(1, std::min<int>(pick_splits(vtiles, kGatherBlocks, current_device_info().sm_count, stages),
                                   static_cast<int>(std::min<int64_t>(stages, 256))));
}

template <typename T>
cudaError_t launch_cells_forward(const MfArgs& a, unsigned char* ws, const CellLayout& l, int splits, cudaStream_t st) {
  const PhaseConsts pc = phase_consts(kMfStartFrequency, a.As, a.fs);
  const double kappa = cells_per_metre(pc.k1, a.S, GatherCells::kOver);
  CellHead* head = reinterpret_cast<CellHead*>(ws + l.head);
  float* bbox = reinterpret_cast<float*>(ws + l.bbox);
  float* basis = reinterpret_cast<float*>(ws + l.basis);
  AntMeta* meta = reinterpret_cast<AntMeta*>(ws + l.meta);
  float2* table = reinterpret_cast<float2*>(ws + l.table);
  const int pb = static_cast<int>(std::min<int64_t>(kPrepBlocks, (std::max<int64_t>(a.N, a.S) + 255) / 256));

  PrepP<T> pp;
  pp.voxel = static_cast<const T*>(a.voxel);
  pp.N = a.N;
  pp.S = static_cast<int>(a.S);
  pp.theta_step = 2.0 * M_PI * pc.k1 / kappa;
  pp.bbox = bbox;
  pp.basis = basis;
  pp.head = head;
  cell_prep_kernel<T, GatherCells::Q><<<pb, 256, 0, st>>>(pp);

  TableP<T> tp;
  tp.real = static_cast<const T*>(a.real);
  tp.imag = static_cast<const T*>(a.imag);
  tp.tx = static_cast<const T*>(a.tx);
  tp.rx = static_cast<const T*>(a.rx);
  tp.bbox = bbox;
  tp.basis = basis;
  tp.meta = meta;
  tp.table = table;
  tp.head = head;
  tp.S = pp.S;
  tp.blocks = pb;
  tp.k1 = pc.k1;
  tp.b1 = pc.b1;
  tp.kappa = kappa;
  mf_cell_table_kernel<T><<<static_cast<unsigned>(a.A), kTableThreads, 0, st>>>(tp);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;

  GatherCellsP<T> gp;
  gp.voxel = pp.voxel;
  gp.out_r = static_cast<T*>(a.out_real);
  gp.out_i = static_cast<T*>(a.out_imag);
  gp.meta = meta;
  gp.table = table;
  gp.partial = reinterpret_cast<float2*>(ws + l.partial);
  gp.head = head;
  gp.status = device_status_ptr();
  gp.A = a.A;
  gp.N = a.N;
  gp.splits = splits;
  const int64_t stages = (a.A + kGatherRows - 1) / kGatherRows;
  gp.ant_per_split = ((stages + splits - 1) / splits) * kGatherRows;
  gp.kappa = static_cast<float>(kappa);
  gp.ph = pair_phase(pc.k0, pc.b0, pc.k1, pc.b1, a.S, kappa);
  const void* fn = a.mode == kNufft ? reinterpret_cast<const void*>(&mf_cell_gather_kernel<T, true>)
                                   : reinterpret_cast<const void*>(&mf_cell_gather_kernel<T, false>);
  const int smem = static_cast<int>(sizeof(GatherSmem));
  err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) return err;
  const int64_t vtiles = (a.N + kGatherThreads * kGatherVpt - 1) / (kGatherThreads * kGatherVpt);
  if (vtiles * splits > 0x7fffffff) return cudaErrorInvalidConfiguration;
  void* args[] = {&gp};
  err = cudaLaunchKernel(fn, dim3(static_cast<unsigned>(vtiles * splits)), dim3(kGatherThreads + 32), args, smem, st);
  if (err != cudaSuccess || splits == 1) return err;
  return launch_finalize_partials(a.dtype, gp.partial, splits, a.N, static_cast<float>(a.A), a.out_real, a.out_imag, st);
}

// ---------------------------------------------------------------------------
// Adjoint.  g[a, n] = (1/A) sum_v G_v e^{+j 2 pi (c0 + n d)}: with w_v = G_v e^{+j 2 pi c}, c the
// phase of carrier and middle sample, the voxels of one cell enter every sample
// through the moments M_q = sum_v w_v x_v^q alone,
//   g[a, n] = (1/A) sum_cells e^{+j 2 pi n' d_k} (sum_q even g_q(n) M_q + j sum_q odd g_q(n) M_q).
// Launches: the boxes of voxels and antennas (partials) and the basis; the common
// band of cells; the moments; the samples from the moments; the direct kernel,
// which returns at once unless the band did not fit.
constexpr int kMomentCap = 24 * MomentCells::kOver;  // cells: 1.8 m of path at 4 GHz swept
constexpr int kBoxFloats = 20;                       // voxels, tx, rx: lo xyz, hi xyz; not for the cells; pad

struct MomentHead {
  int bad;
  int k0, cells;
  int pad;
  double bias;       // |v|^2 bound for leg_antenna
  double center[3];  // of the voxels' box: the origin of the pairs' legs
};

struct MomentLayout {
  size_t head, box, basis, moments, partial, total;
};

MomentLayout moment_layout(int64_t A, int64_t S, int splits, size_t partial_bytes) {
  const size_t apad = static_cast<size_t>((A + 31) / 32) * 32;
  MomentLayout l;
  l.head = 0;
  l.box = 256;
  l.basis = up256(l.box + kPrepBlocks * kBoxFloats * sizeof(float));
  l.moments = up256(l.basis + static_cast<size_t>(S) * MomentCells::Q * sizeof(float));
  l.partial = l.moments + up256(splits * static_cast<size_t>(kMomentCap) * MomentCells::Q * sizeof(float2) * apad);
  l.total = l.partial + up256(partial_bytes);
  return l;
}

template <typename T>
struct BoxP {
  const T* voxel;  // [3, N]
  const T* gr;     // [N]
  const T* gi;
  const T* tx;     // [A, 3]
  const T* rx;
  int64_t N, A;
  int S;
  double theta_step;
  float* box;  // [blocks][kBoxFloats]
  float* basis;
};

template <typename T, int Q>
__global__ void __launch_bounds__(256) moment_prep_kernel(const BoxP<T> p) {
  __shared__ float red[8][kBoxFloats];
  const int64_t gid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t n = gid; n < p.S; n += step) {
    float g[Q];
    cell_basis<Q>(p.theta_step * (static_cast<double>(n) - 0.5 * (p.S - 1)), g);
#pragma unroll
    for (int q = 0; q < Q; ++q) p.basis[n * Q + q] = g[q];
  }
  float b[18];
  float out = 0.0f;  // 1: a NaN antenna, or an infinite gradient, of which the moments' sums would make a NaN
#pragma unroll
  for (int c = 0; c < 18; ++c) b[c] = (c % 6) < 3 ? INFINITY : -INFINITY;
  auto add = [&](float* box, float x, int c) {
    box[c] = fminf(box[c], x);
    box[3 + c] = fmaxf(box[3 + c], x);
  };
  for (int64_t v = gid; v < p.N; v += step) {
#pragma unroll
    for (int c = 0; c < 3; ++c) add(b, ld_f(p.voxel, c * p.N + v), c);
    if (fabsf(ld_f(p.gr, v)) == INFINITY || fabsf(ld_f(p.gi, v)) == INFINITY) out = 1.0f;
  }
  for (int64_t a = gid; a < p.A; a += step) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float t = ld_f(p.tx, a * 3 + c), r = ld_f(p.rx, a * 3 + c);
      if (t != t || r != r) out = 1.0f;
      add(b + 6, t, c);
      add(b + 12, r, c);
    }
  }
#pragma unroll
  for (int c = 0; c < 19; ++c) {
    float x = c < 18 ? b[c < 18 ? c : 0] : out;
    const bool low = c < 18 && (c % 6) < 3;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float y = __shfl_xor_sync(0xffffffffu, x, o);
      x = low ? fminf(x, y) : fmaxf(x, y);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][c] = x;
  }
  __syncthreads();
  const int c = threadIdx.x;
  if (c < 19) {
    float r = red[0][c];
    for (int w = 1; w < 8; ++w) r = c < 18 && (c % 6) < 3 ? fminf(r, red[w][c]) : fmaxf(r, red[w][c]);
    p.box[blockIdx.x * kBoxFloats + c] = r;
  }
}

// The cells that any antenna's path to any voxel can reach, from the boxes.
__global__ void __launch_bounds__(32 * 19) moment_band_kernel(const float* partial, int blocks, double kappa,
                                                             MomentHead* head) {
  __shared__ float s[19];
  const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool low = c < 18 && (c % 6) < 3;
  float x = low ? INFINITY : -INFINITY;
  for (int i = lane; i < blocks; i += 32) {
    const float y = partial[i * kBoxFloats + c];
    x = low ? fminf(x, y) : fmaxf(x, y);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float y = __shfl_xor_sync(0xffffffffu, x, o);
    x = low ? fminf(x, y) : fmaxf(x, y);
  }
  if (lane == 0) s[c] = x;
  __syncthreads();
  if (threadIdx.x != 0) return;
  double near[2] = {0.0, 0.0}, far[2] = {0.0, 0.0}, vv = 0.0;
  for (int k = 0; k < 3; ++k) {
    const double lo = s[k], hi = s[3 + k];
    for (int e = 0; e < 2; ++e) {
      const double alo = s[6 + 6 * e + k], ahi = s[9 + 6 * e + k];
      const double gap = fmax(0.0, fmax(lo - ahi, alo - hi)), reach = fmax(hi - alo, ahi - lo);
      near[e] += gap * gap;
      far[e] += reach * reach;
    }
    const double center = box_center(s[k], s[3 + k]);
    const double m = fmax(fabs(lo - center), fabs(hi - center));
    vv += m * m;
    head->center[k] = center;
  }
  const double ft = sqrt(far[0]), fr = sqrt(far[1]);
  const double lo = floor((sqrt(near[0]) + sqrt(near[1])) * kappa) - 1.0, hi = ceil((ft + fr) * kappa) + 1.0;
  const bool fits = s[18] == 0.0f && ft < kMaxLeg && fr < kMaxLeg && hi - lo + 1.0 <= kMomentCap;  // false for NaN
  head->bad = fits ? 0 : 1;
  head->k0 = fits ? static_cast<int>(lo) : 0;
  head->cells = fits ? static_cast<int>(hi - lo) + 1 : 0;
  head->bias = fits ? vv : 0.0;
}

template <typename T>
struct MomentP {
  const T* voxel;
  const T* gr;
  const T* gi;
  const T* tx;
  const T* rx;
  float4* moments;  // [splits][kMomentCap][Q/2][apad]: pairs of complex moments
  const MomentHead* head;
  int64_t A, N, apad, vox_per_split;
  PairPhase ph;
};

__device__ __forceinline__ void red_add4(float4* dst, float2 a, float2 b) {
  asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(a.x), "f"(a.y), "f"(b.x),
               "f"(b.y)
               : "memory");
}

// One thread per antenna; the voxels of the block's split pass through shared
// memory in tiles and every thread reads the same one (broadcast).  The moments
// of the thread's current cell stay in registers; consecutive voxels mostly
// share a cell, and when it changes, and after each tile (so that a cell that holds
// hundreds of thousands of voxels is summed in two levels: one chain of 200000 terms of one
// sign erred by 2e-5), the moments are added to the antenna's own
// record in memory (vector reductions without a return value: nothing waits for
// them, and no other thread touches the record, so the order of its sums, and the
// result, is the same on every run).  About 88 instructions per 32 pairs (100 where the
// antennas share no positions) at 68% of the issue slots (FMA pipe 40%, XU 20%, FP64 11%;
// 14 warps per SM): 972 antennas x 201 samples x
// 50653 voxels take 0.19 ms here, 2.37 ms by the recurrence of the direct kernel.
constexpr int kMomentTile = 128;
constexpr int kMomentUnroll = 4;  // voxels whose paths overlap (2: 2% slower; 6 blocks per SM and one: 8%)

template <typename T>
__global__ void __launch_bounds__(128, 4) mf_moment_kernel(const MomentP<T> p) {
  constexpr int Q = MomentCells::Q;
  __shared__ double2 sxy[kMomentTile], szv[kMomentTile];
  __shared__ float2 sg[kMomentTile];
  if (p.head->bad) return;
  const int k0 = p.head->k0, cells = p.head->cells;
  const int64_t a = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  const int64_t split = blockIdx.y;
  const int64_t v_begin = split * p.vox_per_split;
  const int64_t v_end = min(p.N, v_begin + p.vox_per_split);
  // The antennas of a warp often share transmitters and receivers (32 channels of a
  // 3 TX x 4 RX scan have about 20 positions): then each lane forms one position's legs
  // and takes its own two from the lanes that hold them.
  double mt[4], mr[4];
  int from_t = 0, from_r = 0;
  bool shared_legs;
  {
    float t[3], r[3];
    const int64_t al = min(a, p.A - 1);
    unsigned same_t = 0xffffffffu, same_r = 0xffffffffu;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      t[c] = ld_f(p.tx, al * 3 + c);
      r[c] = ld_f(p.rx, al * 3 + c);
      same_t &= __match_any_sync(0xffffffffu, __float_as_uint(t[c]));
      same_r &= __match_any_sync(0xffffffffu, __float_as_uint(r[c]));
    }
    const int lane = threadIdx.x & 31;
    const int first_t = __ffs(same_t) - 1, first_r = __ffs(same_r) - 1;
    const unsigned heads_t = __ballot_sync(0xffffffffu, first_t == lane);
    const unsigned heads_r = __ballot_sync(0xffffffffu, first_r == lane);
    const int nt = __popc(heads_t), nr = __popc(heads_r);
    shared_legs = nt + nr <= 32;
    from_t = __popc(heads_t & ((1u << first_t) - 1u));
    from_r = nt + __popc(heads_r & ((1u << first_r) - 1u));
    // lane i < nt takes the i-th transmitter, lane nt + i the i-th receiver
    const int want = lane < nt ? static_cast<int>(__fns(heads_t, 0, lane + 1))
                               : static_cast<int>(__fns(heads_r, 0, min(lane - nt, nr - 1) + 1));
    double own[3], other[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float ht = __shfl_sync(0xffffffffu, t[c], want), hr = __shfl_sync(0xffffffffu, r[c], want);
      own[c] = static_cast<double>(shared_legs ? (lane < nt ? ht : hr) : t[c]) - p.head->center[c];
      other[c] = static_cast<double>(r[c]) - p.head->center[c];
    }
    leg_antenna(own, p.head->bias, mt);
    leg_antenna(other, p.head->bias, mr);
  }
  const bool mine = a < p.apad;
  float4* rec = p.moments + split * kMomentCap * (Q / 2) * p.apad + a;
  if (mine) {
    for (int i = 0; i < cells * (Q / 2); ++i) rec[i * p.apad] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  float2 M[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) M[q] = make_float2(0.0f, 0.0f);
  float cur = __uint_as_float(kRoundMagicBits + static_cast<uint32_t>(k0));
  auto flush = [&]() {
    const int k = static_cast<int>(__float_as_uint(cur) - kRoundMagicBits) - k0;
    float4* dst = rec + static_cast<int64_t>(min(max(k, 0), cells - 1)) * (Q / 2) * p.apad;
#pragma unroll
    for (int q = 0; q < Q; q += 2) {
      if (mine) red_add4(dst + (q / 2) * p.apad, M[q], M[q + 1]);
      M[q] = M[q + 1] = make_float2(0.0f, 0.0f);
    }
  };
  for (int64_t v0 = v_begin; v0 < v_end; v0 += kMomentTile) {
    __syncthreads();
    for (int i = threadIdx.x; i < kMomentTile; i += blockDim.x) {
      const int64_t v = v0 + i;
      double x = 0.0, y = 0.0, z = 0.0;
      float2 g = make_float2(0.0f, 0.0f);
      if (v < v_end) {
        const float fx = ld_f(p.voxel, v), fy = ld_f(p.voxel, p.N + v), fz = ld_f(p.voxel, 2 * p.N + v);
        g = make_float2(ld_f(p.gr, v), ld_f(p.gi, v));
        x = (fx - p.head->center[0]) * kUnit;
        y = (fy - p.head->center[1]) * kUnit;
        z = (fz - p.head->center[2]) * kUnit;
        if (fx != fx || fy != fy || fz != fz) g = make_float2(NAN, NAN);  // its every sample is NaN
      }
      if (v >= v_end || g.x != g.x) {
        // somewhere in the box: the split's first voxel, or the box's centre when that is NaN too
        const float fx = ld_f(p.voxel, v_begin), fy = ld_f(p.voxel, p.N + v_begin), fz = ld_f(p.voxel, 2 * p.N + v_begin);
        const bool ok = fx == fx && fy == fy && fz == fz;
        x = ok ? (fx - p.head->center[0]) * kUnit : 0.0;
        y = ok ? (fy - p.head->center[1]) * kUnit : 0.0;
        z = ok ? (fz - p.head->center[2]) * kUnit : 0.0;
      }
      sxy[i] = make_double2(x, y);
      szv[i] = make_double2(z, fma(x, x, fma(y, y, z * z)));
      sg[i] = g;
    }
    __syncthreads();
    const int count = static_cast<int>(min(static_cast<int64_t>(kMomentTile), v_end - v0));
    auto sum_tile = [&](auto shared) {
      constexpr bool SHARED = decltype(shared)::value;
      for (int i = 0; i < count; i += kMomentUnroll) {
        float x[kMomentUnroll], m[kMomentUnroll];
        float2 w[kMomentUnroll];
#pragma unroll
        for (int u = 0; u < kMomentUnroll; ++u) {
          const double2 xy = sxy[i + u], zv = szv[i + u];
          const float2 g = sg[i + u];
          Leg lt = leg_length(mt[0], mt[1], mt[2], mt[3], xy.x, xy.y, zv.x, zv.y), lr;
          if (SHARED) {
            lr.d = __shfl_sync(0xffffffffu, lt.d, from_r);
            lr.l = __shfl_sync(0xffffffffu, lt.l, from_r);
            lt.d = __shfl_sync(0xffffffffu, lt.d, from_t);
            lt.l = __shfl_sync(0xffffffffu, lt.l, from_t);
          } else {
            lr = leg_length(mr[0], mr[1], mr[2], mr[3], xy.x, xy.y, zv.x, zv.y);
          }
          const float hi = lt.d + lr.d, lo = lt.l + lr.l;
          const CellPos c = pair_cell(p.ph, hi, lo);
          w[u] = cmul(g, cis_cycles_fast(pair_cycles(p.ph, hi, lo)));
          x[u] = c.x;
          m[u] = c.m;
        }
#pragma unroll
        for (int u = 0; u < kMomentUnroll; ++u) {
          if (m[u] != cur) {
            flush();
            cur = m[u];
          }
          // even moments from w, odd ones from w x, both times powers of x^2 (a chain of
          // three products, not seven: 5.03 -> 4.98 ms of the 3072 x 256 x 64^3 step)
          const float2 wx = make_float2(w[u].x * x[u], w[u].y * x[u]);
          M[0] = fadd2(M[0], w[u]);
          M[1] = fadd2(M[1], wx);
          const float sq = x[u] * x[u];
          float pw = sq;
#pragma unroll
          for (int q = 2; q < Q; q += 2) {
            M[q] = ffma2(make_float2(pw, pw), w[u], M[q]);
            M[q + 1] = ffma2(make_float2(pw, pw), wx, M[q + 1]);
            if (q + 2 < Q) pw *= sq;
          }
        }
      }
    };
    if (shared_legs) sum_tile(std::true_type{});
    else sum_tile(std::false_type{});
    flush();  // no chain of sums in registers is longer than a tile
  }
}

// Sums the splits' records into the first one's: block (x: 32 antennas, y: a pair
// of moments of one cell), 16 warps over the splits, in a fixed order and in FP64, as the
// partial sums of the other forms are.
constexpr int kSumWarps = 16;

__global__ void __launch_bounds__(32 * kSumWarps) mf_moment_sum_kernel(float4* moments, const MomentHead* head,
                                                                       int64_t apad, int splits, int pairs) {
  __shared__ double part[kSumWarps][4][32];
  if (head->bad || static_cast<int>(blockIdx.y) >= head->cells * pairs) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t stride = static_cast<int64_t>(kMomentCap) * pairs * apad;
  float4* src = moments + static_cast<int64_t>(blockIdx.y) * apad + blockIdx.x * 32 + lane;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
  for (int k = warp; k < splits; k += kSumWarps) {
    const float4 y = src[k * stride];
    s[0] += y.x;
    s[1] += y.y;
    s[2] += y.z;
    s[3] += y.w;
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) part[warp][c][lane] = s[c];
  __syncthreads();
  if (warp >= 4) return;
  double t = 0.0;  // warp c: component c
  for (int w = 0; w < kSumWarps; ++w) t += part[w][warp][lane];
  (&src->x)[warp] = static_cast<float>(t);
}

template <typename T>
struct SamplesP {
  const float4* moments;
  const float* basis;
  const MomentHead* head;
  T* out_r;
  T* out_i;
  int64_t A, apad;
  int S;
  double k1, b1, inv_kappa;
};

// Samples from the moments: 4 antennas per block, which share the phasors of the cells.
constexpr int kSampleAnts = 4;

template <typename T>
__global__ void __launch_bounds__(128) mf_moment_samples_kernel(const SamplesP<T> p) {
  constexpr int Q = MomentCells::Q;
  __shared__ float4 mom[kMomentCap][Q / 2][kSampleAnts];
  if (p.head->bad) return;
  const int k0 = p.head->k0, cells = p.head->cells;
  const int64_t a0 = blockIdx.x * static_cast<int64_t>(kSampleAnts);
  for (int i = threadIdx.x; i < cells * (Q / 2) * kSampleAnts; i += blockDim.x) {
    (&mom[0][0][0])[i] = p.moments[static_cast<int64_t>(i / kSampleAnts) * p.apad + a0 + i % kSampleAnts];
  }
  __syncthreads();
  const double mid = 0.5 * (p.S - 1);
  const float inv = static_cast<float>(p.A);
  for (int n = blockIdx.y * blockDim.x + threadIdx.x; n < p.S; n += gridDim.y * blockDim.x) {
    float g[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) g[q] = p.basis[n * Q + q];
    float2 acc[kSampleAnts];
#pragma unroll
    for (int u = 0; u < kSampleAnts; ++u) acc[u] = make_float2(0.0f, 0.0f);
    for (int k = 0; k < cells; ++k) {
      const double c = (n - mid) * fma(p.k1, (k0 + k) * p.inv_kappa, p.b1);
      const float2 e = cis_cycles(static_cast<float>(c - rint(c)));
#pragma unroll
      for (int u = 0; u < kSampleAnts; ++u) {
        float2 ev = make_float2(0.0f, 0.0f), od = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int q = 0; q < Q; q += 2) {
          const float4 m = mom[k][q / 2][u];
          ev = ffma2(make_float2(g[q], g[q]), make_float2(m.x, m.y), ev);
          od = ffma2(make_float2(g[q + 1], g[q + 1]), make_float2(m.z, m.w), od);
        }
        const float2 z = cmul(e, make_float2(ev.x - od.y, ev.y + od.x));
        acc[u] = fadd2(acc[u], z);
      }
    }
#pragma unroll
    for (int u = 0; u < kSampleAnts; ++u) {
      if (a0 + u >= p.A) continue;
      p.out_r[(a0 + u) * p.S + n] = from_f<T>(acc[u].x / inv);
      p.out_i[(a0 + u) * p.S + n] = from_f<T>(acc[u].y / inv);
    }
  }
}

struct MomentShape {
  int threads, groups, splits;
  int64_t vox_per_split;
};

// Blocks of up to 128 antennas; enough voxel splits for four 4-warp blocks per SM.
MomentShape moment_shape(int64_t A, int64_t N) {
  MomentShape s;
  s.threads = static_cast<int>(std::min<int64_t>(128, (A + 31) / 32 * 32));
  s.groups = static_cast<int>((A + s.threads - 1) / s.threads);
  const int64_t slots = static_cast<int64_t>(current_device_info().sm_count) * 4 * 128 / s.threads;
  const int64_t tiles = std::max<int64_t>(1, (N + kMomentTile - 1) / kMomentTile);
  int64_t splits = std::max<int64_t>(1, slots / s.groups);
  splits = std::min<int64_t>(std::min<int64_t>(splits, tiles), 2048);
  s.vox_per_split = (((N + splits - 1) / splits + kMomentUnroll - 1) / kMomentUnroll) * kMomentUnroll;
  s.splits = static_cast<int>((N + s.vox_per_split - 1) / s.vox_per_split);
  return s;
}

template <typename T>
cudaError_t launch_cells_backward(const MfArgs& a, unsigned char* ws, cudaStream_t st) {
  const MomentShape sh = moment_shape(a.A, a.N);
  const MomentLayout l = moment_layout(a.A, a.S, sh.splits, 0);
  const PhaseConsts pc = phase_consts(kMfStartFrequency, a.As, a.fs);
  const double kappa = cells_per_metre(pc.k1, a.S, MomentCells::kOver);
  MomentHead* head = reinterpret_cast<MomentHead*>(ws + l.head);
  const int pb = static_cast<int>(std::min<int64_t>(kPrepBlocks, (std::max({a.N, a.S, a.A}) + 255) / 256));

  BoxP<T> bp;
  bp.voxel = static_cast<const T*>(a.voxel);
  bp.gr = static_cast<const T*>(a.grad_real_out);
  bp.gi = static_cast<const T*>(a.grad_imag_out);
  bp.tx = static_cast<const T*>(a.tx);
  bp.rx = static_cast<const T*>(a.rx);
  bp.N = a.N;
  bp.A = a.A;
  bp.S = static_cast<int>(a.S);
  bp.theta_step = 2.0 * M_PI * pc.k1 / kappa;
  bp.box = reinterpret_cast<float*>(ws + l.box);
  bp.basis = reinterpret_cast<float*>(ws + l.basis);
  moment_prep_kernel<T, MomentCells::Q><<<pb, 256, 0, st>>>(bp);
  moment_band_kernel<<<1, 32 * 19, 0, st>>>(bp.box, pb, kappa, head);

  MomentP<T> mp;
  mp.voxel = bp.voxel;
  mp.gr = bp.gr;
  mp.gi = bp.gi;
  mp.tx = bp.tx;
  mp.rx = bp.rx;
  mp.moments = reinterpret_cast<float4*>(ws + l.moments);
  mp.head = head;
  mp.A = a.A;
  mp.N = a.N;
  mp.apad = (a.A + 31) / 32 * 32;
  mp.vox_per_split = sh.vox_per_split;
  mp.ph = pair_phase(pc.k0, pc.b0, pc.k1, pc.b1, a.S, kappa);
  mf_moment_kernel<T><<<dim3(sh.groups, sh.splits), sh.threads, 0, st>>>(mp);

  if (sh.splits > 1) {
    constexpr int pairs = MomentCells::Q / 2;
    mf_moment_sum_kernel<<<dim3(static_cast<unsigned>(mp.apad / 32), kMomentCap * pairs), 32 * kSumWarps, 0, st>>>(
        mp.moments, head, mp.apad, sh.splits, pairs);
  }

  SamplesP<T> sp;
  sp.moments = mp.moments;
  sp.basis = bp.basis;
  sp.head = head;
  sp.out_r = static_cast<T*>(a.out_real);
  sp.out_i = static_cast<T*>(a.out_imag);
  sp.A = a.A;
  sp.apad = mp.apad;
  sp.S = bp.S;
  sp.k1 = pc.k1;
  sp.b1 = pc.b1;
  sp.inv_kappa = 1.0 / kappa;
  const dim3 grid(static_cast<unsigned>((a.A + kSampleAnts - 1) / kSampleAnts), static_cast<unsigned>((a.S + 127) / 128));
  mf_moment_samples_kernel<T><<<grid, 128, 0, st>>>(sp);
  return cudaGetLastError();
}

}  // namespace

// The cells take over where the pairs outweigh the tables and the extra
// launches: enough voxels per table row, and a direct call of more than ~20 us.
// MIXED forwards of up to 128 antennas keep the direct kernel although the cells are the faster and the
// more exact form there too (128 antennas x 256 samples, points along 2048 rays: 1.33 ms against about a
// fifth): the gradient of |y| divides by |y|, which turns the direct kernel's ~2e-6 near theta = 0 into 3e-5
// of a training step's gradients.  The line is drawn for the sake of those values; nothing in the
// kernels asks for it.
// The NUFFT form goes the same way from 8 taps on (fewer taps are a coarser form
// of their own), its forward with the accurate phasor (64-bit error 1.3e-7 by 8 taps,
// 1.2e-7 so, 1.7e-7 with the hardware phasor; the adjoint's 1.1e-6 becomes 5e-7 either way).
bool cells_apply(const MfArgs& a, int taps, int64_t min_antennas) {
  if (a.mode == kPlain || (a.mode == kNufft && taps < 8)) return false;
  return !a.direct_only && a.dtype != kF64 && a.S >= 32 && a.S <= 4096 && a.N >= 512 && a.A >= min_antennas &&
         static_cast<double>(a.A) * a.N * a.S >= 1.0e8;
}

bool mf_cells_forward_applies(const MfArgs& a, int taps) { return cells_apply(a, taps, a.mode == kMixed ? 129 : 24); }

size_t mf_cells_forward_workspace(const MfArgs& a, size_t direct_partial_bytes) {
  const int splits = gather_splits(a.A, a.N);
  const size_t partial = splits > 1 ? static_cast<size_t>(splits) * a.N * sizeof(float2) : 0;
  return cell_layout(a.A, a.S, static_cast<int64_t>(std::max(partial, direct_partial_bytes))).total;
}

size_t mf_cells_forward_partial_offset(const MfArgs& a) { return cell_layout(a.A, a.S, 0).partial; }

bool mf_cells_scale_ok(const MfArgs& a) {
  const PhaseConsts pc = phase_consts(kMfStartFrequency, a.As, a.fs);
  const double kappa = GatherCells::kOver * static_cast<double>(a.S) * std::fabs(pc.k1);
  return std::isfinite(kappa) && kappa >= 1e-2 && kappa <= 1e5;
}

const int* mf_cells_bad_flag(void* ws) { return &static_cast<CellHead*>(ws)->bad; }

cudaError_t mf_cells_forward(const MfArgs& a, void* ws, cudaStream_t st) {
  const int splits = gather_splits(a.A, a.N);
  const CellLayout l = cell_layout(a.A, a.S, 0);
  unsigned char* base = static_cast<unsigned char*>(ws);
  if (a.dtype == kF16) return launch_cells_forward<__half>(a, base, l, splits, st);
  return launch_cells_forward<float>(a, base, l, splits, st);
}

// The adjoint's work is the pairs' too; a lane of its warps is an antenna.
bool mf_cells_backward_applies(const MfArgs& a, int taps) { return cells_apply(a, taps, 24); }

size_t mf_cells_backward_workspace(const MfArgs& a, size_t direct_partial_bytes) {
  return moment_layout(a.A, a.S, moment_shape(a.A, a.N).splits, direct_partial_bytes).total;
}

size_t mf_cells_backward_partial_offset(const MfArgs& a) {
  return moment_layout(a.A, a.S, moment_shape(a.A, a.N).splits, 0).partial;
}

const int* mf_moments_bad_flag(void* ws) { return &static_cast<MomentHead*>(ws)->bad; }

cudaError_t mf_cells_backward(const MfArgs& a, void* ws, cudaStream_t st) {
  unsigned char* base = static_cast<unsigned char*>(ws);
  if (a.dtype == kF16) return launch_cells_backward<__half>(a, base, st);
  return launch_cells_backward<float>(a, base, st);
}

}  // namespace geraf
