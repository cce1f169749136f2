// MIXED tracer adjoint through range cells: per live (point, antenna) pair the sums
// over the residual row g[a, :] that the gradients need come from a polynomial of the
// path length and its derivative (tracer_gradients.cuh), whose coefficients per cell
// are formed once per antenna (range_cells.cuh, the matched filter's table).
//
// Launches: the band of cells from the boxes of the listed points and of the
// antennas, with the interpolation basis; the antennas' tables; the pairs.  Where the
// band does not fit adj_cells() cells, or has more than kFreeCells and too few points for
// them, the pairs are left to the general kernel (tracer_kernels.cu), which returns at once
// otherwise.
#include <algorithm>
#include <cmath>

#include "kernels.h"
#include "tracer_gradients.cuh"

namespace geraf {
namespace {

using namespace tracer;

constexpr int kQ = GatherCells::Q;
constexpr int kBandThreads = 1024;
constexpr int kTableThreads = 256;  // (128: 4 us more for few antennas)
constexpr int kTableCells = 16;  // cells per block of the table kernel, at most
// Up to this many cells cost little whatever the points; more are worth their tables from
// kCellPoints listed points per cell on (64 antennas, 3200 cells, 26000 and 262144 points of 128
// samples: 183 and 411 us, 186 and 1187 us by the general kernel; 5 points per cell: 97 us
// against 86 us).
constexpr int kFreeCells = 512;
constexpr int kCellPoints = 8;
// Cells that a call has room for, per antenna: those that its points can be worth (the tables of 169
// antennas and 4 points would take 50 MB otherwise, not 4), up to 4096 (77 m of path at 4 GHz swept, several
// times the unambiguous path of 1000 samples) and 100 MB of tables; 128 (2.4 m) for large arrays.
int64_t adj_cells(int64_t A, int64_t P) {
  if (A > 2048) return 128;
  const int64_t room = (int64_t{1} << 21) / std::max<int64_t>(A, 1);
  const int64_t worth = std::max<int64_t>(kFreeCells, (P + kCellPoints - 1) / kCellPoints);
  return std::min(std::min<int64_t>(4096, room), worth + kTableCells - 1) / kTableCells * kTableCells;
}
constexpr int kFewAntennas = 64;  // for tables of 4 cells a block
constexpr int kPairThreads = 128;
constexpr int kPairAnts = 32;    // antennas staged at a time

struct AdjHead {
  int bad;
  int k0, cells;
  int pad;
};

struct AdjLayout {
  size_t head, boxes, basis, table, total;
};

size_t up256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

AdjLayout adj_layout(const TracerArgs& a) {
  AdjLayout l;
  l.head = 0;
  l.boxes = 256;
  l.basis = up256(l.boxes + static_cast<size_t>(tracer_point_chunks(a.P)) * 6 * sizeof(float));
  l.table = up256(l.basis + static_cast<size_t>(a.S) * kQ * sizeof(float));
  l.total = up256(l.table + static_cast<size_t>(a.A) * adj_cells(a.A, a.P) * kQ * sizeof(float2));
  return l;
}

template <typename T>
struct BandP {
  const float* boxes;
  int64_t chunks, A;
  const T* tx;
  const T* rx;
  const int* listed;
  AdjHead* head;
  float* basis;
  int max_cells;
  AdjConsts c;
};

// The first block bounds the band; lane groups of 32 x 18 box components would leave most of it idle on
// long chunk lists, so every thread reduces all components over its share.  The others form the
// basis, kBasisSamples each (all of it in the one block took 20 us for 1000 samples).
constexpr int kBasisSamples = 64;
template <typename T>
__global__ void __launch_bounds__(kBandThreads) adj_band_kernel(const BandP<T> p) {
  __shared__ float red[kBandThreads / 32][18];
  __shared__ float box[18];
  if (blockIdx.x > 0) {
    const int n = (blockIdx.x - 1) * kBasisSamples + threadIdx.x;
    if (threadIdx.x >= kBasisSamples || n >= p.c.S) return;
    float g[kQ];
    cell_basis<kQ>(p.c.theta_step * (n - 0.5 * (p.c.S - 1)), g);
#pragma unroll
    for (int q = 0; q < kQ; ++q) p.basis[static_cast<int64_t>(n) * kQ + q] = g[q];
    return;
  }
  float b[18];
#pragma unroll
  for (int c = 0; c < 18; ++c) b[c] = c % 6 < 3 ? INFINITY : -INFINITY;
  for (int64_t i = threadIdx.x; i < p.chunks; i += kBandThreads) {
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const float x = p.boxes[i * 6 + c];
      b[c] = c < 3 ? fminf(b[c], x) : fmaxf(b[c], x);
    }
  }
  for (int64_t a = threadIdx.x; a < p.A; a += kBandThreads) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float t = ld_f(p.tx, a * 3 + c), r = ld_f(p.rx, a * 3 + c);
      // a NaN antenna widens its box to infinity
      b[6 + c] = fminf(b[6 + c], t == t ? t : -INFINITY);
      b[9 + c] = fmaxf(b[9 + c], t == t ? t : INFINITY);
      b[12 + c] = fminf(b[12 + c], r == r ? r : -INFINITY);
      b[15 + c] = fmaxf(b[15 + c], r == r ? r : INFINITY);
    }
  }
#pragma unroll
  for (int c = 0; c < 18; ++c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float y = __shfl_xor_sync(0xffffffffu, b[c], o);
      b[c] = c % 6 < 3 ? fminf(b[c], y) : fmaxf(b[c], y);
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][c] = b[c];
  }
  __syncthreads();
  if (threadIdx.x < 18) {
    const int c = threadIdx.x;
    float r = red[0][c];
    for (int w = 1; w < kBandThreads / 32; ++w) r = c % 6 < 3 ? fminf(r, red[w][c]) : fmaxf(r, red[w][c]);
    box[c] = r;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  double near[2] = {0.0, 0.0}, far[2] = {0.0, 0.0};
  for (int k = 0; k < 3; ++k) {
    const double lo = box[k], hi = box[3 + k];
    for (int e = 0; e < 2; ++e) {
      const double alo = box[6 + 6 * e + k], ahi = box[9 + 6 * e + k];
      const double gap = fmax(0.0, fmax(lo - ahi, alo - hi)), reach = fmax(hi - alo, ahi - lo);
      near[e] += gap * gap;
      far[e] += reach * reach;
    }
  }
  const double lo = floor((sqrt(near[0]) + sqrt(near[1])) * p.c.kappa) - 1.0;
  const double hi = ceil((sqrt(far[0]) + sqrt(far[1])) * p.c.kappa) + 1.0;
  const bool none = box[0] > box[3];  // no listed point: no pairs either
  const double cells = hi - lo + 1.0;
  const bool fits = none || (cells <= p.max_cells && hi < 1073741824.0 &&  // false for NaN
                             (cells <= kFreeCells || cells * kCellPoints <= *p.listed));
  p.head->bad = fits ? 0 : 1;
  p.head->k0 = fits && !none ? static_cast<int>(lo) : 0;
  p.head->cells = fits && !none ? static_cast<int>(hi - lo) + 1 : 0;
}

template <typename T>
struct AdjTableP {
  const T* gr;
  const T* gi;
  const float* basis;
  AdjHead* head;
  float2* table;  // [A][max_cells][kQ]
  int max_cells;
  AdjConsts c;
};

// Block (antenna, groups of CELLS cells y, y + gridDim.y, ...): thread (cell, slice of the samples) as in the
// matched filter's table.  A thread is one chain of its slice's samples, so few antennas take 4
// cells and 64 slices: the adjoint of 1 antenna x 4096 points x 1000 samples 43 us with 16 cells, 27 us so, 48 x
// 100000 x 1000 72 and 55 us, but 64 x 524288 x 128 151 and 152, 250 x 100000 x 128 123 and 135.
template <typename T, int CELLS>
__global__ void __launch_bounds__(kTableThreads) adj_table_kernel(const AdjTableP<T> p) {
  constexpr int kSlices = kTableThreads / CELLS;
  __shared__ float2 red[kSlices][CELLS][kQ];
  const int cells = p.head->cells;
  const int64_t a = blockIdx.x;
  const int slice = threadIdx.x / CELLS;
  const double mid = 0.5 * (p.c.S - 1);
  for (int first = static_cast<int>(blockIdx.y) * CELLS; first < cells; first += gridDim.y * CELLS) {
    const int cell = first + threadIdx.x % CELLS;
    const double dk = fma(p.c.k1, static_cast<double>(p.head->k0 + cell) / p.c.kappa, p.c.b1);
    float2 acc[kQ];
#pragma unroll
    for (int q = 0; q < kQ; ++q) acc[q] = make_float2(0.0f, 0.0f);
    for (int n = slice; n < p.c.S; n += kSlices) {
      const double ph = (n - mid) * dk;
      const float2 e = cis_cycles(static_cast<float>(ph - rint(ph)));
      const float xr = ld_f(p.gr, a * p.c.S + n), xi = ld_f(p.gi, a * p.c.S + n);
      // an infinite residual is the general kernel's (the polynomial would make a NaN of it)
      if (fabsf(xr) == INFINITY || fabsf(xi) == INFINITY) p.head->bad = 1;
      const float2 v = make_float2(fmaf(xr, e.x, xi * e.y), fmaf(xi, e.x, -xr * e.y));
      const float2 w = make_float2(v.y, -v.x);
#pragma unroll
      for (int q = 0; q < kQ; ++q) {
        const float g = p.basis[static_cast<int64_t>(n) * kQ + q];
        acc[q] = ffma2(make_float2(g, g), (q & 1) ? w : v, acc[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < kQ; ++q) red[slice][threadIdx.x % CELLS][q] = acc[q];
    __syncthreads();
    float2* out = p.table + (a * p.max_cells + first) * kQ;
    const int live = min(CELLS, cells - first);
    for (int i = threadIdx.x; i < live * kQ; i += kTableThreads) {
      // slices in fours, then the fours
      float2 s = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int k = 0; k < kSlices; k += 4) {
        const float2 a4 = fadd2((&red[k][0][0])[i], (&red[k + 1][0][0])[i]);
        const float2 b4 = fadd2((&red[k + 2][0][0])[i], (&red[k + 3][0][0])[i]);
        s = fadd2(s, fadd2(a4, b4));
      }
      out[i] = s;
    }
    __syncthreads();
  }
}

template <typename T>
struct AdjPairP {
  const T* normals;
  const T* sigmas;
  const T* points;
  const T* tx;
  const T* rx;
  T* g_normals;
  T* g_sigmas;
  T* g_points;
  const int* plist;
  const int* plist_count;
  const float2* table;
  const AdjHead* head;
  float* partial;  // [splits][P][6]
  int64_t A, P, per_split;
  int splits, max_cells;
  AdjConsts c;
};

// One thread per listed point, the antennas of the block's split in order; nothing is
// shared but the antennas' positions, so the warps run free of barriers.  About 260
// instructions per live pair, independent of the sample count: 64 antennas x 52000 listed
// points take 77 us, 282 us with two recurrences over 128 samples per live pair.
template <typename T, bool WITH_POINTS>
__global__ void __launch_bounds__(kPairThreads, 5) adj_pair_kernel(const AdjPairP<T> p) {
  __shared__ float ant[kPairAnts][6];
  if (p.head->bad) return;
  const int64_t count = *p.plist_count;
  const int64_t tiles = (count + kPairThreads - 1) / kPairThreads * p.splits;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int split = static_cast<int>(tile % p.splits);
    const int64_t base = tile / p.splits * kPairThreads;
    const bool inside = base + threadIdx.x < count;
    const int64_t q = p.plist[min(base + threadIdx.x, count - 1)];
    const int k0 = p.head->k0, cells = p.head->cells;
    float nrm[3], pt[3];
  #pragma unroll
    for (int c = 0; c < 3; ++c) {
      nrm[c] = ld_f(p.normals, q * 3 + c);
      pt[c] = ld_f(p.points, q * 3 + c);
    }
    float gn[3] = {0.0f, 0.0f, 0.0f}, gp[3] = {0.0f, 0.0f, 0.0f};
    const int64_t a_begin = split * p.per_split, a_end = min(p.A, a_begin + p.per_split);
    const float num_points = static_cast<float>(p.P);
    for (int64_t a0 = a_begin; a0 < a_end; a0 += kPairAnts) {
      const int rows = static_cast<int>(min(static_cast<int64_t>(kPairAnts), a_end - a0));
      __syncthreads();
      for (int i = threadIdx.x; i < rows * 6; i += kPairThreads) {
        const int r = i / 6, c = i % 6;
        ant[r][c] = c < 3 ? ld_f(p.tx, (a0 + r) * 3 + c) : ld_f(p.rx, (a0 + r) * 3 + c - 3);
      }
      __syncthreads();
      if (!inside) continue;
      float sigma = ld_f(p.sigmas, a0 * p.P + q);
      for (int r = 0; r < rows; ++r) {
        const int64_t a = a0 + r;
        const float sigma_value = sigma;
        if (r + 1 < rows) sigma = ld_f(p.sigmas, (a + 1) * p.P + q);
        float txp[3], rxp[3];
  #pragma unroll
        for (int c = 0; c < 3; ++c) {
          txp[c] = ant[r][c];
          rxp[c] = ant[r][3 + c];
        }
        PairGeom g;
        if (!pair_geometry(txp, rxp, nrm, pt, g)) {
          p.g_sigmas[a * p.P + q] = from_f<T>(0.0f);
          continue;
        }
        const PairPath path = pair_path(p.c, txp, rxp, pt);
        const int k = min(max(static_cast<int>(path.cell) - k0, 0), cells - 1);
        const float4* row = reinterpret_cast<const float4*>(p.table + (a * p.max_cells + k) * kQ);
        const float4 c2 = __ldg(row + 2), c1 = __ldg(row + 1), c0 = __ldg(row);
        float gs;
        const float2 sums = cell_sums(p.c, path, c0, c1, c2);
        pair_gradients<WITH_POINTS>(g, sums.x, sums.y, sigma_value, nrm, &gs, gn, gp);
        p.g_sigmas[a * p.P + q] = from_f<T>(gs / num_points);
      }
    }
    if (!inside) continue;
    if (p.splits == 1) {
  #pragma unroll
      for (int c = 0; c < 3; ++c) {
        p.g_normals[q * 3 + c] = from_f<T>(gn[c] / num_points);
        if (WITH_POINTS) p.g_points[q * 3 + c] = from_f<T>(gp[c] / num_points);
      }
    } else {
      float* dst = p.partial + (split * p.P + q) * 6;
  #pragma unroll
      for (int c = 0; c < 3; ++c) {
        dst[c] = gn[c];
        dst[3 + c] = gp[c];
      }
    }
  }
}

template <typename T>
cudaError_t launch_adjoint(const TracerArgs& a, unsigned char* ws, PointList list, float* partial, int splits,
                           cudaStream_t st) {
  const AdjLayout l = adj_layout(a);
  const PhaseConsts pc = phase_consts(a.f0, a.As, a.fs);
  const AdjConsts c = adj_consts(pc.k0, pc.b0, pc.k1, pc.b1, a.f0, a.As, a.fs, a.S);
  AdjHead* head = reinterpret_cast<AdjHead*>(ws + l.head);

  BandP<T> bp;
  bp.boxes = reinterpret_cast<const float*>(ws + l.boxes);
  bp.chunks = tracer_point_chunks(a.P);
  bp.A = a.A;
  bp.tx = static_cast<const T*>(a.tx);
  bp.rx = static_cast<const T*>(a.rx);
  bp.listed = list.count;
  bp.head = head;
  bp.basis = reinterpret_cast<float*>(ws + l.basis);
  bp.max_cells = static_cast<int>(adj_cells(a.A, a.P));
  bp.c = c;
  adj_band_kernel<T><<<1 + (c.S + kBasisSamples - 1) / kBasisSamples, kBandThreads, 0, st>>>(bp);

  AdjTableP<T> tp;
  tp.gr = static_cast<const T*>(a.grad_real_out);
  tp.gi = static_cast<const T*>(a.grad_imag_out);
  tp.basis = bp.basis;
  tp.head = head;
  tp.table = reinterpret_cast<float2*>(ws + l.table);
  tp.max_cells = bp.max_cells;
  tp.c = c;
  const unsigned antennas = static_cast<unsigned>(a.A), cells = std::min(bp.max_cells, kFreeCells);
  if (a.A < kFewAntennas) adj_table_kernel<T, 4><<<dim3(antennas, cells / 4), kTableThreads, 0, st>>>(tp);
  else adj_table_kernel<T, kTableCells><<<dim3(antennas, cells / kTableCells), kTableThreads, 0, st>>>(tp);

  AdjPairP<T> pp;
  pp.normals = static_cast<const T*>(a.normals);
  pp.sigmas = static_cast<const T*>(a.sigmas);
  pp.points = static_cast<const T*>(a.points);
  pp.tx = bp.tx;
  pp.rx = bp.rx;
  pp.g_normals = static_cast<T*>(a.grad_normals);
  pp.g_sigmas = static_cast<T*>(a.grad_sigmas);
  pp.g_points = static_cast<T*>(a.grad_points);
  pp.plist = list.list;
  pp.plist_count = list.count;
  pp.table = tp.table;
  pp.head = head;
  pp.partial = partial;
  pp.A = a.A;
  pp.P = a.P;
  pp.splits = splits;
  pp.per_split = (a.A + splits - 1) / splits;
  pp.max_cells = bp.max_cells;
  pp.c = c;
  // the number of listed points is on the device only: a few waves of blocks take its tiles in turn
  const int64_t blocks = std::min<int64_t>((a.P + kPairThreads - 1) / kPairThreads * splits,
                                           static_cast<int64_t>(current_device_info().sm_count) * 40);
  if (a.grad_points != nullptr) adj_pair_kernel<T, true><<<static_cast<unsigned>(blocks), kPairThreads, 0, st>>>(pp);
  else adj_pair_kernel<T, false><<<static_cast<unsigned>(blocks), kPairThreads, 0, st>>>(pp);
  return cudaGetLastError();
}

}  // namespace

bool tracer_adjoint_cells_apply(const TracerArgs& a) {
  return a.mode == kMixed && tracer_point_list_applies(a) && a.A > 0 && a.S >= 32 && a.S <= 4096;
}

size_t tracer_adjoint_cells_workspace(const TracerArgs& a) { return adj_layout(a).total; }

float* tracer_adjoint_cells_boxes(void* ws) { return reinterpret_cast<float*>(static_cast<unsigned char*>(ws) + 256); }

cudaError_t tracer_adjoint_cells(const TracerArgs& a, void* ws, PointList list, float* partial, int splits, cudaStream_t st,
                                 const int** bad) {
  unsigned char* base = static_cast<unsigned char*>(ws);
  *bad = &reinterpret_cast<AdjHead*>(base)->bad;
  if (a.dtype == kF64) return launch_adjoint<double>(a, base, list, partial, splits, st);
  return launch_adjoint<float>(a, base, list, partial, splits, st);
}

}  // namespace geraf
