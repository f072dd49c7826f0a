// Causal attention, exact family: the cached opcodes (probabilities kept in
// the arena) and the tiled opcodes (four statistics per query row, every
// probability recomputed) evaluated with the CPU executor's own expressions —
// dot products accumulated in double in ascending feature order (a product of
// two floats is exact in double, so the fused and unfused forms coincide),
// the 1/sqrt(d) scale and the softmax in f32, output sums in f32 in ascending
// key (or query) order without fused multiply-adds (-fmad=false)
// (reference: runtime/executor/attention.cc:187-343 cached, :448-590 tiled).
// What is not sequential here are the two per-row double sums (softmax
// denominator, the backward's rowsum): lane partials folded by a shuffle
// tree, a fixed order that can differ from the CPU's in the last bit of the
// double.  Activations are [B*S, H*d] row-major with heads interleaved along
// the row.
//
// Two sets of kernels give the same bits.
//
// The tile kernels (AttnFwdTile, AttnDPTile, AttnRowTile, AttnColTile,
// AttnDQTiledTile, AttnDKVTiledTile) are FP64-bound: a block owns 16, 32 or 64
// query (or key) rows of one (sequence, head) and takes the other axis 64 at a
// time.  Both operands of a score tile are widened to double once, while they
// are copied to shared memory (a conversion costs four FMA slots, so per use it
// would be the bound), features slowest, and a thread accumulates RM x 4 pairs
// in registers: RM + 4 shared doubles per 4 RM fused multiply-adds, each
// accumulator one chain over ascending features.  The f32 output sums are the
// same shape of product, 64 columns of the head at a time, RM x 4 outputs per
// thread, each one chain over ascending keys.
// One warp per row with a strided K row per lane (the row kernels below) took
// 3747 us for 8 x 512 positions of 12 heads of 64 features and 320 us for
// 32 x 128 of 4 heads.
//
// The row kernels (one warp owns one row and keeps its whole score row in shared
// memory) remain for rows too long for a tile block's score rows.
#include <initializer_list>
#include <type_traits>

#include "kernels.h"

namespace see::k {

namespace {

constexpr int kWarps = 4;

__device__ __forceinline__ double WarpSumD(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  return v;
}
__device__ __forceinline__ float WarpMaxF(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  return v;
}

// a (in shared memory) . row (global), accumulated in double, ascending c.
__device__ __forceinline__ double DotD(const float* a, const float* __restrict__ row, size_t d) {
  double acc = 0.0;
  for (size_t c = 0; c < d; ++c) acc += static_cast<double>(a[c]) * static_cast<double>(row[c]);
  return acc;
}

__device__ __forceinline__ size_t StatsStart(float stored, size_t i) {
  if (!(stored > 0.0f)) return 0;
  const float cap = static_cast<float>(i);
  return stored >= cap ? i : static_cast<size_t>(stored);
}

struct Unit { size_t b, h, i; };
__device__ __forceinline__ Unit UnitOf(size_t u, size_t H, size_t S) {
  return {u / (H * S), (u / S) % H, u % S};
}

// Shared memory per warp: d floats (the unit's query-side row) then `rows`
// rows of S floats.
__device__ __forceinline__ float* WarpSmem(float* base, size_t d, size_t S, int rows) {
  return base + (threadIdx.x >> 5) * (d + static_cast<size_t>(rows) * S);
}

__global__ void AttnFwdKernel(const float* __restrict__ q, const float* __restrict__ k,
                              const float* __restrict__ v, float* __restrict__ o,
                              float* __restrict__ probs, float* __restrict__ stats, size_t B,
                              size_t S, size_t H, size_t d, const int32_t* __restrict__ starts,
                              float inv_sqrt_d) {
  extern __shared__ float smem[];
  float* qs = WarpSmem(smem, d, S, 1);
  float* prow = qs + d;
  const int lane = threadIdx.x & 31;
  const size_t D = H * d, units = B * H * S;
  for (size_t u = blockIdx.x * static_cast<size_t>(kWarps) + (threadIdx.x >> 5); u < units;
       u += static_cast<size_t>(gridDim.x) * kWarps) {
    const Unit un = UnitOf(u, H, S);
    const size_t b = un.b, h = un.h, i = un.i;
    const float* qi = q + (b * S + i) * D + h * d;
    for (size_t c = lane; c < d; c += 32) qs[c] = qi[c];
    __syncwarp();
    size_t j0 = 0;
    if (starts) {
      const int32_t s0 = starts[b * S + i];
      j0 = s0 <= 0 ? 0 : (static_cast<size_t>(s0) < i ? static_cast<size_t>(s0) : i);
    }
    const float* kb = k + b * S * D + h * d;
    float row_max = -INFINITY;
    for (size_t j = j0 + lane; j <= i; j += 32) {
      const float sc = static_cast<float>(DotD(qs, kb + j * D, d)) * inv_sqrt_d;
      prow[j] = sc;
      row_max = fmaxf(row_max, sc);
    }
    row_max = WarpMaxF(row_max);
    double denom = 0.0;
    for (size_t j = j0 + lane; j <= i; j += 32) {
      const float e = expf(prow[j] - row_max);
      prow[j] = e;
      denom += static_cast<double>(e);
    }
    denom = WarpSumD(denom);
    const float inv_denom = 1.0f / static_cast<float>(denom);
    for (size_t j = j0 + lane; j <= i; j += 32) prow[j] *= inv_denom;
    __syncwarp();
    if (probs) {
      float* grow = probs + u * S;
      for (size_t j = lane; j < S; j += 32) grow[j] = (j >= j0 && j <= i) ? prow[j] : 0.0f;
    }
    const float* vb = v + b * S * D + h * d;
    float* oi = o + (b * S + i) * D + h * d;
    for (size_t c = lane; c < d; c += 32) {
      float acc = 0.0f;
      for (size_t j = j0; j <= i; ++j) acc += prow[j] * vb[j * D + c];
      oi[c] = acc;
    }
    if (stats && lane == 0) {
      float* st = stats + u * kAttnStatsWidth;
      st[0] = row_max;
      st[1] = inv_denom;
      st[2] = 0.0f;
      st[3] = static_cast<float>(j0);
    }
    __syncwarp();
  }
}

// dS = P * (dP - rowsum(dP * P)), the rowsum in double.
__global__ void SoftmaxRowsBwdKernel(const float* __restrict__ probs, const float* __restrict__ dp,
                                     float* __restrict__ ds, size_t rows, size_t cols) {
  const int lane = threadIdx.x & 31;
  for (size_t r = blockIdx.x * static_cast<size_t>(kWarps) + (threadIdx.x >> 5); r < rows;
       r += static_cast<size_t>(gridDim.x) * kWarps) {
    const float* pr = probs + r * cols;
    const float* dpr = dp + r * cols;
    float* dsr = ds + r * cols;
    double dot = 0.0;
    for (size_t c = lane; c < cols; c += 32)
      dot += static_cast<double>(dpr[c]) * static_cast<double>(pr[c]);
    const float sum = static_cast<float>(WarpSumD(dot));
    for (size_t c = lane; c < cols; c += 32) dsr[c] = pr[c] * (dpr[c] - sum);
  }
}

// Tiled dQ: recomputes the row's probabilities and dP, writes delta into the
// stats row, then dQ (reference: runtime/executor/attention.cc:492-531).
__global__ void AttnDQTiledKernel(const float* __restrict__ q, const float* __restrict__ k,
                                  const float* __restrict__ v, const float* __restrict__ dout,
                                  float* __restrict__ stats, float* __restrict__ dq, size_t B,
                                  size_t S, size_t H, size_t d, float inv_sqrt_d) {
  extern __shared__ float smem[];
  // per warp: q row (d), dO row (d) packed as 2d, then prow (S), dprow (S)
  float* base = smem + (threadIdx.x >> 5) * (2 * d + 2 * S);
  float* qs = base;
  float* dos = base + d;
  float* prow = base + 2 * d;
  float* dprow = prow + S;
  const int lane = threadIdx.x & 31;
  const size_t D = H * d, units = B * H * S;
  for (size_t u = blockIdx.x * static_cast<size_t>(kWarps) + (threadIdx.x >> 5); u < units;
       u += static_cast<size_t>(gridDim.x) * kWarps) {
    const Unit un = UnitOf(u, H, S);
    const size_t b = un.b, h = un.h, i = un.i;
    const float* qi = q + (b * S + i) * D + h * d;
    const float* doi = dout + (b * S + i) * D + h * d;
    for (size_t c = lane; c < d; c += 32) {
      qs[c] = qi[c];
      dos[c] = doi[c];
    }
    float* st = stats + u * kAttnStatsWidth;
    const float m = st[0], inv_denom = st[1];
    const size_t j0 = StatsStart(st[3], i);
    __syncwarp();
    const float* kb = k + b * S * D + h * d;
    const float* vb = v + b * S * D + h * d;
    double dot = 0.0;
    for (size_t j = j0 + lane; j <= i; j += 32) {
      const float sc = static_cast<float>(DotD(qs, kb + j * D, d)) * inv_sqrt_d;
      const float p = expf(sc - m) * inv_denom;
      const float dpv = static_cast<float>(DotD(dos, vb + j * D, d));
      prow[j] = p;
      dprow[j] = dpv;
      dot += static_cast<double>(dpv) * static_cast<double>(p);
    }
    const float delta = static_cast<float>(WarpSumD(dot));
    __syncwarp();
    if (lane == 0) st[2] = delta;
    float* dqi = dq + (b * S + i) * D + h * d;
    for (size_t c = lane; c < d; c += 32) {
      float acc = 0.0f;
      for (size_t j = j0; j <= i; ++j) {
        const float dsv = prow[j] * (dprow[j] - delta);
        acc += (dsv * inv_sqrt_d) * kb[j * D + c];
      }
      dqi[c] = acc;
    }
    __syncwarp();
  }
}

// ---- tile kernels ------------------------------------------------------------------

constexpr int kTile = 64;      // keys (or queries) of the streamed axis per step
constexpr int kSlice = 32;     // features of both operands in shared memory at a time
constexpr int kTileThreads = 256;

// Rows [0, rows) of a [., stride] f32 matrix, features [c0, c0 + kSlice) of d, widened into
// dst[feature][kRows]; what lies outside is zero (0 * 0 leaves a chain as it is).
// Lanes take consecutive rows, so that the stores are conflict-free; a row's 128-byte slice is
// read 16 bytes at a time and stays in L1 between them.
template <int kRows, bool kVec>
__device__ __forceinline__ void LoadSlice(double* dst, const float* __restrict__ src, size_t stride, int rows, int c0,
                                          int d) {
  for (int t = threadIdx.x; t < kRows * (kSlice / 4); t += kTileThreads) {
    const int r = t % kRows, c = t / kRows * 4;
    float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (r < rows && c0 + c < d) {
      const float* p = src + static_cast<size_t>(r) * stride + c0 + c;
      if (kVec) {
        const float4 f = *reinterpret_cast<const float4*>(p);
        x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (c0 + c + e < d) x[e] = p[e];
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) dst[(c + e) * kRows + r] = static_cast<double>(x[e]);
  }
}

// acc[r][e] = row (ty RM + r) of `a` . row Col(e) of `b`, in double, ascending features.
// Starts with a barrier (the slices may still be in use) and leaves none behind.
template <int RM, bool kVec>
__device__ __forceinline__ void DotTile(const float* a, int a_rows, const float* b, int b_rows, size_t stride, int d,
                                        double* sa, double* sb, double (&acc)[RM][4]) {
  constexpr int R = 16 * RM;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int r = 0; r < RM; ++r)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[r][e] = 0.0;
  for (int c0 = 0; c0 < d; c0 += kSlice) {
    __syncthreads();
    LoadSlice<R, kVec>(sa, a, stride, a_rows, c0, d);
    LoadSlice<kTile, kVec>(sb, b, stride, b_rows, c0, d);
    __syncthreads();
#pragma unroll 8
    for (int c = 0; c < kSlice; ++c) {
      double x[RM], y[4];
      const double2 y0 = *reinterpret_cast<const double2*>(sb + c * kTile + 2 * tx);
      const double2 y1 = *reinterpret_cast<const double2*>(sb + c * kTile + 32 + 2 * tx);
      y[0] = y0.x; y[1] = y0.y; y[2] = y1.x; y[3] = y1.y;
#pragma unroll
      for (int r = 0; r < RM; ++r) x[r] = sa[c * R + ty * RM + r];
#pragma unroll
      for (int r = 0; r < RM; ++r)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[r][e] = fma(x[r], y[e], acc[r][e]);
    }
  }
}
// The tile column a thread's accumulator e stands for (pairs, so that 16 lanes read 256 contiguous bytes).
__device__ __forceinline__ int Col(int e) { return 2 * static_cast<int>(threadIdx.x & 15) + (e & 1) + (e >> 1) * 32; }

// Rows [0, rows) x columns [c0, c0 + 64) of a [., stride] f32 matrix into dst[64][64] (zero outside).
template <bool kVec>
__device__ __forceinline__ void LoadTileF(float* dst, const float* __restrict__ src, size_t stride, int rows, int c0,
                                          int d) {
  for (int t = threadIdx.x; t < kTile * 16; t += kTileThreads) {
    const int r = t >> 4, c = (t & 15) * 4;
    float4 f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (r < rows && c0 + c < d) {
      const float* p = src + static_cast<size_t>(r) * stride + c0 + c;
      if (kVec) {
        f = *reinterpret_cast<const float4*>(p);
      } else {
        f.x = p[0];
        if (c0 + c + 1 < d) f.y = p[1];
        if (c0 + c + 2 < d) f.z = p[2];
        if (c0 + c + 3 < d) f.w = p[3];
      }
    }
    *reinterpret_cast<float4*>(dst + r * kTile + c) = f;
  }
}

__device__ __forceinline__ void StoreRow4(float* p, const float (&v)[4], int c, int d, bool vec) {
  if (c >= d) return;
  if (vec) {
    *reinterpret_cast<float4*>(p + c) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (c + e < d) p[c + e] = v[e];
  }
}

// acc[r][e] += w[row][j] * x[j][c + e] for j = 0 .. 63 in order; row's weights at w + r * ld.  A row takes
// j in [lo[r], hi[r]) only (a weight outside is not multiplied: x may hold anything there); kAll: every j.
template <int RM, bool kAll>
__device__ __forceinline__ void RowProduct(const float* w, int ld, const float* x, const int (&lo)[RM],
                                           const int (&hi)[RM], float (&acc)[RM][4]) {
  const int c = (threadIdx.x & 15) * 4;
#pragma unroll 2
  for (int j = 0; j < kTile; j += 4) {
    float p[RM][4];
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const float4 f = *reinterpret_cast<const float4*>(w + r * ld + j);
      p[r][0] = f.x; p[r][1] = f.y; p[r][2] = f.z; p[r][3] = f.w;
    }
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      const float4 f = *reinterpret_cast<const float4*>(x + (j + jj) * kTile + c);
      const float xv[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
      for (int r = 0; r < RM; ++r) {
        if (kAll || (j + jj >= lo[r] && j + jj < hi[r])) {
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[r][e] += p[r][jj] * xv[e];
        }
      }
    }
  }
}

__host__ __device__ constexpr size_t SliceBytes(int RM) { return sizeof(double) * kSlice * (16 * RM + kTile); }
// Score rows are stored with a stride of a whole number of key tiles plus 4 floats (a multiple of 16 bytes that
// puts a thread column's rows in different banks).
__host__ __device__ constexpr size_t RowStride(size_t S) { return (S + kTile - 1) / kTile * kTile + 4; }

// A block's tile and (sequence, head), longest tiles first over the whole grid so that the last wave is short
// blocks: query tiles from the end of the sequence, key tiles from its start.
struct TileAt { int tile; size_t bh; };
__device__ __forceinline__ TileAt QueryTile(int tiles, int BH) {
  return {tiles - 1 - static_cast<int>(blockIdx.x) / BH, static_cast<size_t>(static_cast<int>(blockIdx.x) % BH)};
}
__device__ __forceinline__ TileAt KeyTile(int BH) {
  return {static_cast<int>(blockIdx.x) / BH, static_cast<size_t>(static_cast<int>(blockIdx.x) % BH)};
}

// Forward.  Block: 16 RM query rows of one (sequence, head).  Score rows of the whole block stay in shared memory between the three phases.
template <int RM, bool kVec>
__global__ __launch_bounds__(kTileThreads) void AttnFwdTileKernel(
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, float* __restrict__ o,
    float* __restrict__ probs, float* __restrict__ stats, int BH, int S, int H, int d,
    const int32_t* __restrict__ starts, float inv_sqrt_d) {
  extern __shared__ __align__(16) uint8_t raw[];
  constexpr int R = 16 * RM;
  double* sa = reinterpret_cast<double*>(raw);
  double* sb = sa + kSlice * R;
  float* xt = reinterpret_cast<float*>(sb);                       // the V tile, where the K slice was
  float* rows = reinterpret_cast<float*>(raw + SliceBytes(RM));
  const int ld = static_cast<int>(RowStride(S));
  const TileAt tile = QueryTile((S + R - 1) / R, BH);
  const int i0 = tile.tile * R;
  const size_t bh = tile.bh, b = bh / H, h = bh % H, D = static_cast<size_t>(H) * d;
  const int nrows = min(R, S - i0), nkeys = min(i0 + R, S);
  const int ty = threadIdx.x >> 4, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t base = b * S * D + h * d;
  auto first_key = [&](int i) {
    if (!starts) return 0;
    const int32_t s0 = starts[b * S + i];
    return s0 <= 0 ? 0 : (s0 < i ? static_cast<int>(s0) : i);
  };
  for (int k0 = 0; k0 < nkeys; k0 += kTile) {
    double acc[RM][4];
    DotTile<RM, kVec>(q + base + static_cast<size_t>(i0) * D, nrows, k + base + static_cast<size_t>(k0) * D,
                      min(kTile, S - k0), D, d, sa, sb, acc);
#pragma unroll
    for (int r = 0; r < RM; ++r)
#pragma unroll
      for (int e = 0; e < 4; e += 2)
        *reinterpret_cast<float2*>(rows + (ty * RM + r) * ld + k0 + Col(e)) =
            make_float2(static_cast<float>(acc[r][e]) * inv_sqrt_d, static_cast<float>(acc[r][e + 1]) * inv_sqrt_d);
  }
  __syncthreads();
  for (int r = warp; r < nrows; r += kTileThreads / 32) {
    const int i = i0 + r, j0 = first_key(i);
    float* prow = rows + r * ld;
    float row_max = -INFINITY;
    for (int j = j0 + lane; j <= i; j += 32) row_max = fmaxf(row_max, prow[j]);
    row_max = WarpMaxF(row_max);
    double denom = 0.0;
    for (int j = j0 + lane; j <= i; j += 32) {
      const float e = expf(prow[j] - row_max);
      prow[j] = e;
      denom += static_cast<double>(e);
    }
    denom = WarpSumD(denom);
    const float inv_denom = 1.0f / static_cast<float>(denom);
    for (int j = j0 + lane; j <= i; j += 32) prow[j] *= inv_denom;
    const size_t u = bh * S + i;
    if (probs) {
      __syncwarp();
      float* grow = probs + u * S;
      for (int j = lane; j < S; j += 32) grow[j] = (j >= j0 && j <= i) ? prow[j] : 0.0f;
    }
    if (stats && lane == 0) {
      float* st = stats + u * kAttnStatsWidth;
      st[0] = row_max;
      st[1] = inv_denom;
      st[2] = 0.0f;
      st[3] = static_cast<float>(j0);
    }
  }
  const int c = (threadIdx.x & 15) * 4;
  int row_lo[RM], row_hi[RM];
#pragma unroll
  for (int r = 0; r < RM; ++r) {
    const int i = min(i0 + ty * RM + r, S - 1);
    row_lo[r] = first_key(i);
    row_hi[r] = i + 1;
  }
  for (int c0 = 0; c0 < d; c0 += kTile) {
    float acc[RM][4];
#pragma unroll
    for (int r = 0; r < RM; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[r][e] = 0.0f;
    for (int k0 = 0; k0 < nkeys; k0 += kTile) {
      __syncthreads();
      LoadTileF<kVec>(xt, v + base + static_cast<size_t>(k0) * D, D, min(kTile, S - k0), c0, d);
      __syncthreads();
      int lo[RM], hi[RM];
#pragma unroll
      for (int r = 0; r < RM; ++r) { lo[r] = row_lo[r] - k0; hi[r] = row_hi[r] - k0; }
      if (!starts && k0 + kTile <= i0 + 1)
        RowProduct<RM, true>(rows + ty * RM * ld + k0, ld, xt, lo, hi, acc);
      else
        RowProduct<RM, false>(rows + ty * RM * ld + k0, ld, xt, lo, hi, acc);
    }
#pragma unroll
    for (int r = 0; r < RM; ++r)
      if (ty * RM + r < nrows)
        StoreRow4(o + base + static_cast<size_t>(i0 + ty * RM + r) * D, acc[r], c0 + c, d, kVec);
  }
}

// dP[i][j] = dO_i . v_j for j <= i, zero above the diagonal.  Block: one 64 x 64 tile.
template <bool kVec>
__global__ __launch_bounds__(kTileThreads) void AttnDPTileKernel(const float* __restrict__ dout,
                                                                 const float* __restrict__ v, float* __restrict__ dp,
                                                                 int BH, int S, int H, int d) {
  extern __shared__ __align__(16) uint8_t raw[];
  double* sa = reinterpret_cast<double*>(raw);
  double* sb = sa + kSlice * kTile;
  const TileAt tile = KeyTile(BH);
  const int tiles = (S + kTile - 1) / kTile, k0 = tile.tile % tiles * kTile, i0 = tile.tile / tiles * kTile;
  const size_t bh = tile.bh, b = bh / H, h = bh % H, D = static_cast<size_t>(H) * d;
  const size_t base = b * S * D + h * d;
  const int ty = threadIdx.x >> 4;
  double acc[4][4] = {};
  if (k0 <= i0)
    DotTile<4, kVec>(dout + base + static_cast<size_t>(i0) * D, min(kTile, S - i0),
                     v + base + static_cast<size_t>(k0) * D, min(kTile, S - k0), D, d, sa, sb, acc);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + ty * 4 + r;
    if (i >= S) continue;
    float* row = dp + (bh * S + i) * S;
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      const int j = k0 + Col(e);
      const float x0 = j <= i ? static_cast<float>(acc[r][e]) : 0.0f;
      const float x1 = j + 1 <= i ? static_cast<float>(acc[r][e + 1]) : 0.0f;
      if ((S & 1) == 0 && j + 1 < S) {
        *reinterpret_cast<float2*>(row + j) = make_float2(x0, x1);
      } else {
        if (j < S) row[j] = x0;
        if (j + 1 < S) row[j + 1] = x1;
      }
    }
  }
}

// dQ_i[c] = sum over j <= i of (dS[i][j] / sqrt(d)) k_j[c].  Block: 16 RM rows, 64 columns of the head.
template <int RM, bool kVec>
__global__ __launch_bounds__(kTileThreads) void AttnRowTileKernel(const float* __restrict__ ds,
                                                                  const float* __restrict__ k, float* __restrict__ dq,
                                                                  int BH, int S, int H, int d, float inv_sqrt_d) {
  constexpr int R = 16 * RM, kLd = kTile + 4;
  __shared__ __align__(16) float xt[kTile * kTile];
  __shared__ __align__(16) float wt[R * kLd];
  const TileAt tile = QueryTile((S + R - 1) / R, BH);
  const int i0 = tile.tile * R;
  const size_t bh = tile.bh, b = bh / H, h = bh % H, D = static_cast<size_t>(H) * d;
  const size_t base = b * S * D + h * d;
  const int c0 = blockIdx.y * kTile, ty = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
  const int nkeys = min(i0 + R, S);
  float acc[RM][4] = {};
  for (int k0 = 0; k0 < nkeys; k0 += kTile) {
    __syncthreads();
    LoadTileF<kVec>(xt, k + base + static_cast<size_t>(k0) * D, D, min(kTile, S - k0), c0, d);
    for (int t = threadIdx.x; t < R * kTile; t += kTileThreads) {
      const int r = t / kTile, j = t % kTile;
      wt[r * kLd + j] = i0 + r < S && k0 + j < S ? ds[(bh * S + i0 + r) * S + k0 + j] * inv_sqrt_d : 0.0f;
    }
    __syncthreads();
    int lo[RM], hi[RM];
#pragma unroll
    for (int r = 0; r < RM; ++r) { lo[r] = 0; hi[r] = i0 + ty * RM + r + 1 - k0; }
    if (k0 + kTile <= i0 + 1) RowProduct<RM, true>(wt + ty * RM * kLd, kLd, xt, lo, hi, acc);
    else RowProduct<RM, false>(wt + ty * RM * kLd, kLd, xt, lo, hi, acc);
  }
#pragma unroll
  for (int r = 0; r < RM; ++r)
    if (i0 + ty * RM + r < S) StoreRow4(dq + base + static_cast<size_t>(i0 + ty * RM + r) * D, acc[r], c0 + c, d, kVec);
}

// acc[r][e] += w[i][ty RM + r] x[i][c + e] for i = 0 .. rows - 1 in order, where query i reaches key row r:
// i >= lo[r], and key[r] >= start[i] when there are segment starts (kAll: every i reaches every key).
template <int RM, bool kAll>
__device__ __forceinline__ void ColProduct(const float* w, int ldw, const float* x, int rows, const int (&lo)[RM],
                                           float (&acc)[RM][4], const int* start = nullptr, int key = 0) {
  const int c = (threadIdx.x & 15) * 4, ty = threadIdx.x >> 4;
#pragma unroll 4
  for (int i = 0; i < rows; ++i) {
    const float4 f = *reinterpret_cast<const float4*>(x + i * kTile + c);
    const float xv[4] = {f.x, f.y, f.z, f.w};
    const int first = kAll || !start ? 0 : start[i];
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const float g = w[i * ldw + ty * RM + r];
      if (kAll || (i >= lo[r] && key + r >= first)) {
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[r][e] += g * xv[e];
      }
    }
  }
}

// out_j[c] = sum over i >= j of w[i][j] (scale) x_i[c], i ascending.  Block: 16 RM keys, 64 columns.
template <int RM, bool kScaled, bool kVec>
__global__ __launch_bounds__(kTileThreads) void AttnColTileKernel(const float* __restrict__ w,
                                                                  const float* __restrict__ x, float* __restrict__ out,
                                                                  int BH, int S, int H, int d, float inv_sqrt_d) {
  constexpr int R = 16 * RM;
  __shared__ __align__(16) float xt[kTile * kTile];
  __shared__ __align__(16) float wt[kTile * R];
  const TileAt tile = KeyTile(BH);
  const int j0 = tile.tile * R;
  const size_t bh = tile.bh, b = bh / H, h = bh % H, D = static_cast<size_t>(H) * d;
  const size_t base = b * S * D + h * d;
  const int c0 = blockIdx.y * kTile, ty = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
  float acc[RM][4] = {};
  for (int i0 = j0; i0 < S; i0 += kTile) {
    const int rows = min(kTile, S - i0);
    __syncthreads();
    LoadTileF<kVec>(xt, x + base + static_cast<size_t>(i0) * D, D, rows, c0, d);
    for (int t = threadIdx.x; t < kTile * R; t += kTileThreads) {
      const int i = t / R, j = t % R;
      float g = i < rows && j0 + j < S ? w[(bh * S + i0 + i) * S + j0 + j] : 0.0f;
      if (kScaled) g = g * inv_sqrt_d;
      wt[t] = g;
    }
    __syncthreads();
    int lo[RM];
#pragma unroll
    for (int r = 0; r < RM; ++r) lo[r] = j0 + ty * RM + r - i0;
    if (i0 >= j0 + R - 1) ColProduct<RM, true>(wt, R, xt, rows, lo, acc);
    else ColProduct<RM, false>(wt, R, xt, rows, lo, acc);
  }
#pragma unroll
  for (int r = 0; r < RM; ++r)
    if (j0 + ty * RM + r < S) StoreRow4(out + base + static_cast<size_t>(j0 + ty * RM + r) * D, acc[r], c0 + c, d, kVec);
}

// Tiled dQ: the rows' probabilities and dP recomputed into shared memory, delta written into the stats rows,
// then dQ (reference: runtime/executor/attention.cc:492-531).
template <int RM, bool kVec>
__global__ __launch_bounds__(kTileThreads) void AttnDQTiledTileKernel(
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
    const float* __restrict__ dout, float* __restrict__ stats, float* __restrict__ dq, int BH, int S, int H,
    int d, float inv_sqrt_d) {
  extern __shared__ __align__(16) uint8_t raw[];
  constexpr int R = 16 * RM;
  double* sa = reinterpret_cast<double*>(raw);
  double* sb = sa + kSlice * R;
  float* xt = reinterpret_cast<float*>(sb);
  const int ld = static_cast<int>(RowStride(S));
  float* prows = reinterpret_cast<float*>(raw + SliceBytes(RM));
  float* dprows = prows + R * ld;
  const TileAt tile = QueryTile((S + R - 1) / R, BH);
  const int i0 = tile.tile * R;
  const size_t bh = tile.bh, b = bh / H, h = bh % H, D = static_cast<size_t>(H) * d;
  const int nrows = min(R, S - i0), nkeys = min(i0 + R, S);
  const int ty = threadIdx.x >> 4, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t base = b * S * D + h * d, at = base + static_cast<size_t>(i0) * D;
  float* st = stats + (bh * S + i0) * kAttnStatsWidth;
  for (int k0 = 0; k0 < nkeys; k0 += kTile) {
    const size_t kat = base + static_cast<size_t>(k0) * D;
    double acc[RM][4];
    DotTile<RM, kVec>(q + at, nrows, k + kat, min(kTile, S - k0), D, d, sa, sb, acc);
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const int row = min(ty * RM + r, nrows - 1);
      const float m = st[row * kAttnStatsWidth], inv_denom = st[row * kAttnStatsWidth + 1];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        prows[(ty * RM + r) * ld + k0 + Col(e)] = expf(static_cast<float>(acc[r][e]) * inv_sqrt_d - m) * inv_denom;
    }
    DotTile<RM, kVec>(dout + at, nrows, v + kat, min(kTile, S - k0), D, d, sa, sb, acc);
#pragma unroll
    for (int r = 0; r < RM; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) dprows[(ty * RM + r) * ld + k0 + Col(e)] = static_cast<float>(acc[r][e]);
  }
  __syncthreads();
  for (int r = warp; r < nrows; r += kTileThreads / 32) {
    const int i = i0 + r, j0 = static_cast<int>(StatsStart(st[r * kAttnStatsWidth + 3], i));
    float* prow = prows + r * ld;
    const float* dprow = dprows + r * ld;
    double dot = 0.0;
    for (int j = j0 + lane; j <= i; j += 32) dot += static_cast<double>(dprow[j]) * static_cast<double>(prow[j]);
    const float delta = static_cast<float>(WarpSumD(dot));
    if (lane == 0) st[r * kAttnStatsWidth + 2] = delta;
    for (int j = j0 + lane; j <= i; j += 32) {
      const float dsv = prow[j] * (dprow[j] - delta);
      prow[j] = dsv * inv_sqrt_d;
    }
  }
  const int c = (threadIdx.x & 15) * 4;
  int row_lo[RM], row_hi[RM];
  bool whole = true;
#pragma unroll
  for (int r = 0; r < RM; ++r) {
    const int row = min(ty * RM + r, nrows - 1);
    row_lo[r] = static_cast<int>(StatsStart(st[row * kAttnStatsWidth + 3], i0 + row));
    row_hi[r] = i0 + row + 1;
    whole = whole && row_lo[r] == 0;
  }
  for (int c0 = 0; c0 < d; c0 += kTile) {
    float acc[RM][4] = {};
    for (int k0 = 0; k0 < nkeys; k0 += kTile) {
      __syncthreads();
      LoadTileF<kVec>(xt, k + base + static_cast<size_t>(k0) * D, D, min(kTile, S - k0), c0, d);
      __syncthreads();
      int lo[RM], hi[RM];
#pragma unroll
      for (int r = 0; r < RM; ++r) { lo[r] = row_lo[r] - k0; hi[r] = row_hi[r] - k0; }
      if (whole && k0 + kTile <= i0 + 1) RowProduct<RM, true>(prows + ty * RM * ld + k0, ld, xt, lo, hi, acc);
      else RowProduct<RM, false>(prows + ty * RM * ld + k0, ld, xt, lo, hi, acc);
    }
#pragma unroll
    for (int r = 0; r < RM; ++r)
      if (ty * RM + r < nrows) StoreRow4(dq + at + static_cast<size_t>(ty * RM + r) * D, acc[r], c0 + c, d, kVec);
  }
}

// Tiled dK (kWantDK) or dV over the query rows i >= j of 16 RM keys, 64 columns of the head per block (a wider
// head repeats the scores; reference: runtime/executor/attention.cc:533-590).
template <int RM, bool kWantDK, bool kVec>
__global__ __launch_bounds__(kTileThreads) void AttnDKVTiledTileKernel(
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
    const float* __restrict__ dout, const float* __restrict__ stats, float* __restrict__ out, int BH, int S, int H,
    int d, float inv_sqrt_d) {
  extern __shared__ __align__(16) uint8_t raw[];
  constexpr int R = 16 * RM, kLd = R + 4;
  double* sa = reinterpret_cast<double*>(raw);
  double* sb = sa + kSlice * R;
  float* xt = reinterpret_cast<float*>(sb);
  float* wt = reinterpret_cast<float*>(raw + SliceBytes(RM));   // [64 queries][R keys]
  __shared__ int first[kTile];                                   // the first key each query reaches
  const TileAt tile = KeyTile(BH);
  const int j0 = tile.tile * R;
  const size_t bh = tile.bh, b = bh / H, h = bh % H, D = static_cast<size_t>(H) * d;
  const size_t base = b * S * D + h * d, at = base + static_cast<size_t>(j0) * D;
  const int c0 = blockIdx.y * kTile, ty = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
  const int nkeys = min(R, S - j0);
  float acc[RM][4] = {};
  for (int i0 = j0 / kTile * kTile; i0 < S; i0 += kTile) {
    const int rows = min(kTile, S - i0);
    const size_t iat = base + static_cast<size_t>(i0) * D;
    double sc[RM][4], dp[RM][4];
    DotTile<RM, kVec>(k + at, nkeys, q + iat, rows, D, d, sa, sb, sc);
    if (kWantDK) DotTile<RM, kVec>(v + at, nkeys, dout + iat, rows, D, d, sa, sb, dp);
    __syncthreads();
    LoadTileF<kVec>(xt, (kWantDK ? q : dout) + iat, D, rows, c0, d);
    bool late = false;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i0 + Col(e);
      const float* st = stats + (bh * S + min(i, S - 1)) * kAttnStatsWidth;
      const int start = static_cast<int>(StatsStart(st[3], static_cast<size_t>(i)));
      late = late || (i < S && start > j0);
      if (ty == 0) first[Col(e)] = start;
#pragma unroll
      for (int r = 0; r < RM; ++r) {
        const int j = j0 + ty * RM + r;
        float g = 0.0f;
        if (i < S && j <= i && j >= start) {
          const float p = expf(static_cast<float>(sc[r][e]) * inv_sqrt_d - st[0]) * st[1];
          if (kWantDK) {
            const float dsv = p * (static_cast<float>(dp[r][e]) - st[2]);
            g = dsv * inv_sqrt_d;
          } else {
            g = p;
          }
        }
        wt[Col(e) * kLd + ty * RM + r] = g;
      }
    }
    const bool segments = __syncthreads_or(late);
    int lo[RM];
#pragma unroll
    for (int r = 0; r < RM; ++r) lo[r] = j0 + ty * RM + r - i0;
    if (i0 >= j0 + R - 1 && !segments) ColProduct<RM, true>(wt, kLd, xt, rows, lo, acc);
    else ColProduct<RM, false>(wt, kLd, xt, rows, lo, acc, first, j0 + ty * RM);
  }
#pragma unroll
  for (int r = 0; r < RM; ++r)
    if (ty * RM + r < nkeys) StoreRow4(out + at + static_cast<size_t>(ty * RM + r) * D, acc[r], c0 + c, d, kVec);
}

inline unsigned UnitBlocks(size_t units) {
  size_t b = (units + kWarps - 1) / kWarps;
  if (b < 1) b = 1;
  if (b > 148 * 16) b = 148 * 16;
  return static_cast<unsigned>(b);
}

template <typename Kernel>
inline bool AllowSmem(Kernel kernel, size_t bytes) {
  if (bytes <= 48 * 1024) return true;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(bytes)) == cudaSuccess;
}

}  // namespace

namespace {

constexpr size_t kMaxSmem = 227 * 1024;
constexpr size_t kTwoPerSm = 113 * 1024;

// 16 RM rows per block: four rows per thread (the most arithmetic per shared-memory read) while the grid still has
// four blocks per SM, else two while it has two, else one.
inline int RowsPerThread(size_t BH, size_t S, size_t chunks = 1) {
  for (int rm : {4, 2})
    if (BH * ((S + 16 * rm - 1) / (16 * rm)) * chunks >= (rm == 4 ? 4u : 2u) * 148u) return rm;
  return 1;
}
// The same for the kernels whose score rows (`arrays` f32 rows of S keys per query row) live in shared memory: no more
// rows than let two blocks share an SM, or one block of 16 rows; 0: not even that fits.
inline int RowsPerThreadWithScores(size_t BH, size_t S, int arrays) {
  auto bytes = [&](int rm) { return SliceBytes(rm) + static_cast<size_t>(arrays) * 16 * rm * RowStride(S) * sizeof(float); };
  for (int rm = RowsPerThread(BH, S); rm >= 1; rm /= 2)
    if (bytes(rm) <= kTwoPerSm) return rm;
  return bytes(1) <= kMaxSmem ? 1 : 0;
}
inline bool Vec(size_t d, std::initializer_list<const void*> ps) {
  if (d % 4 != 0) return false;
  for (const void* p : ps)
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;
  return true;
}
template <int RM>
using RowsTag = std::integral_constant<int, RM>;
// f(rows tag, vector tag) with the constants of this launch.
template <typename F>
inline void WithTile(int rm, bool vec, F f) {
  auto with_rows = [&](auto v) {
    if (rm == 4) f(RowsTag<4>{}, v);
    else if (rm == 2) f(RowsTag<2>{}, v);
    else f(RowsTag<1>{}, v);
  };
  if (vec) with_rows(std::true_type{});
  else with_rows(std::false_type{});
}
inline dim3 TileGrid(size_t BH, size_t tiles, size_t d) {
  return dim3(static_cast<unsigned>(BH * tiles), static_cast<unsigned>((d + kTile - 1) / kTile));
}

}  // namespace

// The dot-product identity a.b = b.a holds bit for bit here (each product is
// exact in double and the order over c is the same), so the tiled backward may
// take the key rows as the first operand and stream the query rows.

void AttnFwd(const float* q, const float* k, const float* v, float* o, float* probs,
             float* stats, size_t B, size_t S, size_t H, size_t d, const int32_t* starts,
             cudaStream_t s) {
  const size_t units = B * H * S;
  if (units == 0) return;
  const float inv_sqrt_d = 1.0f / sqrtf(static_cast<float>(d));
  if (const int rm = RowsPerThreadWithScores(B * H, S, 1); rm > 0) {
    WithTile(rm, Vec(d, {q, k, v, o}), [&](auto rows, auto vec) {
      constexpr int RM = decltype(rows)::value;
      const size_t bytes = SliceBytes(RM) + 16 * RM * RowStride(S) * sizeof(float);
      AllowSmem(AttnFwdTileKernel<RM, decltype(vec)::value>, bytes);
      AttnFwdTileKernel<RM, decltype(vec)::value><<<static_cast<unsigned>(B * H * ((S + 16 * RM - 1) / (16 * RM))), kTileThreads, bytes, s>>>(
          q, k, v, o, probs, stats, static_cast<int>(B * H), static_cast<int>(S), static_cast<int>(H), static_cast<int>(d),
          starts, inv_sqrt_d);
    });
    return;
  }
  const size_t bytes = kWarps * (d + S) * sizeof(float);
  AllowSmem(AttnFwdKernel, bytes);
  AttnFwdKernel<<<UnitBlocks(units), kWarps * 32, bytes, s>>>(q, k, v, o, probs, stats, B, S, H, d,
                                                             starts, inv_sqrt_d);
}

void AttnDP(const float* dout, const float* v, float* dp, size_t B, size_t S, size_t H, size_t d,
            cudaStream_t s) {
  if (B * H * S == 0) return;
  const size_t tiles = (S + kTile - 1) / kTile;
  const unsigned blocks = static_cast<unsigned>(B * H * tiles * tiles);
  const int BH = static_cast<int>(B * H);
  auto launch = [&](auto kernel) {
    kernel<<<blocks, kTileThreads, SliceBytes(4), s>>>(dout, v, dp, BH, static_cast<int>(S), static_cast<int>(H),
                                                       static_cast<int>(d));
  };
  if (Vec(d, {dout, v})) launch(AttnDPTileKernel<true>);
  else launch(AttnDPTileKernel<false>);
}

namespace {

template <bool kScaled>
void ColSum(const float* w, const float* x, float* out, size_t B, size_t S, size_t H, size_t d, float scale,
            cudaStream_t s) {
  if (B * H * S == 0) return;
  WithTile(RowsPerThread(B * H, S, (d + kTile - 1) / kTile), Vec(d, {x, out}), [&](auto rows, auto vec) {
    constexpr int RM = decltype(rows)::value;
    AttnColTileKernel<RM, kScaled, decltype(vec)::value>
        <<<TileGrid(B * H, (S + 16 * RM - 1) / (16 * RM), d), kTileThreads, 0, s>>>(
            w, x, out, static_cast<int>(B * H), static_cast<int>(S), static_cast<int>(H), static_cast<int>(d), scale);
  });
}

}  // namespace

void AttnDV(const float* probs, const float* dout, float* dv, size_t B, size_t S, size_t H,
            size_t d, cudaStream_t s) {
  ColSum<false>(probs, dout, dv, B, S, H, d, 1.0f, s);
}

void AttnDK(const float* ds, const float* q, float* dk, size_t B, size_t S, size_t H, size_t d,
            cudaStream_t s) {
  ColSum<true>(ds, q, dk, B, S, H, d, 1.0f / sqrtf(static_cast<float>(d)), s);
}

void AttnDQ(const float* ds, const float* k, float* dq, size_t B, size_t S, size_t H, size_t d,
            cudaStream_t s) {
  if (B * H * S == 0) return;
  const float inv_sqrt_d = 1.0f / sqrtf(static_cast<float>(d));
  WithTile(RowsPerThread(B * H, S, (d + kTile - 1) / kTile), Vec(d, {k, dq}), [&](auto rows, auto vec) {
    constexpr int RM = decltype(rows)::value;
    AttnRowTileKernel<RM, decltype(vec)::value>
        <<<TileGrid(B * H, (S + 16 * RM - 1) / (16 * RM), d), kTileThreads, 0, s>>>(
            ds, k, dq, static_cast<int>(B * H), static_cast<int>(S), static_cast<int>(H), static_cast<int>(d), inv_sqrt_d);
  });
}

void SoftmaxRowsBwd(const float* probs, const float* dp, float* ds, size_t rows, size_t cols,
                    cudaStream_t s) {
  if (rows == 0) return;
  SoftmaxRowsBwdKernel<<<UnitBlocks(rows), kWarps * 32, 0, s>>>(probs, dp, ds, rows, cols);
}

void AttnDQTiled(const float* q, const float* k, const float* v, const float* dout, float* stats,
                 float* dq, size_t B, size_t S, size_t H, size_t d, cudaStream_t s) {
  const size_t units = B * H * S;
  if (units == 0) return;
  const float inv_sqrt_d = 1.0f / sqrtf(static_cast<float>(d));
  if (const int rm = RowsPerThreadWithScores(B * H, S, 2); rm > 0) {
    WithTile(rm, Vec(d, {q, k, v, dout, dq}), [&](auto rows, auto vec) {
      constexpr int RM = decltype(rows)::value;
      const size_t bytes = SliceBytes(RM) + 2 * 16 * RM * RowStride(S) * sizeof(float);
      AllowSmem(AttnDQTiledTileKernel<RM, decltype(vec)::value>, bytes);
      AttnDQTiledTileKernel<RM, decltype(vec)::value>
          <<<static_cast<unsigned>(B * H * ((S + 16 * RM - 1) / (16 * RM))), kTileThreads, bytes, s>>>(
              q, k, v, dout, stats, dq, static_cast<int>(B * H), static_cast<int>(S), static_cast<int>(H),
              static_cast<int>(d), inv_sqrt_d);
    });
    return;
  }
  const size_t bytes = kWarps * (2 * d + 2 * S) * sizeof(float);
  AllowSmem(AttnDQTiledKernel, bytes);
  AttnDQTiledKernel<<<UnitBlocks(units), kWarps * 32, bytes, s>>>(q, k, v, dout, stats, dq, B, S, H,
                                                                 d, inv_sqrt_d);
}

void AttnDKVTiled(bool want_dk, const float* q, const float* k, const float* v, const float* dout,
                  const float* stats, float* out, size_t B, size_t S, size_t H, size_t d,
                  cudaStream_t s) {
  if (B * H * S == 0) return;
  const float inv_sqrt_d = 1.0f / sqrtf(static_cast<float>(d));
  WithTile(RowsPerThread(B * H, S, (d + kTile - 1) / kTile), Vec(d, {q, k, v, dout, out}), [&](auto rows, auto vec) {
    constexpr int RM = decltype(rows)::value;
    const size_t bytes = SliceBytes(RM) + kTile * (16 * RM + 4) * sizeof(float);
    auto launch = [&](auto kernel) {
      AllowSmem(kernel, bytes);
      kernel<<<TileGrid(B * H, (S + 16 * RM - 1) / (16 * RM), d), kTileThreads, bytes, s>>>(
          q, k, v, dout, stats, out, static_cast<int>(B * H), static_cast<int>(S), static_cast<int>(H),
          static_cast<int>(d), inv_sqrt_d);
    };
    if (want_dk) launch(AttnDKVTiledTileKernel<RM, true, decltype(vec)::value>);
    else launch(AttnDKVTiledTileKernel<RM, false, decltype(vec)::value>);
  });
}

}  // namespace see::k
