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
// (Where the bits are not observed the tile kernels take their double dots on the FP64 tensor instruction and contract
// the output sums: DotTile and MulAdd.)
//
// The tile kernels (AttnFwdTile, AttnDPTile, AttnRowTile, AttnColTile,
// AttnDQTiledTile, AttnDKVTiledTile) are bound by FP64 and shared memory: a block owns 8, 16 or 32
// query (or key) rows of one (sequence, head) and takes the other axis 64 at a
// time.  Both operands of a score tile are widened to double once, on their way
// into shared memory (a conversion costs four FMA slots, so per use it would be
// the bound): the block's own rows for good, the streamed ones 8 features at a
// time with the next 8 already in registers; a thread accumulates RM x 4 pairs:
// RM + 4 shared doubles per 4 RM fused multiply-adds, each accumulator one chain
// over ascending features.  The f32 output sums are the same shape of product,
// 64 columns of the head at a time, RM x 4 outputs per thread, each one chain over
// ascending keys, the keys' rows arriving by asynchronous copies.
// One warp per row with a strided K row per lane (the row kernels below) took
// 3747 us for 8 x 512 positions of 12 heads of 64 features and 320 us for
// 32 x 128 of 4 heads.
//
// The row kernels (one warp owns one row and keeps its whole score row in shared
// memory) remain for rows too long for a tile block's score rows.
#include <initializer_list>
#include <type_traits>

#include "kernels.h"
#include "launch.cuh"

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
  AwaitPrevious();
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
  AwaitPrevious();
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
  AwaitPrevious();
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
// A block of eight warps owns R = 8 RM rows of one axis (its "own" rows) and streams the other axis 64 rows at a time: two
// groups of four warps take alternate tiles, each with slice buffers and barriers of its own (the score rows leave room
// for two blocks per SM; one group per block, eight warps on an SM, issued 1.9 instructions per cycle).

constexpr int kTile = 64;      // rows of the streamed axis per step
constexpr int kSlice = 8;      // features of a streamed tile in shared memory at a time
constexpr int kTileThreads = 256;
constexpr int kGroup = 128;            // threads of a group
constexpr int kStreamLd = kTile + 2;   // doubles per feature of a streamed slice (a multiple of 16 bytes; 2-way store conflicts)
// Where row r of feature c lies in a streamed slice, and among the block's own rows.  kMma: the tensor instruction's
// fragments are four features of the same rows at once, so these turn the rows into four different quarters of the banks.
// (Padding did that too, at an eighth to a half more shared memory, and fewer rows fitted a block: forward of 8 x 480
// positions of 12 heads of 128 406 us, 284 turned; dQ of 8 x 448 of those 903 and 556, of 8 x 600 of 12 heads of 64 798 and 500;
// 8 x 512 of 12 heads of 64 185 and 184.)
template <bool kMma>
__device__ __forceinline__ int StreamAt(int c, int r) {
  return kMma ? c * kTile + (r ^ ((c & 3) << 2) ^ ((c & 4) << 1)) : c * kStreamLd + r;
}
template <bool kMma, int kRows>
__device__ __forceinline__ int OwnAt(int c, int r) {
  return c * kRows + (kMma ? r ^ (kRows == 8 ? (c & 2) << 1 : (c & 3) << 2) : r);
}
constexpr int kChunkRows = 32;         // rows of an f32 tile in shared memory at a time

__host__ __device__ constexpr int PaddedFeatures(int d) { return (d + kSlice - 1) / kSlice * kSlice; }

__device__ __forceinline__ float4 LoadFour(const float* __restrict__ p, int left, bool vec) {   // left: elements there are
  if (left <= 0) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (vec) return *reinterpret_cast<const float4*>(p);
  return make_float4(p[0], left > 1 ? p[1] : 0.0f, left > 2 ? p[2] : 0.0f, left > 3 ? p[3] : 0.0f);
}

// The block's own rows, widened to double once: dst[feature][kRows], zero outside (0 * 0 leaves a chain as it is).
template <int kRows, bool kVec, bool kMma>
__device__ __forceinline__ void LoadOwn(double* dst, const float* __restrict__ src, size_t stride, int rows, int d) {
  const int quads = PaddedFeatures(d) / 4;
  for (int t = threadIdx.x; t < kRows * quads; t += kTileThreads) {
    const int r = t / quads, c = t % quads * 4;
    const float4 f = LoadFour(src + static_cast<size_t>(min(r, rows - 1)) * stride + c, r < rows ? d - c : 0, kVec);
    dst[OwnAt<kMma, kRows>(c, r)] = f.x;
    dst[OwnAt<kMma, kRows>(c + 1, r)] = f.y;
    dst[OwnAt<kMma, kRows>(c + 2, r)] = f.z;
    dst[OwnAt<kMma, kRows>(c + 3, r)] = f.w;
  }
}

__device__ __forceinline__ int GroupOf() { return static_cast<int>(threadIdx.x) / kGroup; }
__device__ __forceinline__ int InGroup() { return static_cast<int>(threadIdx.x) % kGroup; }
__device__ __forceinline__ void GroupSync() {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + GroupOf()), "n"(kGroup) : "memory");
}
// A multiply-add of an output sum: two roundings as the CPU executor makes them, or one where the bits are not observed.
template <bool kFused>
__device__ __forceinline__ float MulAdd(float a, float b, float c) {
  return kFused ? fmaf(a, b, c) : c + a * b;
}

// A streamed tile's slice on its way: a row's four features per thread of the group.
struct SliceRegs { float4 v; };
template <bool kVec>
__device__ __forceinline__ void FetchSlice(SliceRegs* s, const float* __restrict__ src, size_t stride, int rows, int c0,
                                           int d) {
  const int r = InGroup() >> 1, c = c0 + (InGroup() & 1) * 4;
  s->v = LoadFour(src + static_cast<size_t>(min(r, rows - 1)) * stride + c, r < rows ? d - c : 0, kVec);
}
template <bool kMma>
__device__ __forceinline__ void StoreSlice(double* dst, const SliceRegs& s) {
  const int r = InGroup() >> 1, c = (InGroup() & 1) * 4;
  dst[StreamAt<kMma>(c, r)] = s.v.x;
  dst[StreamAt<kMma>(c + 1, r)] = s.v.y;
  dst[StreamAt<kMma>(c + 2, r)] = s.v.z;
  dst[StreamAt<kMma>(c + 3, r)] = s.v.w;
}

// Which pair (row of the block's own, row of the streamed tile) a thread's accumulator acc[r][e] stands for; e and e + 1
// (e even) are neighbours.  kMma: the fragments of the tensor instruction, a warp to 16 streamed rows; else the thread
// grid of 8 x 16 (16 lanes read 256 contiguous bytes).
template <bool kMma, int RM>
__device__ __forceinline__ int RowAt(int r) {
  return kMma ? r * 8 + static_cast<int>(threadIdx.x & 31) / 4 : (InGroup() >> 4) * RM + r;
}
template <bool kMma>
__device__ __forceinline__ int Col(int e) {
  return kMma ? (InGroup() >> 5) * 16 + (e >> 1) * 8 + 2 * static_cast<int>(threadIdx.x & 3) + (e & 1)
              : 2 * static_cast<int>(threadIdx.x & 15) + (e & 1) + (e >> 1) * 32;
}

// c += a b in double: 16 x 8 += 16 x 8 . 8 x 8 (8 x 8 += 8 x 4 . 4 x 8).
__device__ __forceinline__ void DMma16(double (&c0)[4], double (&c1)[4], int e, const double (&a)[4], const double (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+d"(c0[e]), "+d"(c0[e + 1]), "+d"(c1[e]), "+d"(c1[e + 1])
               : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}
__device__ __forceinline__ void DMma8(double (&c)[4], int e, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[e]), "+d"(c[e + 1]) : "d"(a), "d"(b));
}

// acc[r][e] = own row RowAt(r) . streamed row Col(e), in double.  `regs` holds the tile's first
// slice on entry and the first slice of `next` (rows of the same stride; null: nothing) on exit, so that a global load is
// always a whole slice of arithmetic ahead of its use.  `turn` alternates the two slice buffers: one barrier per slice.
// kMma false: every accumulator one chain over ascending features, the CPU's.  kMma true (where the bits are not
// observed): the FP64 tensor instruction, whose sums of eight are doubles all the same.  Both run at the FP64 pipe's
// rate at best; a thread grid of RM x 4 pairs reads RM + 4 doubles of shared memory for 4 RM multiply-adds, the fragments
// 2 RM + 4 a lane for 64 RM a lane of a slice.  Measured, thread grid / tensor instruction: forward of 8 x 512 positions
// of 12 heads of 64 226 / 176 us (shared memory 68 % busy, the FP64 pipe 29), of 32 x 128 of 4 heads 37.3 / 30.5, dP of those
// 21.4 / 16.6.
template <int RM, bool kVec, bool kMma>
__device__ __forceinline__ void DotTile(const double* own, const float* b, int rows, const float* next, int next_rows,
                                        size_t stride, int d, double* slices, int* turn, SliceRegs* regs,
                                        double (&acc)[RM][4]) {
  constexpr int R = 8 * RM;
  const int tx = threadIdx.x & 15, ty = InGroup() >> 4;
#pragma unroll
  for (int r = 0; r < RM; ++r)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[r][e] = 0.0;
  // kMma: this lane's fragments in a slice and among the own rows, the even and the odd eights of rows; four features on,
  // own rows lie as they did and a slice's eights have changed places.
  [[maybe_unused]] const int g = static_cast<int>(threadIdx.x & 31) / 4, t = threadIdx.x & 3, w = (InGroup() >> 5) * 16 + g;
  [[maybe_unused]] const int f0 = StreamAt<true>(t, w), f1 = StreamAt<true>(t, w + 8);
  [[maybe_unused]] const int e0 = OwnAt<true, R>(t, g), e1 = OwnAt<true, R>(t, g + 8);
  for (int c0 = 0; c0 < d; c0 += kSlice) {
    double* sb = slices + *turn * (kSlice * kStreamLd);
    *turn ^= 1;
    StoreSlice<kMma>(sb, *regs);
    GroupSync();
    if (c0 + kSlice < d) FetchSlice<kVec>(regs, b, stride, rows, c0 + kSlice, d);
    else if (next) FetchSlice<kVec>(regs, next, stride, next_rows, 0, d);
    if constexpr (kMma) {
      const double* sa = own + c0 * R;
      double y[2][2];
      y[0][0] = sb[f0];
      y[1][0] = sb[f1];
      y[0][1] = sb[f1 + 4 * kTile];
      y[1][1] = sb[f0 + 4 * kTile];
      if constexpr (RM == 1) {
        const double x0 = sa[e0], x1 = sa[e0 + 4 * R];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          DMma8(acc[0], 2 * n, x0, y[n][0]);
          DMma8(acc[0], 2 * n, x1, y[n][1]);
        }
      } else {
#pragma unroll
        for (int m = 0; m + 1 < RM; m += 2) {
          const double x[4] = {sa[e0 + 8 * m], sa[e1 + 8 * m], sa[e0 + 4 * R + 8 * m], sa[e1 + 4 * R + 8 * m]};
#pragma unroll
          for (int n = 0; n < 2; ++n) DMma16(acc[m], acc[m + 1], 2 * n, x, y[n]);
        }
      }
    } else {
      const double* sa = own + c0 * R + ty * RM;
#pragma unroll
      for (int c = 0; c < kSlice; ++c) {
        const double2 y0 = *reinterpret_cast<const double2*>(sb + c * kStreamLd + 2 * tx);
        const double2 y1 = *reinterpret_cast<const double2*>(sb + c * kStreamLd + 32 + 2 * tx);
        const double y[4] = {y0.x, y0.y, y1.x, y1.y};
        double x[RM];
#pragma unroll
        for (int r = 0; r < RM; ++r) x[r] = sa[c * R + r];
#pragma unroll
        for (int r = 0; r < RM; ++r)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[r][e] = fma(x[r], y[e], acc[r][e]);
      }
    }
  }
}

__host__ __device__ constexpr size_t GroupBytes() { return 2 * sizeof(double) * kSlice * kStreamLd; }
__host__ __device__ constexpr size_t StreamBytes() { return 2 * GroupBytes(); }
__host__ __device__ constexpr size_t OwnBytes(int RM, int d) { return sizeof(double) * PaddedFeatures(d) * 8 * RM; }

// Rows [0, rows) x columns [c0, c0 + 64) of a [., stride] f32 matrix into dst[32][64] by asynchronous copies (zero
// outside); one commit group.
template <bool kVec>
__device__ __forceinline__ void CopyChunk(float* dst, const float* __restrict__ src, size_t stride, int rows, int c0,
                                          int d) {
  for (int t = threadIdx.x; t < kChunkRows * 16; t += kTileThreads) {
    const int r = t >> 4, c = (t & 15) * 4;
    const int left = r < rows ? d - (c0 + c) : 0;
    const float* p = src + static_cast<size_t>(r < rows ? r : 0) * stride + (left > 0 ? c0 + c : 0);
    const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(dst + r * kTile + c));
    if (kVec) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(p), "r"(left > 0 ? 16 : 0) : "memory");
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
                     ::"r"(to + 4 * e), "l"(left > e ? p + e : src), "r"(left > e ? 4 : 0) : "memory");
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
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

// acc[r][e] += w[row][j] * x[j][c + e] for j = 0 .. 31 in order; row's weights at w + r * ld.  A row takes
// j in [lo[r], hi[r]) only (a weight outside is not multiplied: x may hold anything there); kAll: every j.
template <bool kFused, int RM, bool kAll>
__device__ __forceinline__ void RowProduct(const float* w, int ld, const float* x, const int (&lo)[RM],
                                           const int (&hi)[RM], float (&acc)[RM][4]) {
  const int c = (threadIdx.x & 15) * 4;
#pragma unroll 2
  for (int j = 0; j < kChunkRows; j += 4) {
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
          for (int e = 0; e < 4; ++e) acc[r][e] = MulAdd<kFused>(p[r][jj], xv[e], acc[r][e]);
        }
      }
    }
  }
}

// Row sums over a whole score row: acc = sum over keys [0, nkeys) of w[row][key] * x[key][c0 ..], keys ascending, 32
// keys at a time through the two chunk buffers at `xt`.  Ends with a barrier.
template <bool kFused, int RM, bool kVec>
__device__ __forceinline__ void RowSum(const float* w, int ld, const float* __restrict__ x, size_t stride, int nkeys, int S,
                                       int c0, int d, const int (&row_lo)[RM], const int (&row_hi)[RM], int all_below,
                                       float* xt, float (&acc)[RM][4]) {
  int buf = 0;
  CopyChunk<kVec>(xt, x, stride, min(kChunkRows, S), c0, d);
  for (int k0 = 0; k0 < nkeys; k0 += kChunkRows, buf ^= 1) {
    if (k0 + kChunkRows < nkeys) {
      CopyChunk<kVec>(xt + (buf ^ 1) * (kChunkRows * kTile), x + static_cast<size_t>(k0 + kChunkRows) * stride, stride,
                      min(kChunkRows, S - k0 - kChunkRows), c0, d);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    int lo[RM], hi[RM];
#pragma unroll
    for (int r = 0; r < RM; ++r) { lo[r] = row_lo[r] - k0; hi[r] = row_hi[r] - k0; }
    const float* xs = xt + buf * (kChunkRows * kTile);
    if (k0 + kChunkRows <= all_below) RowProduct<kFused, RM, true>(w + k0, ld, xs, lo, hi, acc);
    else RowProduct<kFused, RM, false>(w + k0, ld, xs, lo, hi, acc);
    __syncthreads();   // the buffer is refilled two chunks on
  }
}

// In the output sums all 256 threads share the block's rows: OutRows(RM) each, 16 groups of 16 column quads.
__host__ __device__ constexpr int OutRows(int RM) { return RM > 1 ? RM / 2 : 1; }

// Score rows are stored with a stride of a whole number of tiles plus 4 floats (a multiple of 16 bytes that
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

// Forward.  Block: 8 RM query rows of one (sequence, head).  Score rows of the whole block stay in shared memory
// between the three phases.
template <int RM, bool kFused, bool kVec>
__global__ __launch_bounds__(kTileThreads) void AttnFwdTileKernel(
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v, float* __restrict__ o,
    float* __restrict__ probs, float* __restrict__ stats, int BH, int S, int H, int d,
    const int32_t* __restrict__ starts, float inv_sqrt_d) {
  AwaitPrevious();
  extern __shared__ __align__(16) uint8_t raw[];
  constexpr int R = 8 * RM;
  double* slices = reinterpret_cast<double*>(raw + GroupOf() * GroupBytes());
  float* xt = reinterpret_cast<float*>(raw);                       // the V chunks, where the K slices were
  double* own = reinterpret_cast<double*>(raw + StreamBytes());
  float* rows = reinterpret_cast<float*>(raw + StreamBytes() + OwnBytes(RM, d));
  const int ld = static_cast<int>(RowStride(S));
  const TileAt tile = QueryTile((S + R - 1) / R, BH);
  const int i0 = tile.tile * R;
  const size_t bh = tile.bh, b = bh / H, h = bh % H, D = static_cast<size_t>(H) * d;
  const int nrows = min(R, S - i0), nkeys = min(i0 + R, S);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t base = b * S * D + h * d;
  auto first_key = [&](int i) {
    if (!starts) return 0;
    const int32_t s0 = starts[b * S + i];
    return s0 <= 0 ? 0 : (s0 < i ? static_cast<int>(s0) : i);
  };
  SliceRegs regs;
  int turn = 0;
  const int first = GroupOf() * kTile;
  if (first < nkeys) FetchSlice<kVec>(&regs, k + base + static_cast<size_t>(first) * D, D, min(kTile, S - first), 0, d);
  LoadOwn<R, kVec, kFused>(own, q + base + static_cast<size_t>(i0) * D, D, nrows, d);
  __syncthreads();
  for (int k0 = first; k0 < nkeys; k0 += 2 * kTile) {
    double acc[RM][4];
    const float* kb = k + base + static_cast<size_t>(k0) * D;
    DotTile<RM, kVec, kFused>(own, kb, min(kTile, S - k0), k0 + 2 * kTile < nkeys ? kb + 2 * kTile * D : nullptr,
                              min(kTile, S - k0 - 2 * kTile), D, d, slices, &turn, &regs, acc);
#pragma unroll
    for (int r = 0; r < RM; ++r)
#pragma unroll
      for (int e = 0; e < 4; e += 2)
        *reinterpret_cast<float2*>(rows + RowAt<kFused, RM>(r) * ld + k0 + Col<kFused>(e)) =
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
  __syncthreads();
  constexpr int OR = OutRows(RM);
  const int r0 = (threadIdx.x >> 4) * OR;   // this thread's rows of the output sums
  int row_lo[OR], row_hi[OR];
#pragma unroll
  for (int r = 0; r < OR; ++r) {
    const int i = min(i0 + r0 + r, S - 1);
    row_lo[r] = first_key(i);
    row_hi[r] = i + 1;
  }
  for (int c0 = 0; c0 < d; c0 += kTile) {
    float acc[OR][4] = {};
    RowSum<kFused, OR, kVec>(rows + min(r0, R - OR) * ld, ld, v + base, D, nkeys, S, c0, d, row_lo, row_hi,
                             starts ? 0 : i0 + 1, xt, acc);
#pragma unroll
    for (int r = 0; r < OR; ++r)
      if (r0 + r < nrows)
        StoreRow4(o + base + static_cast<size_t>(i0 + r0 + r) * D, acc[r], c0 + (threadIdx.x & 15) * 4, d, kVec);
  }
}

// dP for a head too wide for a tile block's own rows: a thread per pair.
__global__ void AttnDPWideKernel(const float* __restrict__ dout, const float* __restrict__ v, float* __restrict__ dp,
                                 size_t BH, size_t S, size_t H, size_t d) {
  AwaitPrevious();
  const size_t pairs = BH * S * S, D = H * d;
  for (size_t t = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; t < pairs;
       t += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t j = t % S, i = t / S % S, bh = t / (S * S), at = bh / H * S * D + bh % H * d;
    dp[t] = j <= i ? static_cast<float>(DotD(dout + at + i * D, v + at + j * D, d)) : 0.0f;
  }
}

// dP[i][j] = dO_i . v_j for j <= i, zero above the diagonal.  Block: 8 RM query rows, every key tile.
template <int RM, bool kMma, bool kVec>
__global__ __launch_bounds__(kTileThreads) void AttnDPTileKernel(const float* __restrict__ dout,
                                                                 const float* __restrict__ v, float* __restrict__ dp,
                                                                 int BH, int S, int H, int d) {
  AwaitPrevious();
  extern __shared__ __align__(16) uint8_t raw[];
  constexpr int R = 8 * RM;
  double* slices = reinterpret_cast<double*>(raw + GroupOf() * GroupBytes());
  double* own = reinterpret_cast<double*>(raw + StreamBytes());
  const TileAt tile = QueryTile((S + R - 1) / R, BH);
  const int i0 = tile.tile * R, nkeys = min(i0 + R, S);
  const size_t bh = tile.bh, b = bh / H, h = bh % H, D = static_cast<size_t>(H) * d;
  const size_t base = b * S * D + h * d;
  const bool pairs = (S & 1) == 0 && (reinterpret_cast<uintptr_t>(dp) & 7) == 0;   // (j is even: 8-byte stores)
  SliceRegs regs;
  int turn = 0;
  const int first = GroupOf() * kTile;
  if (first < nkeys) FetchSlice<kVec>(&regs, v + base + static_cast<size_t>(first) * D, D, min(kTile, S - first), 0, d);
  LoadOwn<R, kVec, kMma>(own, dout + base + static_cast<size_t>(i0) * D, D, min(R, S - i0), d);
  __syncthreads();
  for (int k0 = first; k0 < S; k0 += 2 * kTile) {
    double acc[RM][4] = {};
    if (k0 < nkeys) {
      const float* vb = v + base + static_cast<size_t>(k0) * D;
      DotTile<RM, kVec, kMma>(own, vb, min(kTile, S - k0), k0 + 2 * kTile < nkeys ? vb + 2 * kTile * D : nullptr,
                              min(kTile, S - k0 - 2 * kTile), D, d, slices, &turn, &regs, acc);
    }
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const int i = i0 + RowAt<kMma, RM>(r);
      if (i >= S) continue;
      float* row = dp + (bh * S + i) * S;
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const int j = k0 + Col<kMma>(e);
        const float x0 = j <= i ? static_cast<float>(acc[r][e]) : 0.0f;
        const float x1 = j + 1 <= i ? static_cast<float>(acc[r][e + 1]) : 0.0f;
        if (pairs && j + 1 < S) {
          *reinterpret_cast<float2*>(row + j) = make_float2(x0, x1);
        } else {
          if (j < S) row[j] = x0;
          if (j + 1 < S) row[j + 1] = x1;
        }
      }
    }
  }
}

// dQ_i[c] = sum over j <= i of (dS[i][j] / sqrt(d)) k_j[c].  Block: 16 RM rows, 64 columns of the head.
template <int RM, bool kFused, bool kVec>
__global__ __launch_bounds__(kTileThreads) void AttnRowTileKernel(const float* __restrict__ ds,
                                                                  const float* __restrict__ k, float* __restrict__ dq,
                                                                  int BH, int S, int H, int d, float inv_sqrt_d) {
  AwaitPrevious();
  constexpr int R = 16 * RM, kLd = kChunkRows + 4;
  __shared__ __align__(16) float xt[2 * kChunkRows * kTile];
  __shared__ __align__(16) float wt[2 * R * kLd];
  const TileAt tile = QueryTile((S + R - 1) / R, BH);
  const int i0 = tile.tile * R;
  const size_t bh = tile.bh, b = bh / H, h = bh % H, D = static_cast<size_t>(H) * d;
  const size_t base = b * S * D + h * d;
  const int c0 = blockIdx.y * kTile, ty = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
  const int nkeys = min(i0 + R, S);
  constexpr int kPer = R * kChunkRows / kTileThreads;   // weights a thread carries for the next chunk
  float w[kPer];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int idx = static_cast<int>(threadIdx.x) + t * kTileThreads, r = idx / kChunkRows, j = idx % kChunkRows;
      w[t] = i0 + r < S && k0 + j < S ? ds[(bh * S + i0 + r) * S + k0 + j] : 0.0f;
    }
  };
  float acc[RM][4] = {};
  fetch(0);
  CopyChunk<kVec>(xt, k + base, D, min(kChunkRows, S), c0, d);
  int buf = 0;
  for (int k0 = 0; k0 < nkeys; k0 += kChunkRows, buf ^= 1) {
    float* ws = wt + buf * (R * kLd);
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int idx = static_cast<int>(threadIdx.x) + t * kTileThreads;
      ws[idx / kChunkRows * kLd + idx % kChunkRows] = w[t] * inv_sqrt_d;
    }
    if (k0 + kChunkRows < nkeys) {
      fetch(k0 + kChunkRows);
      CopyChunk<kVec>(xt + (buf ^ 1) * (kChunkRows * kTile), k + base + static_cast<size_t>(k0 + kChunkRows) * D, D,
                      min(kChunkRows, S - k0 - kChunkRows), c0, d);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    int lo[RM], hi[RM];
#pragma unroll
    for (int r = 0; r < RM; ++r) { lo[r] = 0; hi[r] = i0 + ty * RM + r + 1 - k0; }
    const float* xs = xt + buf * (kChunkRows * kTile);
    if (k0 + kChunkRows <= i0 + 1) RowProduct<kFused, RM, true>(ws + ty * RM * kLd, kLd, xs, lo, hi, acc);
    else RowProduct<kFused, RM, false>(ws + ty * RM * kLd, kLd, xs, lo, hi, acc);
    __syncthreads();   // xs is refilled two chunks on
  }
#pragma unroll
  for (int r = 0; r < RM; ++r)
    if (i0 + ty * RM + r < S) StoreRow4(dq + base + static_cast<size_t>(i0 + ty * RM + r) * D, acc[r], c0 + c, d, kVec);
}

// acc[r][e] += w[i][r] x[i][c + e] for i = 0 .. rows - 1 in order (w at this thread's first key), where query i reaches
// key r: i >= lo[r], and key + r >= start[i] when there are segment starts (kAll: every i reaches every key).
template <bool kFused, int RM, bool kAll>
__device__ __forceinline__ void ColProduct(const float* w, int ldw, const float* x, int rows, const int (&lo)[RM],
                                           float (&acc)[RM][4], const int* start = nullptr, int key = 0) {
  const int c = (threadIdx.x & 15) * 4;
#pragma unroll 4
  for (int i = 0; i < rows; ++i) {
    const float4 f = *reinterpret_cast<const float4*>(x + i * kTile + c);
    const float xv[4] = {f.x, f.y, f.z, f.w};
    const int first = kAll || !start ? 0 : start[i];
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const float g = w[i * ldw + r];
      if (kAll || (i >= lo[r] && key + r >= first)) {
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[r][e] = MulAdd<kFused>(g, xv[e], acc[r][e]);
      }
    }
  }
}

// out_j[c] = sum over i >= j of w[i][j] (scale) x_i[c], i ascending.  Block: 16 RM keys, 64 columns.
template <int RM, bool kFused, bool kScaled, bool kVec>
__global__ __launch_bounds__(kTileThreads) void AttnColTileKernel(const float* __restrict__ w,
                                                                  const float* __restrict__ x, float* __restrict__ out,
                                                                  int BH, int S, int H, int d, float inv_sqrt_d) {
  AwaitPrevious();
  constexpr int R = 16 * RM;
  __shared__ __align__(16) float xt[2 * kChunkRows * kTile];
  __shared__ __align__(16) float wt[2 * kChunkRows * R];
  const TileAt tile = KeyTile(BH);
  const int j0 = tile.tile * R;
  const size_t bh = tile.bh, b = bh / H, h = bh % H, D = static_cast<size_t>(H) * d;
  const size_t base = b * S * D + h * d;
  const int c0 = blockIdx.y * kTile, ty = threadIdx.x >> 4, c = (threadIdx.x & 15) * 4;
  constexpr int kPer = R * kChunkRows / kTileThreads;
  float g[kPer];
  auto fetch = [&](int i0) {
#pragma unroll
    for (int t = 0; t < kPer; ++t) {
      const int idx = static_cast<int>(threadIdx.x) + t * kTileThreads, i = idx / R, j = idx % R;
      g[t] = i0 + i < S && j0 + j < S ? w[(bh * S + i0 + i) * S + j0 + j] : 0.0f;
    }
  };
  float acc[RM][4] = {};
  fetch(j0);
  CopyChunk<kVec>(xt, x + base + static_cast<size_t>(j0) * D, D, min(kChunkRows, S - j0), c0, d);
  int buf = 0;
  for (int i0 = j0; i0 < S; i0 += kChunkRows, buf ^= 1) {
    float* ws = wt + buf * (kChunkRows * R);
#pragma unroll
    for (int t = 0; t < kPer; ++t) ws[threadIdx.x + t * kTileThreads] = kScaled ? g[t] * inv_sqrt_d : g[t];
    if (i0 + kChunkRows < S) {
      fetch(i0 + kChunkRows);
      CopyChunk<kVec>(xt + (buf ^ 1) * (kChunkRows * kTile), x + base + static_cast<size_t>(i0 + kChunkRows) * D, D,
                      min(kChunkRows, S - i0 - kChunkRows), c0, d);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    int lo[RM];
#pragma unroll
    for (int r = 0; r < RM; ++r) lo[r] = j0 + ty * RM + r - i0;
    const float* xs = xt + buf * (kChunkRows * kTile);
    const int rows = min(kChunkRows, S - i0);
    if (i0 >= j0 + R - 1) ColProduct<kFused, RM, true>(ws + ty * RM, R, xs, rows, lo, acc);
    else ColProduct<kFused, RM, false>(ws + ty * RM, R, xs, rows, lo, acc);
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < RM; ++r)
    if (j0 + ty * RM + r < S) StoreRow4(out + base + static_cast<size_t>(j0 + ty * RM + r) * D, acc[r], c0 + c, d, kVec);
}

// Tiled dQ: the rows' probabilities and dP recomputed into shared memory, delta written into the stats rows,
// then dQ (reference: runtime/executor/attention.cc:492-531).
template <int RM, bool kFused, bool kVec>
__global__ __launch_bounds__(kTileThreads) void AttnDQTiledTileKernel(
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
    const float* __restrict__ dout, float* __restrict__ stats, float* __restrict__ dq, int BH, int S, int H,
    int d, float inv_sqrt_d) {
  AwaitPrevious();
  extern __shared__ __align__(16) uint8_t raw[];
  constexpr int R = 8 * RM;
  double* slices = reinterpret_cast<double*>(raw + GroupOf() * GroupBytes());
  float* xt = reinterpret_cast<float*>(raw);
  double* own_q = reinterpret_cast<double*>(raw + StreamBytes());
  double* own_do = reinterpret_cast<double*>(raw + StreamBytes() + OwnBytes(RM, d));
  const int ld = static_cast<int>(RowStride(S));
  float* prows = reinterpret_cast<float*>(raw + StreamBytes() + 2 * OwnBytes(RM, d));
  float* dprows = prows + R * ld;
  const TileAt tile = QueryTile((S + R - 1) / R, BH);
  const int i0 = tile.tile * R;
  const size_t bh = tile.bh, b = bh / H, h = bh % H, D = static_cast<size_t>(H) * d;
  const int nrows = min(R, S - i0), nkeys = min(i0 + R, S);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t base = b * S * D + h * d, at = base + static_cast<size_t>(i0) * D;
  float* st = stats + (bh * S + i0) * kAttnStatsWidth;
  SliceRegs regs;
  int turn = 0;
  const int first = GroupOf() * kTile;
  if (first < nkeys) FetchSlice<kVec>(&regs, k + base + static_cast<size_t>(first) * D, D, min(kTile, S - first), 0, d);
  LoadOwn<R, kVec, kFused>(own_q, q + at, D, nrows, d);
  LoadOwn<R, kVec, kFused>(own_do, dout + at, D, nrows, d);
  __syncthreads();
  for (int k0 = first; k0 < nkeys; k0 += 2 * kTile) {
    const float *kb = k + base + static_cast<size_t>(k0) * D, *vb = v + base + static_cast<size_t>(k0) * D;
    const int rows = min(kTile, S - k0);
    double acc[RM][4];
    DotTile<RM, kVec, kFused>(own_q, kb, rows, vb, rows, D, d, slices, &turn, &regs, acc);
#pragma unroll
    for (int r = 0; r < RM; ++r) {
      const int row = min(RowAt<kFused, RM>(r), nrows - 1);
      const float m = st[row * kAttnStatsWidth], inv_denom = st[row * kAttnStatsWidth + 1];
#pragma unroll
      for (int e = 0; e < 4; ++e)
        prows[RowAt<kFused, RM>(r) * ld + k0 + Col<kFused>(e)] = expf(static_cast<float>(acc[r][e]) * inv_sqrt_d - m) * inv_denom;
    }
    DotTile<RM, kVec, kFused>(own_do, vb, rows, k0 + 2 * kTile < nkeys ? kb + 2 * kTile * D : nullptr, min(kTile, S - k0 - 2 * kTile), D, d,
                      slices, &turn, &regs, acc);
#pragma unroll
    for (int r = 0; r < RM; ++r)
#pragma unroll
      for (int e = 0; e < 4; ++e) dprows[RowAt<kFused, RM>(r) * ld + k0 + Col<kFused>(e)] = static_cast<float>(acc[r][e]);
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
  __syncthreads();
  constexpr int OR = OutRows(RM);
  const int r0 = (threadIdx.x >> 4) * OR;
  int row_lo[OR], row_hi[OR];
  bool whole = true;
#pragma unroll
  for (int r = 0; r < OR; ++r) {
    const int row = min(r0 + r, nrows - 1);
    row_lo[r] = static_cast<int>(StatsStart(st[row * kAttnStatsWidth + 3], i0 + row));
    row_hi[r] = i0 + row + 1;
    whole = whole && row_lo[r] == 0;
  }
  for (int c0 = 0; c0 < d; c0 += kTile) {
    float acc[OR][4] = {};
    RowSum<kFused, OR, kVec>(prows + min(r0, R - OR) * ld, ld, k + base, D, nkeys, S, c0, d, row_lo, row_hi,
                             whole ? i0 + 1 : 0, xt, acc);
#pragma unroll
    for (int r = 0; r < OR; ++r)
      if (r0 + r < nrows)
        StoreRow4(dq + at + static_cast<size_t>(r0 + r) * D, acc[r], c0 + (threadIdx.x & 15) * 4, d, kVec);
  }
}

// Tiled dK (kWantDK) or dV over the query rows i >= j of 8 RM keys, 64 columns of the head per block (a wider
// head repeats the scores; reference: runtime/executor/attention.cc:533-590).  The groups form the weights of two query
// tiles at a time, then all threads add both, the earlier tile first.
template <int RM, bool kWantDK, bool kFused, bool kVec>
__global__ __launch_bounds__(kTileThreads) void AttnDKVTiledTileKernel(
    const float* __restrict__ q, const float* __restrict__ k, const float* __restrict__ v,
    const float* __restrict__ dout, const float* __restrict__ stats, float* __restrict__ out, int BH, int S, int H,
    int d, float inv_sqrt_d) {
  AwaitPrevious();
  extern __shared__ __align__(16) uint8_t raw[];
  constexpr int R = 8 * RM, kLd = R + 4;
  const int group = GroupOf();
  double* slices = reinterpret_cast<double*>(raw + group * GroupBytes());
  double* own_k = reinterpret_cast<double*>(raw + StreamBytes());
  double* own_v = reinterpret_cast<double*>(raw + StreamBytes() + OwnBytes(RM, d));
  float* xt = reinterpret_cast<float*>(raw + StreamBytes() + (kWantDK ? 2 : 1) * OwnBytes(RM, d));   // [128 queries][64]
  float* wt = xt + 2 * kTile * kTile;                                                                 // [128 queries][kLd]
  __shared__ int first[2 * kTile];   // the first key each query reaches
  const TileAt tile = KeyTile(BH);
  const int j0 = tile.tile * R;
  const size_t bh = tile.bh, b = bh / H, h = bh % H, D = static_cast<size_t>(H) * d;
  const size_t base = b * S * D + h * d, at = base + static_cast<size_t>(j0) * D;
  const int c0 = blockIdx.y * kTile, c = (threadIdx.x & 15) * 4;
  const int nkeys = min(R, S - j0);
  const float* x = kWantDK ? q : dout;
  constexpr int OR = OutRows(RM);
  const int r0 = (threadIdx.x >> 4) * OR, r_at = min(r0, R - OR);   // this thread's keys of the output sums
  float acc[OR][4] = {};
  SliceRegs regs;
  int turn = 0;
  const int i_first = j0 / kTile * kTile, mine = i_first + group * kTile;
  if (mine < S) FetchSlice<kVec>(&regs, q + base + static_cast<size_t>(mine) * D, D, min(kTile, S - mine), 0, d);
  LoadOwn<R, kVec, kFused>(own_k, k + at, D, nkeys, d);
  if (kWantDK) LoadOwn<R, kVec, kFused>(own_v, v + at, D, nkeys, d);
  __syncthreads();
  for (int pair = i_first; pair < S; pair += 2 * kTile) {
    // The rows of x these tiles need, on their way while the scores are formed.
    for (int t = 0; t < 2 * kTile; t += kChunkRows) {
      const int rows = min(kChunkRows, S - pair - t);
      CopyChunk<kVec>(xt + t * kTile, x + base + static_cast<size_t>(rows > 0 ? pair + t : pair) * D, D, max(0, rows), c0, d);
    }
    const int i0 = pair + group * kTile;
    bool late = false;
    if (i0 < S) {
      const int rows = min(kTile, S - i0);
      const size_t iat = base + static_cast<size_t>(i0) * D;
      const float* q_next = i0 + 2 * kTile < S ? q + iat + 2 * kTile * D : nullptr;
      const int next_rows = min(kTile, S - i0 - 2 * kTile);
      double sc[RM][4], dp[RM][4];
      DotTile<RM, kVec, kFused>(own_k, q + iat, rows, kWantDK ? dout + iat : q_next, kWantDK ? rows : next_rows, D, d, slices, &turn,
                        &regs, sc);
      if (kWantDK) DotTile<RM, kVec, kFused>(own_v, dout + iat, rows, q_next, next_rows, D, d, slices, &turn, &regs, dp);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = i0 + Col<kFused>(e);
        const float* st = stats + (bh * S + min(i, S - 1)) * kAttnStatsWidth;
        const int start = static_cast<int>(StatsStart(st[3], static_cast<size_t>(i)));
        late = late || (i < S && start > j0);
        if (RowAt<kFused, RM>(0) == 0) first[group * kTile + Col<kFused>(e)] = start;
#pragma unroll
        for (int r = 0; r < RM; ++r) {
          const int j = j0 + RowAt<kFused, RM>(r);
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
          wt[(group * kTile + Col<kFused>(e)) * kLd + RowAt<kFused, RM>(r)] = g;
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    const bool segments = __syncthreads_or(late);
    const int rows = min(2 * kTile, S - pair);
    int lo[OR];
#pragma unroll
    for (int r = 0; r < OR; ++r) lo[r] = j0 + r_at + r - pair;
    if (pair >= j0 + R - 1 && !segments) ColProduct<kFused, OR, true>(wt + r_at, kLd, xt, rows, lo, acc);
    else ColProduct<kFused, OR, false>(wt + r_at, kLd, xt, rows, lo, acc, first, j0 + r_at);
    __syncthreads();   // wt, xt and first are rewritten for the next pair
  }
#pragma unroll
  for (int r = 0; r < OR; ++r)
    if (r0 + r < nkeys) StoreRow4(out + at + static_cast<size_t>(r0 + r) * D, acc[r], c0 + c, d, kVec);
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

// Rows per thread (per_rm of them times 16 or 8 to a block): four, the most arithmetic per shared-memory read, while
// the grid still has two blocks per SM, else two while it has one, else one.
inline int RowsPerThread(size_t BH, size_t S, int rows_per_rm, size_t chunks = 1) {
  for (int rm : {4, 2})
    if (BH * ((S + rows_per_rm * rm - 1) / (rows_per_rm * rm)) * chunks >= (rm == 4 ? 2u : 1u) * 148u) return rm;
  return 1;
}
// The same for the kernels whose score rows (`arrays` f32 rows of S keys, and as many own operands, per query row) live
// in shared memory: no more rows than let two blocks share an SM, or one block of 8 rows; 0: not even that fits.
inline size_t ScoreBytes(int rm, size_t S, size_t d, int arrays) {
  return StreamBytes() + static_cast<size_t>(arrays) * (OwnBytes(rm, static_cast<int>(d)) + 8 * rm * RowStride(S) * sizeof(float));
}
inline int RowsPerThreadWithScores(size_t BH, size_t S, size_t d, int arrays) {
  for (int rm = RowsPerThread(BH, S, 8); rm >= 1; rm /= 2)
    if (ScoreBytes(rm, S, d, arrays) <= kTwoPerSm) return rm;
  return ScoreBytes(1, S, d, arrays) <= kMaxSmem ? 1 : 0;
}
inline bool Vec(size_t d, std::initializer_list<const void*> ps) {
  if (d % 4 != 0) return false;
  for (const void* p : ps)
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;
  return true;
}
template <int RM>
using RowsTag = std::integral_constant<int, RM>;
// f(rows tag, fused tag, vector tag) with the constants of this launch.
template <typename F>
inline void WithTile(int rm, bool fused, bool vec, F f) {
  auto with_rows = [&](auto fu, auto v) {
    if (rm == 4) f(RowsTag<4>{}, fu, v);
    else if (rm == 2) f(RowsTag<2>{}, fu, v);
    else f(RowsTag<1>{}, fu, v);
  };
  auto with_fused = [&](auto v) {
    if (fused) with_rows(std::true_type{}, v);
    else with_rows(std::false_type{}, v);
  };
  if (vec) with_fused(std::true_type{});
  else with_fused(std::false_type{});
}
inline dim3 TileGrid(size_t BH, size_t tiles, size_t d) {
  return dim3(static_cast<unsigned>(BH * tiles), static_cast<unsigned>((d + kTile - 1) / kTile));
}

}  // namespace

// The dot-product identity a.b = b.a holds bit for bit here (each product is
// exact in double and the order over c is the same), so the tiled backward may
// take the key rows as the first operand and stream the query rows.

int AttnTileRows(size_t BH, size_t S, size_t d, bool score_rows) {
  return score_rows ? RowsPerThreadWithScores(BH, S, d, 1) : RowsPerThread(BH, S, 8);
}

void AttnFwd(const float* q, const float* k, const float* v, float* o, float* probs,
             float* stats, size_t B, size_t S, size_t H, size_t d, const int32_t* starts,
             bool fused, cudaStream_t s) {
  const size_t units = B * H * S;
  if (units == 0) return;
  const float inv_sqrt_d = 1.0f / sqrtf(static_cast<float>(d));
  if (const int rm = RowsPerThreadWithScores(B * H, S, d, 1); rm > 0) {
    WithTile(rm, fused, Vec(d, {q, k, v, o}), [&](auto rows, [[maybe_unused]] auto fu, auto vec) {
      constexpr int RM = decltype(rows)::value;
      const size_t bytes = ScoreBytes(RM, S, d, 1);
      AllowSmem(AttnFwdTileKernel<RM, decltype(fu)::value, decltype(vec)::value>, bytes);
      Next(AttnFwdTileKernel<RM, decltype(fu)::value, decltype(vec)::value>, static_cast<unsigned>(B * H * ((S + 8 * RM - 1) / (8 * RM))), kTileThreads, bytes, s)(
          q, k, v, o, probs, stats, static_cast<int>(B * H), static_cast<int>(S), static_cast<int>(H), static_cast<int>(d),
          starts, inv_sqrt_d);
    });
    return;
  }
  const size_t bytes = kWarps * (d + S) * sizeof(float);
  AllowSmem(AttnFwdKernel, bytes);
  Next(AttnFwdKernel, UnitBlocks(units), kWarps * 32, bytes, s)(q, k, v, o, probs, stats, B, S, H, d,
                                                             starts, inv_sqrt_d);
}

void AttnDP(const float* dout, const float* v, float* dp, size_t B, size_t S, size_t H, size_t d, bool own_order,
            cudaStream_t s) {
  if (B * H * S == 0) return;
  auto bytes = [&](int rm) { return StreamBytes() + OwnBytes(rm, static_cast<int>(d)); };
  int rm = RowsPerThread(B * H, S, 8);
  while (rm > 1 && bytes(rm) > kTwoPerSm) rm /= 2;
  if (bytes(rm) > kMaxSmem) {
    Next(AttnDPWideKernel, 148 * 8, 256, 0, s)(dout, v, dp, B * H, S, H, d);
    return;
  }
  WithTile(rm, own_order, Vec(d, {dout, v}), [&](auto rows, [[maybe_unused]] auto fu, auto vec) {
    constexpr int RM = decltype(rows)::value;
    AllowSmem(AttnDPTileKernel<RM, decltype(fu)::value, decltype(vec)::value>, bytes(RM));
    Next(AttnDPTileKernel<RM, decltype(fu)::value, decltype(vec)::value>, static_cast<unsigned>(B * H * ((S + 8 * RM - 1) / (8 * RM))), kTileThreads, bytes(RM), s)(
            dout, v, dp, static_cast<int>(B * H), static_cast<int>(S), static_cast<int>(H), static_cast<int>(d));
  });
}

namespace {

template <bool kScaled>
void ColSum(const float* w, const float* x, float* out, size_t B, size_t S, size_t H, size_t d, float scale,
            bool fused, cudaStream_t s) {
  if (B * H * S == 0) return;
  WithTile(RowsPerThread(B * H, S, 16, (d + kTile - 1) / kTile), fused, Vec(d, {x, out}), [&](auto rows, [[maybe_unused]] auto fu, auto vec) {
    constexpr int RM = decltype(rows)::value;
    Next(AttnColTileKernel<RM, decltype(fu)::value, kScaled, decltype(vec)::value>, TileGrid(B * H, (S + 16 * RM - 1) / (16 * RM), d), kTileThreads, 0, s)(
            w, x, out, static_cast<int>(B * H), static_cast<int>(S), static_cast<int>(H), static_cast<int>(d), scale);
  });
}

}  // namespace

void AttnDV(const float* probs, const float* dout, float* dv, size_t B, size_t S, size_t H,
            size_t d, bool fused, cudaStream_t s) {
  ColSum<false>(probs, dout, dv, B, S, H, d, 1.0f, fused, s);
}

void AttnDK(const float* ds, const float* q, float* dk, size_t B, size_t S, size_t H, size_t d, bool fused,
            cudaStream_t s) {
  ColSum<true>(ds, q, dk, B, S, H, d, 1.0f / sqrtf(static_cast<float>(d)), fused, s);
}

void AttnDQ(const float* ds, const float* k, float* dq, size_t B, size_t S, size_t H, size_t d,
            bool fused, cudaStream_t s) {
  if (B * H * S == 0) return;
  const float inv_sqrt_d = 1.0f / sqrtf(static_cast<float>(d));
  WithTile(RowsPerThread(B * H, S, 16, (d + kTile - 1) / kTile), fused, Vec(d, {k, dq}), [&](auto rows, [[maybe_unused]] auto fu, auto vec) {
    constexpr int RM = decltype(rows)::value;
    Next(AttnRowTileKernel<RM, decltype(fu)::value, decltype(vec)::value>, TileGrid(B * H, (S + 16 * RM - 1) / (16 * RM), d), kTileThreads, 0, s)(
            ds, k, dq, static_cast<int>(B * H), static_cast<int>(S), static_cast<int>(H), static_cast<int>(d), inv_sqrt_d);
  });
}

void SoftmaxRowsBwd(const float* probs, const float* dp, float* ds, size_t rows, size_t cols,
                    cudaStream_t s) {
  if (rows == 0) return;
  Next(SoftmaxRowsBwdKernel, UnitBlocks(rows), kWarps * 32, 0, s)(probs, dp, ds, rows, cols);
}

void AttnDQTiled(const float* q, const float* k, const float* v, const float* dout, float* stats,
                 float* dq, size_t B, size_t S, size_t H, size_t d, bool fused, cudaStream_t s) {
  const size_t units = B * H * S;
  if (units == 0) return;
  const float inv_sqrt_d = 1.0f / sqrtf(static_cast<float>(d));
  if (const int rm = RowsPerThreadWithScores(B * H, S, d, 2); rm > 0) {
    WithTile(rm, fused, Vec(d, {q, k, v, dout, dq}), [&](auto rows, [[maybe_unused]] auto fu, auto vec) {
      constexpr int RM = decltype(rows)::value;
      const size_t bytes = ScoreBytes(RM, S, d, 2);
      AllowSmem(AttnDQTiledTileKernel<RM, decltype(fu)::value, decltype(vec)::value>, bytes);
      Next(AttnDQTiledTileKernel<RM, decltype(fu)::value, decltype(vec)::value>, static_cast<unsigned>(B * H * ((S + 8 * RM - 1) / (8 * RM))), kTileThreads, bytes, s)(
              q, k, v, dout, stats, dq, static_cast<int>(B * H), static_cast<int>(S), static_cast<int>(H),
              static_cast<int>(d), inv_sqrt_d);
    });
    return;
  }
  const size_t bytes = kWarps * (2 * d + 2 * S) * sizeof(float);
  AllowSmem(AttnDQTiledKernel, bytes);
  Next(AttnDQTiledKernel, UnitBlocks(units), kWarps * 32, bytes, s)(q, k, v, dout, stats, dq, B, S, H,
                                                                 d, inv_sqrt_d);
}

void AttnDKVTiled(bool want_dk, const float* q, const float* k, const float* v, const float* dout,
                  const float* stats, float* out, size_t B, size_t S, size_t H, size_t d,
                  bool fused, cudaStream_t s) {
  if (B * H * S == 0) return;
  const float inv_sqrt_d = 1.0f / sqrtf(static_cast<float>(d));
  WithTile(RowsPerThread(B * H, S, 8, (d + kTile - 1) / kTile), fused, Vec(d, {q, k, v, dout, out}), [&](auto rows, [[maybe_unused]] auto fu, auto vec) {
    constexpr int RM = decltype(rows)::value;
    const size_t bytes = StreamBytes() + (want_dk ? 2 : 1) * OwnBytes(RM, static_cast<int>(d)) +
                         2 * kTile * (kTile + 8 * RM + 4) * sizeof(float);
    auto launch = [&](auto kernel) {
      AllowSmem(kernel, bytes);
      Next(kernel, TileGrid(B * H, (S + 8 * RM - 1) / (8 * RM), d), kTileThreads, bytes, s)(
          q, k, v, dout, stats, out, static_cast<int>(B * H), static_cast<int>(S), static_cast<int>(H),
          static_cast<int>(d), inv_sqrt_d);
    };
    if (want_dk) launch(AttnDKVTiledTileKernel<RM, true, decltype(fu)::value, decltype(vec)::value>);
    else launch(AttnDKVTiledTileKernel<RM, false, decltype(fu)::value, decltype(vec)::value>);
  });
}

}  // namespace see::k
