// The low-rank (LoRA) side of an adapted projection, engine mode.
//
// An adapted projection is y = x W + s (x A) B with W frozen and A [k_in, r],
// B [r, n_out] trainable, r = 4..16.  The plan spells it as separate rank-r
// products (reference: compiler/analysis/algebra/lora_grafter.cc:170-206); the
// reference's own GPU backend folds the expand product C' = s T B + C into the
// base GEMM (reference: runtime/executor/metal_backend.mm:1155-1316).  Here the
// fold rides the tensor cores: the f32 factors are cut into three bf16 pieces
// each, t = t0 + t1 + t2, b = b0 + b1 + b2 (every piece the bf16 rounding of
// what the earlier pieces left, so the pieces are exact and the remainder is
// below 2^-24 |t|), and the six products with the largest weight
//
//     t0 b0 + t0 b1 + t1 b0 + t0 b2 + t1 b1 + t2 b0
//
// are appended to the base product's reduction as 6 r extra columns of K
// (zero-padded to a multiple of 64), smallest products first: the tensor core
// adds each 16-term group into its f32 accumulator with truncation, an error of
// up to one unit in the last place of the ACCUMULATOR per group and always
// toward zero, so the many small terms go in while the accumulator is still
// small and only the K/16 groups of t0 b0 meet it at full size (measured at
// K = 8192: 4.7e-6 of sum|a b| with the large products first, against 2e-6 asked).  bf16 x bf16 products are exact in the
// f32 accumulator, so the appended term equals the f32 product t . b to a few
// 2^-24 of |t| |b|: the accuracy class of the exact kernels, at the cost of one
// or two more K blocks on a tensor pipe that is idle most of the time at these
// shapes.  (The dropped products t1 b2, t2 b1, t2 b2 are below 2^-24 |t||b|.)
//
// This file holds the operand preparation: SplitRows turns a [M, r] f32 factor
// into its [M, KX] bf16 row operand, SplitWeights turns every adapter matrix of
// a range into its [N, KX] operand in one launch.  Compiled WITH fused
// multiply-add: nothing here reproduces a CPU rounding sequence bit for bit.
#include "kernels.h"
#include "launch.cuh"
#include "lora_split.cuh"

namespace see::k {

namespace {

// One thread per (row, four columns of t): 4 values in, their pieces out to the six
// segments; the threads of a row also zero its padding columns [6 R, KX).
template <int R>
__global__ void SplitRowsKernel(const float* __restrict__ t, uint16_t* __restrict__ out, uint32_t M, uint32_t KX) {
  AwaitPrevious();
  constexpr uint32_t kQuads = R / 4;
  const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t row = idx / kQuads, j = (idx - row * kQuads) * 4;
  if (row >= M) return;
  const float4 v = *reinterpret_cast<const float4*>(t + static_cast<size_t>(row) * R + j);
  uint16_t piece[4][3];
  Split3(v.x, piece[0]); Split3(v.y, piece[1]); Split3(v.z, piece[2]); Split3(v.w, piece[3]);
  uint16_t* dst = out + static_cast<size_t>(row) * KX;
#pragma unroll
  for (int s = 0; s < 6; ++s) {
    const int pc = PieceOf(0, s);
    uint2 w;
    w.x = static_cast<uint32_t>(piece[0][pc]) | (static_cast<uint32_t>(piece[1][pc]) << 16);
    w.y = static_cast<uint32_t>(piece[2][pc]) | (static_cast<uint32_t>(piece[3][pc]) << 16);
    *reinterpret_cast<uint2*>(dst + s * R + j) = w;
  }
  for (uint32_t k = 6 * R + j; k < KX; k += R) *reinterpret_cast<uint2*>(dst + k) = make_uint2(0u, 0u);
}

// One thread per (entry, output column n, four neighbouring columns of its operand row): r is a multiple of four, so
// the four are one piece of four neighbouring factor values, scaled and cut, and a warp writes whole lines of the
// [N, KX] operand.  (A thread per row, two bytes at a time, took 82 us for the 96 matrices of twelve layers of
// 768 x 16; cutting every value once per segment costs less than its stores did.)
__global__ void SplitWeightsKernel(const LoraWeight* __restrict__ table, int count) {
  AwaitPrevious();
  const LoraWeight e = table[blockIdx.y];
  const uint32_t quads = e.kx / 4, idx = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t n = idx / quads, c = (idx - n * quads) * 4;
  if (n >= e.n_out) return;
  uint32_t w[2] = {0u, 0u};   // past the six segments: zero padding
  if (c < 6 * e.r) {
    // What the base product's epilogue will multiply the whole tile by has to be
    // divided out of the low-rank term first.
    const float tile_scale = e.col_scale ? e.col_scale[n] : e.tile_alpha;
    const uint32_t s = c / e.r, j0 = c - s * e.r;
    const int piece = PieceOf(1, static_cast<int>(s));
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
      const uint32_t j = j0 + q;
      const float v = e.by_column ? e.src[static_cast<size_t>(n) * e.r + j]       // A [n_out, r]
                                  : e.src[static_cast<size_t>(j) * e.n_out + n];  // B [r, n_out]
      uint16_t p[3];
      Split3(e.alpha * v / tile_scale, p);
      const uint32_t bits = piece == 0 ? p[0] : piece == 1 ? p[1] : p[2];
      w[q >> 1] |= bits << (16 * (q & 1));
    }
  }
  *reinterpret_cast<uint2*>(e.dst + static_cast<size_t>(n) * e.kx + c) = make_uint2(w[0], w[1]);
}

// ---- whole matrices: an f32 GEMM on the bf16 tensor cores -------------------------------
// dst [rows][3 Kp] bf16, Kp = cols rounded up to 64: piece p of element c at column p Kp + c, zero padding after
// cols.  src is [rows][cols], or [cols][rows] when transposed (then a 32 x 32 tile goes through shared memory so both
// sides stay coalesced).  An element is multiplied by k_scale[c] first when that is given.  HBM-bound (4 bytes read,
// 6 written per element); which pieces a product multiplies, and in which order, is the GEMM's segment list.
// A thread takes eight columns: 32 bytes in, 16 bytes out per piece.
template <bool kVec>
__global__ void SplitMatrixKernel(const float* __restrict__ src, uint16_t* __restrict__ dst, uint32_t rows,
                                  uint32_t cols, uint32_t kp, const float* __restrict__ k_scale) {
  AwaitPrevious();
  const uint32_t per_row = kp / 8;
  const size_t octs = static_cast<size_t>(rows) * per_row;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t q = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; q < octs; q += stride) {
    const uint32_t row = static_cast<uint32_t>(q / per_row), c = static_cast<uint32_t>(q % per_row) * 8;
    const float* p = src + static_cast<size_t>(row) * cols + c;
    float v[8];
    if (kVec) {   // cols % 4 == 0: four elements are all in or all out
#pragma unroll
      for (uint32_t h = 0; h < 8; h += 4) {
        const float4 f = c + h < cols ? *reinterpret_cast<const float4*>(p + h) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[h] = f.x; v[h + 1] = f.y; v[h + 2] = f.z; v[h + 3] = f.w;
      }
    } else {
#pragma unroll
      for (uint32_t e = 0; e < 8; ++e) v[e] = c + e < cols ? p[e] : 0.0f;
    }
    if (k_scale) {
#pragma unroll
      for (uint32_t e = 0; e < 8; ++e)
        if (c + e < cols) v[e] = v[e] * k_scale[c + e];
    }
    uint32_t w[3][4];
#pragma unroll
    for (uint32_t e = 0; e < 8; e += 2) {
      uint16_t lo[3], hi[3];
      Split3(v[e], lo);
      Split3(v[e + 1], hi);
#pragma unroll
      for (uint32_t i = 0; i < 3; ++i) w[i][e / 2] = static_cast<uint32_t>(lo[i]) | (static_cast<uint32_t>(hi[i]) << 16);
    }
    uint16_t* out = dst + static_cast<size_t>(row) * 3 * kp + c;
#pragma unroll
    for (uint32_t i = 0; i < 3; ++i)
      *reinterpret_cast<uint4*>(out + static_cast<size_t>(i) * kp) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
  }
}

// src [cols][rows] -> dst row r, column c = src[c][r].
__global__ void SplitMatrixTransposedKernel(const float* __restrict__ src, uint16_t* __restrict__ dst,
                                            uint32_t rows, uint32_t cols, uint32_t kp, const float* __restrict__ k_scale) {
  AwaitPrevious();
  __shared__ float tile[32][33];
  const uint32_t r0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  for (uint32_t i = threadIdx.y; i < 32; i += blockDim.y) {
    const uint32_t c = c0 + i, r = r0 + threadIdx.x;
    float v = c < cols && r < rows ? src[static_cast<size_t>(c) * rows + r] : 0.0f;
    if (k_scale && c < cols) v = v * k_scale[c];
    tile[i][threadIdx.x] = v;
  }
  __syncthreads();
  // Two neighbouring columns per thread: 4-byte stores, sixteen threads per row.
  const uint32_t t = threadIdx.y * 32 + threadIdx.x, c2 = (t & 15) * 2;
  for (uint32_t i = t >> 4; i < 32; i += blockDim.y * 2) {
    const uint32_t r = r0 + i;
    if (r >= rows) continue;
    uint16_t lo[3], hi[3];
    Split3(tile[c2][i], lo);
    Split3(tile[c2 + 1][i], hi);
    uint16_t* out = dst + static_cast<size_t>(r) * 3 * kp + c0 + c2;
#pragma unroll
    for (int p = 0; p < 3; ++p)
      *reinterpret_cast<uint32_t*>(out + static_cast<size_t>(p) * kp) =
          static_cast<uint32_t>(lo[p]) | (static_cast<uint32_t>(hi[p]) << 16);
  }
}

}  // namespace

void SplitMatrix(const float* src, uint16_t* dst, size_t rows, size_t cols, bool transposed, const float* k_scale,
                 cudaStream_t s) {
  if (rows == 0 || cols == 0) return;
  const uint32_t kp = static_cast<uint32_t>((cols + 63) / 64 * 64);
  const uint32_t r = static_cast<uint32_t>(rows), c = static_cast<uint32_t>(cols);
  if (transposed) {
    const dim3 grid((r + 31) / 32, kp / 32), block(32, 8);
    Next(SplitMatrixTransposedKernel, grid, block, 0, s)(src, dst, r, c, kp, k_scale);
    return;
  }
  size_t blocks = (rows * (kp / 8) + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  const bool vec = cols % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  if (vec) Next(SplitMatrixKernel<true>, static_cast<unsigned>(blocks), 256, 0, s)(src, dst, r, c, kp, k_scale);
  else Next(SplitMatrixKernel<false>, static_cast<unsigned>(blocks), 256, 0, s)(src, dst, r, c, kp, k_scale);
}

uint32_t LoraSplitColumns(uint32_t r) { return (6 * r + 63) / 64 * 64; }

bool LoraSplitRows(const float* t, uint16_t* out, size_t M, uint32_t r, cudaStream_t s) {
  if ((reinterpret_cast<uintptr_t>(t) & 15) != 0 || (reinterpret_cast<uintptr_t>(out) & 15) != 0) return false;
  const uint32_t KX = LoraSplitColumns(r);
  const unsigned blocks = static_cast<unsigned>((M * (r / 4) + 255) / 256);
  switch (r) {
    case 4: Next(SplitRowsKernel<4>, blocks, 256, 0, s)(t, out, static_cast<uint32_t>(M), KX); return true;
    case 8: Next(SplitRowsKernel<8>, blocks, 256, 0, s)(t, out, static_cast<uint32_t>(M), KX); return true;
    case 12: Next(SplitRowsKernel<12>, blocks, 256, 0, s)(t, out, static_cast<uint32_t>(M), KX); return true;
    case 16: Next(SplitRowsKernel<16>, blocks, 256, 0, s)(t, out, static_cast<uint32_t>(M), KX); return true;
    default: return false;
  }
}

void LoraSplitWeights(const LoraWeight* table, int count, uint32_t max_n_out, uint32_t max_kx, cudaStream_t s) {
  if (count <= 0 || max_n_out == 0) return;
  const size_t quads = static_cast<size_t>(max_n_out) * (max_kx / 4);
  const dim3 grid(static_cast<unsigned>((quads + 255) / 256), static_cast<unsigned>(count));
  Next(SplitWeightsKernel, grid, 256, 0, s)(table, count);
}

}  // namespace see::k
