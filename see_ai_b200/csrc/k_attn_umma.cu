// Causal attention on the tensor cores, for the tiled attention opcodes that
// carry the relaxed permission (reference: source/plan/instruction.h:174-190,
// 356-382; the reference's own relaxed attention is the matrix-tile family of
// runtime/executor/metal_backend.mm:1742-1802).  Same contract as the exact
// tiled family (reference: runtime/executor/attention.cc:448-590): the forward
// writes O and the stats row {score max, 1/denominator, 0, start}; dQ writes
// delta into the stats row and dQ; dK and dV read the stats row.
//
// Blackwell-native: the operands are held once as bf16 in the tensors' own
// row-major layout [B*S, H*d] (written by the kernel that produces the tensor,
// or converted once), a (sequence, head) tile arrives by one 4-D TMA load
// (128-byte swizzle), every product
// (Q K^T, P V, dO V^T, dS K, dS^T Q, P^T dO) is a tcgen05.mma with its
// accumulator in tensor memory, and the softmax / softmax-backward arithmetic
// runs in f32 registers on values read with tcgen05.ld; P and dS go back to
// shared memory as bf16 for the second product.  Statistics are exact f32
// reductions of the bf16 products: two walks over the keys (first the row
// statistics, then the products), so no accumulator is ever rescaled.
//
// Sequences of several tiles and a step's backward run on dedicated warps (AttnFwdPairKernel, AttnBwdKernel, with their
// own comments below).  In the other kernels a CTA is 128 threads, one query row (or key row) per thread, and takes the
// other axis 64 positions per step, which keeps its footprint at 48-72 KB of
// shared memory and 128-256 columns of tensor memory: two to four CTAs share an
// SM and fill each other's load, MMA and exp latencies.  Thread 0 issues TMA
// and MMA; one tcgen05.commit per step covers the step's first product(s) and
// the previous step's second product.  Every mbarrier wait is bounded; a wait
// that runs out raises DeviceStatus::wait_timeout and the CTA stores nothing.
#include <cuda.h>

#include <type_traits>

#include "attn_umma.h"
#include "kernels.h"
#include "launch.cuh"
#include "shadow.cuh"
#include "umma_device.cuh"

namespace see::k {

using namespace umma_dev;

namespace {

constexpr uint32_t kTile = 128;          // query rows / key rows per tile
constexpr uint32_t kSubTileBytes = 128 * 64 * 2;   // [128 rows][64 bf16], swizzled
constexpr uint32_t kPBytes = 2 * kSubTileBytes;    // P / dS tile: 128 x 128 bf16

// ---- operand copies: f32 [B*S, H*d] -> bf16, same layout --------------------------------
// (Every operand tile of the kernels below is cut out of this copy by a 4-D tensor map
// {d, S, H, B}: 64 head-dimension elements x R positions of one head of one sequence land
// as [R][128 bytes] — the K-major tile of a product over the head dimension, and through an
// MN-major descriptor the operand of a product over the positions.)
__device__ __forceinline__ uint32_t Bf16Bits(float f) {   // round to nearest even; NaN stays NaN
  uint32_t u = __float_as_uint(f);
  if ((u & 0x7FFFFFFFu) > 0x7F800000u) return (u >> 16) | 0x0040u;
  u += 0x7FFFu + ((u >> 16) & 1u);
  return u >> 16;
}

__global__ void __launch_bounds__(256)
PackRowsKernel(const float* __restrict__ x, uint16_t* __restrict__ rows, size_t quads) {
  AwaitPrevious();
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t q = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; q < quads; q += stride) {
    const float4 f = reinterpret_cast<const float4*>(x)[q];
    reinterpret_cast<uint2*>(rows)[q] =
        make_uint2(Bf16Bits(f.x) | (Bf16Bits(f.y) << 16), Bf16Bits(f.z) | (Bf16Bits(f.w) << 16));
  }
}

struct Ctl {
  uint64_t bar_a;   // operands of the step's first product(s) have landed
  uint64_t bar_b;   // operand of the step's second product has landed
  uint64_t mma;     // the tensor core finished everything issued so far
  uint32_t tmem_base;
  uint32_t pad;
};

constexpr uint32_t kHalf = 64;                    // keys (or queries) per step
constexpr uint32_t kHalfTileBytes = 128 * 64 * 2; // P / dS step tile: [128 rows][64] bf16, swizzled
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float Exp2Approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Two f32 operations per instruction, each rounded as the scalar one.
using F2 = unsigned long long;
__device__ __forceinline__ F2 Pair(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float Lo(F2 v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ float Hi(F2 v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }
__device__ __forceinline__ F2 Fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ F2 Add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 Mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Loads [R positions][D] of head h of sequence b ({d, S, H, B} map with box {64, R, 1, 1}) as
// D/64 sub-tiles of R * 128 bytes; positions past the end of the sequence arrive as zeros.
template <int D, int R>
__device__ __forceinline__ void LoadRows(uint8_t* dst, const CUtensorMap* map, uint64_t* bar,
                                         uint32_t row0, uint32_t h, uint32_t b) {
#pragma unroll
  for (int kb = 0; kb < D / 64; ++kb)
    TmaLoad4D(dst + kb * (R * 128), map, bar, kb * 64, static_cast<int32_t>(row0), static_cast<int32_t>(h),
              static_cast<int32_t>(b));
}
// acc[128 x NB] = A[128 rows][D] . B[NB rows][D]^T, both row tiles in shared memory.
template <int D, int NB>
__device__ __forceinline__ void MmaRowRow(uint32_t tmem, const uint8_t* a, const uint8_t* b) {
  const uint32_t idesc = MakeInstrDesc(128, NB);
#pragma unroll
  for (int kb = 0; kb < D / 64; ++kb) {
    const uint64_t da = MakeSmemDesc(SmemAddr(a + kb * (128 * 128)));
    const uint64_t db = MakeSmemDesc(SmemAddr(b + kb * (NB * 128)));
#pragma unroll
    for (int k = 0; k < 4; ++k) UmmaBf16(tmem, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
  }
}
// acc[128 x D] (+)= P[128 rows][64] . T with T given as a ROW tile [64 positions][D]
// (the positions are the reduction index: an MN-major B operand), D / 64 sub-tiles of
// [64][64] as LoadRows<D, 64> leaves them.
template <int D>
__device__ __forceinline__ void MmaPRows(uint32_t tmem, const uint8_t* p, const uint8_t* t_rows,
                                         uint32_t accumulate) {
  const uint32_t idesc = MakeInstrDesc(128, D) | kInstrDescBMnMajor;
  const uint64_t da = MakeSmemDesc(SmemAddr(p));
  const uint32_t tb = SmemAddr(t_rows);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    UmmaBf16(tmem, da + 2 * k, MakeSmemDescMn(tb + k * 2048, 64 * 128), idesc, (accumulate | k) != 0 ? 1u : 0u);
}

// Writes 32 consecutive values of this thread's row (columns c0 .. c0+31 of the 64-wide
// step tile) into the swizzled bf16 tile.
__device__ __forceinline__ void StoreRowChunk(uint8_t* p_tile, uint32_t row, uint32_t c0,
                                              const float (&v)[32]) {
  const uint32_t chunk0 = c0 >> 3;   // first 16-byte chunk (8 bf16) of the four
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint4 w;
    w.x = PackBf16x2(v[8 * q + 0], v[8 * q + 1]);
    w.y = PackBf16x2(v[8 * q + 2], v[8 * q + 3]);
    w.z = PackBf16x2(v[8 * q + 4], v[8 * q + 5]);
    w.w = PackBf16x2(v[8 * q + 6], v[8 * q + 7]);
    *reinterpret_cast<uint4*>(p_tile + Sw128Offset(row, chunk0 + q)) = w;
  }
}

__device__ __forceinline__ uint8_t* AlignSmem(uint8_t* raw) {
  return raw + ((1024u - (SmemAddr(raw) & 1023u)) & 1023u);
}

// Stores a warp's 32 output rows (D accumulator columns starting at t_out, one row per
// thread, times the thread's `scale`).  The rows turn through a per-warp slab of shared
// memory (the operand tiles are idle by now) so that HBM sees whole rows: 16-byte chunks
// XOR-swizzled with the row, conflict-free both for the row-per-thread writes and the
// row-per-(half-)warp reads.  `out0` points at (first row, this head's first column) of
// the [B*S, H*d] tensor, `flat0` is that element's index (for the bf16 shadow), `col0`
// its column, `rows_live` how many of the 32 rows exist.
template <int D>
__device__ __forceinline__ void StoreOutRows(uint32_t t_out, float* slab, uint32_t lane, float scale,
                                             float* out0, size_t pitch, uint32_t rows_live,
                                             const Shadow& sh, size_t flat0, uint32_t col0,
                                             float* keep = nullptr) {
  constexpr uint32_t kChunks = D / 4;          // 16-byte chunks per row: 16 or 32
  constexpr uint32_t kRowsPerPass = 32 / kChunks;
#pragma unroll 1
  for (uint32_t c0 = 0; c0 < D; c0 += 32) {
    uint32_t r[32];
    TmemLoad32(t_out + c0, r);
    TmemWaitLd();
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q) {
      const uint32_t chunk = ((c0 >> 2) + q) ^ (lane & (kChunks - 1));
      *reinterpret_cast<float4*>(slab + lane * D + chunk * 4) =
          make_float4(__uint_as_float(r[4 * q]) * scale, __uint_as_float(r[4 * q + 1]) * scale,
                      __uint_as_float(r[4 * q + 2]) * scale, __uint_as_float(r[4 * q + 3]) * scale);
    }
  }
  __syncwarp();
  const uint32_t sub = lane / kChunks, cl = lane % kChunks;
#pragma unroll 4
  for (uint32_t rr = sub; rr < rows_live; rr += kRowsPerPass) {
    const float4 v = *reinterpret_cast<const float4*>(slab + rr * D + ((cl ^ (rr & (kChunks - 1))) * 4));
    *reinterpret_cast<float4*>(out0 + rr * pitch + cl * 4) = v;
    if (sh.dst) ShadowStore4(sh, (flat0 + rr * pitch + cl * 4) / 4, col0 + cl * 4, v);
    if (keep) *reinterpret_cast<float4*>(keep + flat0 + rr * pitch + cl * 4) = v;
  }
}

constexpr uint32_t TmemColsFor(uint32_t need) { return need <= 128 ? 128 : (need <= 256 ? 256 : 512); }

// ---- forward -------------------------------------------------------------------------
// A CTA owns 128 query rows of one (sequence, head) and walks the keys ONCE, 64 at
// a time.  Per step: S = Q K_h^T (128 x 64, tensor memory columns 0..63), read back
// one row per thread; p = 2^(s c - ref) against a per-row reference exponent, P
// written to shared memory as bf16, O += P V_h (columns 64..64+D) unnormalised.
// The reference follows the running maximum lazily: it moves (and the row's O
// and sum are multiplied by 2^(old - new), a read-modify-write of the row's
// tensor-memory lane) only when a step's maximum exceeds it by more than 2^8, so
// p stays below 256 — exact in f32 sums, the same relative rounding in bf16 —
// and most steps rescale nothing.  The true maximum is tracked beside it and the
// stats row gets {max, 1 / sum relative to that max}, what the backward kernels
// and the exact family expect.  Small footprint on purpose (48 KB of shared
// memory and 128 tensor-memory columns for d = 64): four CTAs share an SM and
// cover each other's waits.
constexpr float kRescaleSlack = 8.0f;   // log2 units

template <int D>
__global__ void __launch_bounds__(128)
AttnFwdUmmaKernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                  const __grid_constant__ CUtensorMap map_v, AttnUmmaArgs a) {
  extern __shared__ uint8_t smem_raw[];
  Ctl* ctl = reinterpret_cast<Ctl*>(smem_raw);             // barriers first, tiles 1024-aligned after
  uint8_t* smem = AlignSmem(smem_raw + sizeof(Ctl));
  constexpr uint32_t kQBytes = 128 * D * 2, kKBytes = 64 * D * 2, kVBytes = D * 128;
  uint8_t* q_s = smem;
  uint8_t* k_s = q_s + kQBytes;
  uint8_t* v_s = k_s + kKBytes;
  uint8_t* p_s = v_s + kVBytes;
  constexpr uint32_t kTmemCols = TmemColsFor(64 + D);

  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  const uint32_t n_qt = (a.S + kTile - 1) / kTile;
  const uint32_t it = n_qt - 1 - blockIdx.x;               // heaviest tiles first
  const uint32_t bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
  const uint32_t all_h = (a.S + kHalf - 1) / kHalf;
  const uint32_t total = 2 * (it + 1) < all_h ? 2 * (it + 1) : all_h;   // key steps up to the diagonal

  if (tid == 0) {
    MbarInit(&ctl->bar_a, 1); MbarInit(&ctl->bar_b, 1); MbarInit(&ctl->mma, 1);
    MbarInitFence();
  }
  if (warp == 0) TmemAlloc(&ctl->tmem_base, kTmemCols);
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  AwaitPrevious();
  const uint32_t tmem = ctl->tmem_base;
  const uint32_t t_s = tmem + ((warp * 32) << 16);
  const uint32_t t_o = t_s + 64;

  auto issue_a = [&](uint32_t t) {
    MbarExpectTx(&ctl->bar_a, kKBytes + (t == 0 ? kQBytes : 0));
    if (t == 0) LoadRows<D, 128>(q_s, &map_q, &ctl->bar_a, it * kTile, h, b);
    LoadRows<D, 64>(k_s, &map_k, &ctl->bar_a, t * kHalf, h, b);
  };
  auto issue_b = [&](uint32_t t) {
    MbarExpectTx(&ctl->bar_b, kVBytes);
    LoadRows<D, 64>(v_s, &map_v, &ctl->bar_b, t * kHalf, h, b);   // V_h as rows: the MN-major operand of P V
  };

  const uint32_t row = it * kTile + tid;                   // this thread's query row
  const float c1 = a.inv_sqrt_d * kLog2e;
  float raw_max = -INFINITY;   // the row's true score maximum so far
  float ref = -INFINITY;       // the exponent (log2 units) its p, sum and O are relative to
  float l = 0.0f;
  int failed = 0;
  if (tid == 0) issue_a(0);

  for (uint32_t t = 0; t < total; ++t) {
    if (warp == 0 && ElectOne()) {   // only the issuing thread needs the operands' arrival
      if (!MbarWait(&ctl->bar_a, t & 1)) failed = 1;
      TcFenceAfter();
      if (!failed) MmaRowRow<D, 64>(tmem, q_s, k_s);
      UmmaCommit(&ctl->mma);
    }
    // This commit also covers the previous step's O += P V, so p_s, v_s and k_s
    // are all free again once it arrives, and O is at rest.
    if (!MbarWait(&ctl->mma, t & 1)) failed = 1;
    TcFenceAfter();
    if (warp == 0 && ElectOne() && !failed) {
      if (t + 1 < total) issue_a(t + 1);
      issue_b(t);
    }
    const uint32_t key0 = t * kHalf;
    const bool diagonal = key0 + kHalf > it * kTile;   // some keys of this step lie above the diagonal
    uint32_t r[64];
    {
      uint32_t lo[32], hi[32];
      TmemLoad32(t_s, lo);
      TmemLoad32(t_s + 32, hi);
      TmemWaitLd();
#pragma unroll
      for (int j = 0; j < 32; ++j) { r[j] = lo[j]; r[32 + j] = hi[j]; }
    }
    float step_max = -INFINITY;
    if (diagonal) {
#pragma unroll
      for (int j = 0; j < 64; ++j)
        if (key0 + j <= row) step_max = fmaxf(step_max, __uint_as_float(r[j]));
    } else {
#pragma unroll
      for (int j = 0; j < 64; ++j) step_max = fmaxf(step_max, __uint_as_float(r[j]));
    }
    raw_max = fmaxf(raw_max, step_max);
    const float step_ref = step_max * c1;
    const bool moves = step_ref > ref + kRescaleSlack;   // always at a row's first live key (ref = -inf)
    float alpha = 1.0f;
    if (moves) {
      alpha = Exp2Approx(ref - step_ref);                // 0 the first time
      l *= alpha;
      ref = step_ref;
    }
    if (t > 0 && __any_sync(0xFFFFFFFFu, moves)) {       // the warp's rows rescale their O lanes together
#pragma unroll 1
      for (uint32_t c0 = 0; c0 < D; c0 += 32) {
        uint32_t o[32];
        TmemLoad32(t_o + c0, o);
        TmemWaitLd();
#pragma unroll
        for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
        TmemStore32(t_o + c0, o);
      }
      TmemWaitSt();
    }
#pragma unroll
    for (uint32_t c0 = 0; c0 < kHalf; c0 += 32) {
      float v[32];
      if (diagonal) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          v[j] = (key0 + c0 + j <= row) ? Exp2Approx(fmaf(__uint_as_float(r[c0 + j]), c1, -ref)) : 0.0f;
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = Exp2Approx(fmaf(__uint_as_float(r[c0 + j]), c1, -ref));
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) l += v[j];
      StoreRowChunk(p_s, tid, c0, v);
    }
    FenceProxyAsync();
    TcFenceBefore();
    if (__syncthreads_or(failed)) { failed = 1; break; }
    if (warp == 0 && ElectOne()) {
      if (!MbarWait(&ctl->bar_b, t & 1)) failed = 1;
      TcFenceAfter();
      if (!failed) MmaPRows<D>(tmem + 64, p_s, v_s, t != 0);
    }
  }
  if (warp == 0 && ElectOne()) UmmaCommit(&ctl->mma);
  if (!failed && !MbarWait(&ctl->mma, total & 1)) failed = 1;
  TcFenceAfter();
  failed = __syncthreads_or(failed);
  if (failed) {
    if (tid == 0) a.status->wait_timeout = 1;
    DrainDelay();
  } else {
    const bool live = row < a.S;
    const size_t HD = static_cast<size_t>(a.H) * D;
    const uint32_t row0w = it * kTile + warp * 32;
    const uint32_t rows_live = row0w < a.S ? (a.S - row0w < 32 ? a.S - row0w : 32) : 0;
    const size_t flat0 = (static_cast<size_t>(b) * a.S + row0w) * HD + static_cast<size_t>(h) * D;
    const float inv_l = 1.0f / l;
    StoreOutRows<D>(t_o, reinterpret_cast<float*>(smem) + warp * 32 * D, tid & 31, inv_l,
                    a.out + flat0, HD, rows_live, a.shadow, flat0, h * D, a.keep);
    if (live) {
      // The stats row speaks of the true maximum: the sum relative to it is l 2^(ref - max c).
      const float m = raw_max * a.inv_sqrt_d;
      const float inv_l_at_max = 1.0f / (l * Exp2Approx(ref - raw_max * c1));
      float* st = a.stats + (static_cast<size_t>(bh) * a.S + row) * kAttnStatsWidth;
      *reinterpret_cast<float4*>(st) = make_float4(m, inv_l_at_max, 0.0f, 0.0f);
    }
  }
  TcFenceBefore();
  __syncthreads();
  if (warp == 0) {
    TcFenceAfter();
    TmemFree(tmem, kTmemCols);
  }
}

// ---- dQ (and delta) --------------------------------------------------------------------
// Per 128 query rows, the keys 64 at a time.  Per step S = Q K_h^T (columns
// 0..63) and dP = dO V_h^T (64..127); dS = P (dP - delta) / sqrt(d) goes to shared
// memory as bf16 and dQ += dS K (columns 128..128+D).  A first walk over the keys sums
// delta_i = sum_j P_ij dP_ij; where the forward's kept copy of O is at hand the kernel
// with dedicated warps below takes the instruction instead.
template <int D>
__global__ void __launch_bounds__(128)
AttnDQUmmaKernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                 const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                 AttnUmmaArgs a) {
  extern __shared__ uint8_t smem_raw[];
  Ctl* ctl = reinterpret_cast<Ctl*>(smem_raw);
  uint8_t* smem = AlignSmem(smem_raw + sizeof(Ctl));
  constexpr uint32_t kFull = 128 * D * 2, kHalfRows = 64 * D * 2;
  uint8_t* q_s = smem;
  uint8_t* do_s = q_s + kFull;
  uint8_t* k_s = do_s + kFull;          // two buffers: step t's K_h also feeds dQ += dS K_h after the softmax,
  uint8_t* v_s = k_s + 2 * kHalfRows;   // while step t + 1's is already on its way
  uint8_t* p_s = v_s + kHalfRows;
  constexpr uint32_t kTmemCols = TmemColsFor(128 + D);

  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  const uint32_t n_qt = (a.S + kTile - 1) / kTile;
  const uint32_t it = n_qt - 1 - blockIdx.x;
  const uint32_t bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
  const uint32_t all_h = (a.S + kHalf - 1) / kHalf;
  const uint32_t n_h = 2 * (it + 1) < all_h ? 2 * (it + 1) : all_h;
  const uint32_t total = 2 * n_h;

  if (tid == 0) {
    MbarInit(&ctl->bar_a, 1); MbarInit(&ctl->bar_b, 1); MbarInit(&ctl->mma, 1);
    MbarInitFence();
  }
  if (warp == 0) TmemAlloc(&ctl->tmem_base, kTmemCols);
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  AwaitPrevious();
  const uint32_t tmem = ctl->tmem_base;
  const uint32_t t_lane = tmem + ((warp * 32) << 16);

  auto issue_a = [&](uint32_t t) {
    MbarExpectTx(&ctl->bar_a, 2 * kHalfRows + (t == 0 ? 2 * kFull : 0));
    if (t == 0) {
      LoadRows<D, 128>(q_s, &map_q, &ctl->bar_a, it * kTile, h, b);
      LoadRows<D, 128>(do_s, &map_do, &ctl->bar_a, it * kTile, h, b);
    }
    LoadRows<D, 64>(k_s + (t & 1) * kHalfRows, &map_k, &ctl->bar_a, (t % n_h) * kHalf, h, b);
    LoadRows<D, 64>(v_s, &map_v, &ctl->bar_a, (t % n_h) * kHalf, h, b);
  };

  const uint32_t row = it * kTile + tid;
  const bool live = row < a.S;
  float* st_row = a.stats + (static_cast<size_t>(bh) * a.S + (live ? row : 0)) * kAttnStatsWidth;
  const float c1 = a.inv_sqrt_d * kLog2e;
  // P = 2^(s * log2(e)/sqrt(d) - M) with M = max * log2(e) - log2(1/denominator).
  const float m2l = live ? st_row[0] * kLog2e - log2f(st_row[1]) : 0.0f;
  float delta = 0.0f;
  int failed = 0;
  if (tid == 0) issue_a(0);

  for (uint32_t t = 0; t < total; ++t) {
    const uint32_t jh = t % n_h;
    const bool second = t >= n_h;
    if (tid == 0) {
      if (!MbarWait(&ctl->bar_a, t & 1)) failed = 1;
      TcFenceAfter();
      if (!failed) {
        MmaRowRow<D, 64>(tmem, q_s, k_s + (t & 1) * kHalfRows);   // S  = Q K_h^T
        MmaRowRow<D, 64>(tmem + 64, do_s, v_s);    // dP = dO V_h^T
      }
      UmmaCommit(&ctl->mma);   // also covers the previous step's dQ += dS K_h
    }
    if (!MbarWait(&ctl->mma, t & 1)) failed = 1;
    TcFenceAfter();
    if (tid == 0 && !failed && t + 1 < total) issue_a(t + 1);
    __syncwarp();
    const uint32_t key0 = jh * kHalf;
    const bool diagonal = key0 + kHalf > it * kTile;
#pragma unroll 1
    for (uint32_t c0 = 0; c0 < kHalf; c0 += 32) {
      uint32_t rs[32], rp[32];
      TmemLoad32(t_lane + c0, rs);
      TmemLoad32(t_lane + 64 + c0, rp);
      TmemWaitLd();
      float pr[32];   // P = exp(s - max) / denominator, zero above the diagonal
      if (diagonal) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          pr[j] = (key0 + c0 + j <= row) ? Exp2Approx(fmaf(__uint_as_float(rs[j]), c1, -m2l)) : 0.0f;
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) pr[j] = Exp2Approx(fmaf(__uint_as_float(rs[j]), c1, -m2l));
      }
      if (!second) {
#pragma unroll
        for (int j = 0; j < 32; ++j) delta = fmaf(pr[j], __uint_as_float(rp[j]), delta);
      } else {
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = pr[j] * (__uint_as_float(rp[j]) - delta) * a.inv_sqrt_d;
        StoreRowChunk(p_s, tid, c0, v);
      }
    }
    if (second) FenceProxyAsync();
    TcFenceBefore();
    if (__syncthreads_or(failed)) { failed = 1; break; }
    if (second && tid == 0) {
      TcFenceAfter();
      MmaPRows<D>(tmem + 128, p_s, k_s + (t & 1) * kHalfRows, jh != 0);   // dQ += dS K_h (K_h as the MN-major operand)
    }
  }
  if (tid == 0) UmmaCommit(&ctl->mma);
  if (!failed && !MbarWait(&ctl->mma, total & 1)) failed = 1;
  TcFenceAfter();
  failed = __syncthreads_or(failed);
  if (failed) {
    if (tid == 0) a.status->wait_timeout = 1;
    DrainDelay();
  } else {
    const size_t HD = static_cast<size_t>(a.H) * D;
    const uint32_t row0w = it * kTile + warp * 32;
    const uint32_t rows_live = row0w < a.S ? (a.S - row0w < 32 ? a.S - row0w : 32) : 0;
    const size_t flat0 = (static_cast<size_t>(b) * a.S + row0w) * HD + static_cast<size_t>(h) * D;
    StoreOutRows<D>(t_lane + 128, reinterpret_cast<float*>(smem) + warp * 32 * D, tid & 31, 1.0f,
                    a.out + flat0, HD, rows_live, a.shadow, flat0, h * D);
    if (live) st_row[2] = delta;
  }
  TcFenceBefore();
  __syncthreads();
  if (warp == 0) {
    TcFenceAfter();
    TmemFree(tmem, kTmemCols);
  }
}

// ---- dK / dV ---------------------------------------------------------------------------
// Per 128 key rows, over the queries at or below the diagonal 64 at a time, in
// the transposed frame (one key row per thread, query index along the columns):
// S^T = K Q_h^T; P^T from the stats rows of those queries, folded into one
// number per query, M = max * log2(e) - log2(1/denominator), so that
// P^T = 2^(s * log2(e)/sqrt(d) - M).  dV += P^T dO_h, or
// dS^T = P^T (dP^T - delta) / sqrt(d) with dP^T = V dO_h^T and dK += dS^T Q_h.
// (The plan's kAttnDKTiled / kAttnDVTiled pair on the same operands goes to the kernel with
// dedicated warps below, which makes both in one walk.)
template <int D, bool kWantDK>
__global__ void __launch_bounds__(128)
AttnDKVUmmaKernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                  const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_do,
                  AttnUmmaArgs a) {
  extern __shared__ uint8_t smem_raw[];
  Ctl* ctl = reinterpret_cast<Ctl*>(smem_raw);
  uint8_t* smem = AlignSmem(smem_raw + sizeof(Ctl));
  constexpr uint32_t kFull = 128 * D * 2, kHalfRows = 64 * D * 2;
  uint8_t* k_s = smem;
  uint8_t* v_s = k_s + kFull;                                // dK only
  // Q_h and dO_h are double-buffered: a step's tiles also feed its second products
  // (as MN-major operands) after the softmax, while the next step's are on their way.
  uint8_t* q_s = v_s + (kWantDK ? kFull : 0);
  uint8_t* do_s = q_s + 2 * kHalfRows;
  uint8_t* p_s = do_s + 2 * kHalfRows;
  float* stat_s = reinterpret_cast<float*>(p_s + kHalfTileBytes);   // M[64], delta[64]
  constexpr uint32_t kOutCol = kWantDK ? 128 : 64;
  constexpr uint32_t kTmemCols = TmemColsFor(kOutCol + D);

  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  const uint32_t jt = blockIdx.x;                          // key tile; low tiles have the most work
  const uint32_t bh = blockIdx.y, b = bh / a.H, h = bh % a.H;
  const uint32_t all_h = (a.S + kHalf - 1) / kHalf;
  const uint32_t h0 = 2 * jt;                              // first query step: the diagonal
  const uint32_t total = all_h - h0;

  if (tid == 0) {
    MbarInit(&ctl->bar_a, 1); MbarInit(&ctl->bar_b, 1); MbarInit(&ctl->mma, 1);
    MbarInitFence();
  }
  if (warp == 0) TmemAlloc(&ctl->tmem_base, kTmemCols);
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  AwaitPrevious();
  const uint32_t tmem = ctl->tmem_base;
  const uint32_t t_lane = tmem + ((warp * 32) << 16);

  auto issue_a = [&](uint32_t t) {
    constexpr uint32_t kPer = 2 * kHalfRows, kOnce = (kWantDK ? 2 : 1) * kFull;
    MbarExpectTx(&ctl->bar_a, kPer + (t == 0 ? kOnce : 0));
    if (t == 0) {
      LoadRows<D, 128>(k_s, &map_k, &ctl->bar_a, jt * kTile, h, b);
      if (kWantDK) LoadRows<D, 128>(v_s, &map_v, &ctl->bar_a, jt * kTile, h, b);
    }
    LoadRows<D, 64>(q_s + (t & 1) * kHalfRows, &map_q, &ctl->bar_a, (h0 + t) * kHalf, h, b);
    LoadRows<D, 64>(do_s + (t & 1) * kHalfRows, &map_do, &ctl->bar_a, (h0 + t) * kHalf, h, b);
  };

  const uint32_t key = jt * kTile + tid;                    // this thread's key row
  const float c1 = a.inv_sqrt_d * kLog2e;
  int failed = 0;
  if (tid == 0) issue_a(0);

  for (uint32_t t = 0; t < total; ++t) {
    const uint32_t q0 = (h0 + t) * kHalf;
    if (tid < kHalf) {   // this step's queries (the previous step's readers passed a barrier)
      const uint32_t qi = q0 + tid;
      float M = INFINITY, dl = 0.0f;   // past the end of the sequence: P = 2^-inf = 0
      if (qi < a.S) {
        const float4 sv = *reinterpret_cast<const float4*>(
            a.stats + (static_cast<size_t>(bh) * a.S + qi) * kAttnStatsWidth);
        M = sv.x * kLog2e - log2f(sv.y);
        dl = sv.z;
      }
      stat_s[tid] = M;
      stat_s[kHalf + tid] = dl;
    }
    if (tid == 0) {
      if (!MbarWait(&ctl->bar_a, t & 1)) failed = 1;
      TcFenceAfter();
      if (!failed) {
        MmaRowRow<D, 64>(tmem, k_s, q_s + (t & 1) * kHalfRows);                          // S^T  = K Q_h^T
        if (kWantDK) MmaRowRow<D, 64>(tmem + 64, v_s, do_s + (t & 1) * kHalfRows);       // dP^T = V dO_h^T
      }
      UmmaCommit(&ctl->mma);   // also covers the previous step's second product
    }
    __syncthreads();           // stat_s is written
    if (!MbarWait(&ctl->mma, t & 1)) failed = 1;
    TcFenceAfter();
    if (tid == 0 && !failed && t + 1 < total) issue_a(t + 1);
    __syncwarp();
    const bool diagonal = q0 < jt * kTile + kTile;   // some (key, query) pairs are masked
#pragma unroll 1
    for (uint32_t c0 = 0; c0 < kHalf; c0 += 32) {
      uint32_t rs[32], rp[32];
      TmemLoad32(t_lane + c0, rs);
      if (kWantDK) TmemLoad32(t_lane + 64 + c0, rp);
      TmemWaitLd();
      float v[32];
#pragma unroll
      for (int j4 = 0; j4 < 32; j4 += 4) {
        const float4 M4 = *reinterpret_cast<const float4*>(&stat_s[c0 + j4]);
        const float Mv[4] = {M4.x, M4.y, M4.z, M4.w};
        float dv[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (kWantDK) {
          const float4 d4 = *reinterpret_cast<const float4*>(&stat_s[kHalf + c0 + j4]);
          dv[0] = d4.x; dv[1] = d4.y; dv[2] = d4.z; dv[3] = d4.w;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = j4 + u;
          float p = Exp2Approx(fmaf(__uint_as_float(rs[j]), c1, -Mv[u]));
          if (diagonal && key > q0 + c0 + j) p = 0.0f;
          v[j] = kWantDK ? p * (__uint_as_float(rp[j]) - dv[u]) * a.inv_sqrt_d : p;
        }
      }
      StoreRowChunk(p_s, tid, c0, v);
    }
    FenceProxyAsync();
    TcFenceBefore();
    if (__syncthreads_or(failed)) { failed = 1; break; }
    if (tid == 0) {   // the step's own Q_h / dO_h tiles again, now as the MN-major operands
      TcFenceAfter();
      const uint8_t* qh = q_s + (t & 1) * kHalfRows;
      const uint8_t* doh = do_s + (t & 1) * kHalfRows;
      MmaPRows<D>(tmem + kOutCol, p_s, kWantDK ? qh : doh, t != 0);   // dK += dS^T Q_h, or dV += P^T dO_h
    }
  }
  if (tid == 0) UmmaCommit(&ctl->mma);
  if (!failed && !MbarWait(&ctl->mma, total & 1)) failed = 1;
  TcFenceAfter();
  failed = __syncthreads_or(failed);
  if (failed) {
    if (tid == 0) a.status->wait_timeout = 1;
    DrainDelay();
  } else {
    const size_t HD = static_cast<size_t>(a.H) * D;
    const uint32_t row0w = jt * kTile + warp * 32;
    const uint32_t rows_live = row0w < a.S ? (a.S - row0w < 32 ? a.S - row0w : 32) : 0;
    const size_t flat0 = (static_cast<size_t>(b) * a.S + row0w) * HD + static_cast<size_t>(h) * D;
    StoreOutRows<D>(t_lane + kOutCol, reinterpret_cast<float*>(smem) + warp * 32 * D, tid & 31, 1.0f,
                    a.out + flat0, HD, rows_live, a.shadow, flat0, h * D);
  }
  TcFenceBefore();
  __syncthreads();
  if (warp == 0) {
    TcFenceAfter();
    TmemFree(tmem, kTmemCols);
  }
}


// ---- backward on dedicated warps -----------------------------------------------------------
// dQ (with delta from the forward's kept copy) and dK + dV in one walk, as one persistent CTA
// per SM whose warps have one job each, so that the chain load -> product -> exponentials ->
// product of one step overlaps the next step's and the next tile's:
//   warp 13      TMA: a tile's own 128 rows (double-buffered at d = 64) and a ring of 64-row steps
//   warp 12      first products: keeps two steps of S and dP in tensor memory ahead of the softmax
//   warps 0-7    the elementwise part: thread = row x 32 of the step's 64 columns; P and dS go back
//                to tensor memory as bf16, over the S and dP columns they came from, and are the A
//                operand of the second products there (no shared-memory tile, no proxy fence)
//   warp 14      second products, as soon as a step's P and dS are there
//   warps 8-11   outputs of the finished tile, and for dQ the row statistics of the next one
// Same products, operands and summation order as the kernels above, so the same bits.
//
// What bounds it: a 128 x 64 x 16 product holds the tensor pipe 62 cycles, so a step's twelve (dQ)
// or sixteen (dK/dV) take 750 or 990; the exponentials of 64 columns x 128 rows 512 cycles of the
// exp pipe.  A step takes about 1250 and 1350 cycles, the second products' commit on its way round
// the chain; one 128-thread CTA that did everything in turn took 4200, two to an SM.
// Measured: forward + dQ + dK/dV of 8 x 2048 positions of 16 heads 1024 -> 676 us (667 to 771 from run to run).  Two issuing
// warps because one spent as long waiting and issuing as the pipe worked (dQ of that size: 233 us
// with one, 202 with two, 178 with the element arithmetic in pairs).
template <int D, bool kKV>
struct BwdShape {
  static constexpr uint32_t kFix = 128 * D * 2;              // one own-row tile
  static constexpr uint32_t kStep = 64 * D * 2;              // one 64-row step tile
  static constexpr uint32_t kFixBufs = D == 64 ? 2 : 1;
  static constexpr uint32_t kStages = D == 64 ? 4 : 3;
  static constexpr uint32_t kOutCols = (kKV ? 2 : 1) * D;
  static constexpr uint32_t kOutBufs = 2 * kOutCols <= 256 ? 2 : 1;
  static constexpr uint32_t kOutCol = 256;                   // after two {S, dP} pairs of 64 + 64 columns
  static constexpr uint32_t kSlab = 32 * 64 * 4;             // a storing warp's staging
  static constexpr uint32_t kStats = 2 * 2 * 128 * 4 + 8 * 64 * 4;
  static constexpr size_t kSmem = kFixBufs * 2 * kFix + kStages * 2 * kStep + 4 * kSlab + kStats + 512 + 1024;
};

struct BwdCtl {
  uint64_t fix_full[2], fix_empty[2];
  uint64_t full[4], empty[4];
  uint64_t acc_full[2], p_full[2];
  uint64_t out_full[2], out_empty[2];
  uint64_t stat_full[2], stat_empty[2];
  uint32_t tmem_base;
  volatile uint32_t failed;   // some role's wait ran out: the others stop too
};
static_assert(sizeof(BwdCtl) <= 512, "control block");

// A bounded wait that also ends when another role of the CTA has given up.
template <typename Control>
__device__ __forceinline__ bool RoleWait(Control* ctl, uint64_t* bar, uint32_t parity) {
  const uint32_t addr = SmemAddr(bar);
  for (uint32_t it = 0; it < kWaitLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(addr), "r"(parity)
        : "memory");
    if (done) return true;
    if ((it & 255) == 255 && ctl->failed) return false;
  }
  ctl->failed = 1;
  return false;
}
// The same by a whole warp, with one answer: when another role gives up, lanes that still saw their barrier complete
// leave with the others instead of issuing a warp-wide tensor-memory access alone (and what follows stays warp-uniform
// for the compiler).
template <typename Control>
__device__ __forceinline__ bool WarpWait(Control* ctl, uint64_t* bar, uint32_t parity) {
  return __all_sync(0xFFFFFFFFu, RoleWait(ctl, bar, parity));
}

// The tiles of a CTA: heaviest first, dealt out in rounds that alternate direction (within 1.5 % of
// an even load from S = 2048 on, 10 % at 384 tiles of S = 512).
struct BwdTile { uint32_t row_tile, bh, steps, step0; };
template <bool kKV>
__device__ __forceinline__ bool BwdTileAt(uint32_t round, uint32_t S, uint32_t BH, BwdTile* t) {
  const uint32_t n_t = (S + kTile - 1) / kTile, all_h = (S + kHalf - 1) / kHalf;
  const uint32_t at = round * gridDim.x + ((round & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
  if (at >= n_t * BH) return false;   // only in the last round
  const uint32_t rank = at / BH;
  t->bh = at - rank * BH;
  t->row_tile = kKV ? rank : n_t - 1 - rank;
  t->step0 = kKV ? 2 * rank : 0;      // dK/dV: queries from the diagonal on; dQ: keys up to it
  const uint32_t upto = 2 * (t->row_tile + 1) < all_h ? 2 * (t->row_tile + 1) : all_h;
  t->steps = kKV ? all_h - t->step0 : upto;
  return true;
}

constexpr uint32_t kBwdThreads = 15 * 32;

// kKV false: x, y = Q, dO rows; u, w = K, V steps; out = dQ.
// kKV true:  x, y = K, V rows;  u, w = Q, dO steps; out = dK, out2 = dV (transposed frame).
template <int D, bool kKV>
__global__ void __launch_bounds__(kBwdThreads, 1)
AttnBwdKernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_y,
              const __grid_constant__ CUtensorMap map_u, const __grid_constant__ CUtensorMap map_w,
              AttnUmmaArgs a) {
  using Sh = BwdShape<D, kKV>;
  extern __shared__ uint8_t smem_raw[];
  BwdCtl* ctl = reinterpret_cast<BwdCtl*>(smem_raw);
  uint8_t* fix_s = AlignSmem(smem_raw + 512);
  uint8_t* ring_s = fix_s + Sh::kFixBufs * 2 * Sh::kFix;
  uint8_t* slab_s = ring_s + Sh::kStages * 2 * Sh::kStep;
  float* row_stat_s = reinterpret_cast<float*>(slab_s + 4 * Sh::kSlab);   // dQ: [2][{M, delta}][128]
  float* col_stat_s = row_stat_s + 2 * 2 * 128;                           // dK/dV: per warp {-M[32], -delta[32]}

  const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
  const uint32_t BH = a.B * a.H;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      MbarInit(&ctl->fix_full[i], 1); MbarInit(&ctl->fix_empty[i], 1);
      MbarInit(&ctl->acc_full[i], 1); MbarInit(&ctl->p_full[i], 8);
      MbarInit(&ctl->out_full[i], 1); MbarInit(&ctl->out_empty[i], 4);
      MbarInit(&ctl->stat_full[i], 4); MbarInit(&ctl->stat_empty[i], 8);
    }
    for (int i = 0; i < 4; ++i) { MbarInit(&ctl->full[i], 1); MbarInit(&ctl->empty[i], 1); }
    ctl->failed = 0;
    MbarInitFence();
  }
  if (warp == 12) TmemAlloc(&ctl->tmem_base, 512);
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  AwaitPrevious();
  constexpr uint32_t tmem = 0;   // all 512 columns are this CTA's

  if (warp == 13) {
    // ---- loads ----
    if (lane == 0) {
      uint32_t g = 0, i = 0;
      bool ok = true;
      BwdTile tl;
      for (; ok && BwdTileAt<kKV>(i, a.S, BH, &tl); ++i) {
        const uint32_t b = tl.bh / a.H, h = tl.bh - b * a.H;
        const uint32_t fb = i % Sh::kFixBufs;
        if (!(ok = RoleWait(ctl, &ctl->fix_empty[fb], ((i / Sh::kFixBufs) & 1) ^ 1))) break;
        uint8_t* fx = fix_s + fb * 2 * Sh::kFix;
        MbarExpectTx(&ctl->fix_full[fb], 2 * Sh::kFix);
        LoadRows<D, 128>(fx, &map_x, &ctl->fix_full[fb], tl.row_tile * kTile, h, b);
        LoadRows<D, 128>(fx + Sh::kFix, &map_y, &ctl->fix_full[fb], tl.row_tile * kTile, h, b);
        for (uint32_t t = 0; t < tl.steps; ++t, ++g) {
          const uint32_t s = g % Sh::kStages;
          if (!(ok = RoleWait(ctl, &ctl->empty[s], ((g / Sh::kStages) & 1) ^ 1))) break;
          uint8_t* st = ring_s + s * 2 * Sh::kStep;
          MbarExpectTx(&ctl->full[s], 2 * Sh::kStep);
          LoadRows<D, 64>(st, &map_u, &ctl->full[s], (tl.step0 + t) * kHalf, h, b);
          LoadRows<D, 64>(st + Sh::kStep, &map_w, &ctl->full[s], (tl.step0 + t) * kHalf, h, b);
        }
      }
      // Every slot's last release has arrived before the CTA may end.
      for (uint32_t k = 0; ok && k < Sh::kStages; ++k, ++g)
        ok = RoleWait(ctl, &ctl->empty[g % Sh::kStages], ((g / Sh::kStages) & 1) ^ 1);
      for (uint32_t k = 0; ok && k < Sh::kFixBufs; ++k, ++i)
        ok = RoleWait(ctl, &ctl->fix_empty[i % Sh::kFixBufs], ((i / Sh::kFixBufs) & 1) ^ 1);
    }
  } else if (warp == 12) {
    // ---- first products: S (or S^T) and dP of one step into its half of the accumulators ----
    // (the whole warp walks and waits; one elected lane issues)
    BwdTile tl;
    uint32_t g = 0;
    bool ok = true;
    for (uint32_t i = 0; ok && BwdTileAt<kKV>(i, a.S, BH, &tl); ++i) {
      const uint32_t fb = i % Sh::kFixBufs;
      if (!(ok = WarpWait(ctl, &ctl->fix_full[fb], (i / Sh::kFixBufs) & 1))) break;
      const uint8_t* fx = fix_s + fb * 2 * Sh::kFix;
      for (uint32_t t = 0; t < tl.steps; ++t, ++g) {
        const uint32_t s = g % Sh::kStages;
        if (!(ok = WarpWait(ctl, &ctl->full[s], (g / Sh::kStages) & 1))) break;
        // The accumulators' last reader: the second products two steps ago (which release their ring slot with it).
        if (g >= 2 && !(ok = WarpWait(ctl, &ctl->empty[(g - 2) % Sh::kStages], ((g - 2) / Sh::kStages) & 1))) break;
        TcFenceAfter();
        const uint8_t* st = ring_s + s * 2 * Sh::kStep;
        const uint32_t acc = tmem + (g & 1) * 128;
        if (ElectOne()) {
          MmaRowRow<D, 64>(acc, fx, st);
          MmaRowRow<D, 64>(acc + 64, fx + Sh::kFix, st + Sh::kStep);
          UmmaCommit(&ctl->acc_full[g & 1]);
          if (t + 1 == tl.steps) UmmaCommit(&ctl->fix_empty[fb]);
        }
        __syncwarp();
      }
    }
  } else if (warp == 14) {
    // ---- second products: dQ += dS K_h, or dK += dS^T Q_h and dV += P^T dO_h ----
    BwdTile tl;
    uint32_t g = 0;
    bool ok = true;
    const uint32_t idesc = MakeInstrDesc(128, D) | kInstrDescBMnMajor;
    for (uint32_t i = 0; ok && BwdTileAt<kKV>(i, a.S, BH, &tl); ++i) {
      const uint32_t ob = i % Sh::kOutBufs;
      const uint32_t out = tmem + Sh::kOutCol + ob * Sh::kOutCols;
      if (!(ok = WarpWait(ctl, &ctl->out_empty[ob], ((i / Sh::kOutBufs) & 1) ^ 1))) break;
      for (uint32_t t = 0; t < tl.steps; ++t, ++g) {
        const uint32_t s = g % Sh::kStages;
        if (!(ok = WarpWait(ctl, &ctl->p_full[g & 1], (g >> 1) & 1))) break;
        TcFenceAfter();
        const uint32_t acc = tmem + (g & 1) * 128;
        const uint32_t u = SmemAddr(ring_s + s * 2 * Sh::kStep);
        if (ElectOne()) {
#pragma unroll
          for (uint32_t k = 0; k < 4; ++k)   // 16 positions of the step: columns {0, 8} of each 32-column half
            UmmaBf16TmemA(out, acc + (k >> 1) * 32 + (k & 1) * 8, MakeSmemDescMn(u + k * 2048, 64 * 128), idesc,
                          (t | k) != 0 ? 1u : 0u);
          if constexpr (kKV) {
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
              UmmaBf16TmemA(out + D, acc + 64 + (k >> 1) * 32 + (k & 1) * 8,
                            MakeSmemDescMn(u + Sh::kStep + k * 2048, 64 * 128), idesc, (t | k) != 0 ? 1u : 0u);
          }
          UmmaCommit(&ctl->empty[s]);
          if (t + 1 == tl.steps) UmmaCommit(&ctl->out_full[ob]);
        }
        __syncwarp();
      }
    }
  } else if (warp < 8) {
    // ---- P and dS ----
    const uint32_t half = warp >> 2, quarter = warp & 3;
    const uint32_t r_in = quarter * 32 + lane;
    const uint32_t t_lane = tmem + ((quarter * 32) << 16) + half * 32;
    const float c1 = a.inv_sqrt_d * kLog2e;
    float* col_m = col_stat_s + warp * 64;
    uint32_t g = 0;
    bool ok = true;
    BwdTile tl;
    for (uint32_t i = 0; ok && BwdTileAt<kKV>(i, a.S, BH, &tl); ++i) {
      const uint32_t row0 = tl.row_tile * kTile, row = row0 + r_in;
      float m2l = 0.0f, delta = 0.0f;
      [[maybe_unused]] float4 next = make_float4(INFINITY, 1.0f, 0.0f, 0.0f);
      const float4* stats = reinterpret_cast<const float4*>(a.stats) + static_cast<size_t>(tl.bh) * a.S;
      if constexpr (kKV) {
        const uint32_t qi = tl.step0 * kHalf + half * 32 + lane;
        if (qi < a.S) next = stats[qi];   // past the end of the sequence: P = 2^-inf = 0
      } else {
        if (!(ok = WarpWait(ctl, &ctl->stat_full[i & 1], (i >> 1) & 1))) break;
        m2l = row_stat_s[(i & 1) * 256 + r_in];
        delta = row_stat_s[(i & 1) * 256 + 128 + r_in];
        __syncwarp();
        if (lane == 0) MbarArrive(&ctl->stat_empty[i & 1]);
      }
      for (uint32_t t = 0; t < tl.steps; ++t, ++g) {
        const uint32_t col0 = (tl.step0 + t) * kHalf + half * 32;   // this thread's first key (query)
        if constexpr (kKV) {
          __syncwarp();   // the previous step's readers
          col_m[lane] = -(next.x * kLog2e - log2f(next.y));
          col_m[32 + lane] = -next.z;
          next = make_float4(INFINITY, 1.0f, 0.0f, 0.0f);
          if (t + 1 < tl.steps && col0 + kHalf + lane < a.S) next = stats[col0 + kHalf + lane];
          __syncwarp();
        }
        if (!(ok = WarpWait(ctl, &ctl->acc_full[g & 1], (g >> 1) & 1))) break;
        TcFenceAfter();
        const uint32_t acc = t_lane + (g & 1) * 128;
        uint32_t rs[32], rp[32], w[16];
        TmemLoad32(acc, rs);
        TmemLoad32(acc + 64, rp);
        TmemWaitLd();
        [[maybe_unused]] uint32_t pw[16];
        // P = 2^(s c1 - M), dS = P (dP - delta) / sqrt(d); kDiag: some of the step's pairs are masked.
        auto elements = [&](auto diag) {
          constexpr bool kDiag = decltype(diag)::value;
#pragma unroll
          for (int j4 = 0; j4 < 32; j4 += 4) {
            F2 nm[2], nd[2];   // -M and -delta, of the row (dQ) or of the columns (dK/dV)
            if constexpr (kKV) {
              const float4 m4 = *reinterpret_cast<const float4*>(col_m + j4);
              const float4 d4 = *reinterpret_cast<const float4*>(col_m + 32 + j4);
              nm[0] = Pair(m4.x, m4.y); nm[1] = Pair(m4.z, m4.w);
              nd[0] = Pair(d4.x, d4.y); nd[1] = Pair(d4.z, d4.w);
            } else {
              nm[0] = nm[1] = Pair(-m2l, -m2l);
              nd[0] = nd[1] = Pair(-delta, -delta);
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const int j = j4 + 2 * q;
              const F2 x = Fma2(Pair(__uint_as_float(rs[j]), __uint_as_float(rs[j + 1])), Pair(c1, c1), nm[q]);
              float p0 = Exp2Approx(Lo(x)), p1 = Exp2Approx(Hi(x));
              if constexpr (kDiag) {
                if (kKV ? row > col0 + j : col0 + j > row) p0 = 0.0f;
                if (kKV ? row > col0 + j + 1 : col0 + j + 1 > row) p1 = 0.0f;
              }
              const F2 ds = Mul2(Mul2(Pair(p0, p1), Add2(Pair(__uint_as_float(rp[j]), __uint_as_float(rp[j + 1])), nd[q])),
                                 Pair(a.inv_sqrt_d, a.inv_sqrt_d));
              w[j / 2] = PackBf16x2(Lo(ds), Hi(ds));
              if constexpr (kKV) pw[j / 2] = PackBf16x2(p0, p1);
            }
          }
        };
        if (kKV ? col0 < row0 + kTile : col0 + 32 > row0) elements(std::true_type{});
        else elements(std::false_type{});
        if constexpr (kKV) TmemStore16(acc + 64, pw);
        TmemStore16(acc, w);
        TmemWaitSt();
        TcFenceBefore();
        __syncwarp();
        if (lane == 0) MbarArrive(&ctl->p_full[g & 1]);
      }
    }
  } else {
    // ---- outputs, and dQ's row statistics ----
    const uint32_t quarter = warp & 3, r_in = quarter * 32 + lane;
    float* slab = reinterpret_cast<float*>(slab_s + quarter * Sh::kSlab);
    const size_t HD = static_cast<size_t>(a.H) * D;
    bool ok = true;
    // dQ: P = 2^(s * log2(e)/sqrt(d) - M) with M = max * log2(e) - log2(1/denominator), and
    // delta_i = dO_i . O_i from the forward's kept copy of O.
    auto row_stats = [&](uint32_t i) {
      BwdTile tl;
      if (!BwdTileAt<kKV>(i, a.S, BH, &tl)) return;
      if (!(ok = WarpWait(ctl, &ctl->stat_empty[i & 1], ((i >> 1) & 1) ^ 1))) return;
      const uint32_t row = tl.row_tile * kTile + r_in, b = tl.bh / a.H, h = tl.bh - b * a.H;
      float m2l = 0.0f, delta = 0.0f;
      if (row < a.S) {
        float* st_row = a.stats + (static_cast<size_t>(tl.bh) * a.S + row) * kAttnStatsWidth;
        m2l = st_row[0] * kLog2e - log2f(st_row[1]);
        const size_t at = (static_cast<size_t>(b) * a.S + row) * HD + static_cast<size_t>(h) * D;
        const float4* orow = reinterpret_cast<const float4*>(a.fwd_keep + at);
        const uint2* drow = reinterpret_cast<const uint2*>(a.dout_bf16 + at);   // four bf16 per load
#pragma unroll 8
        for (int c = 0; c < D / 4; ++c) {
          const float4 o = orow[c];
          const uint2 e = drow[c];
          delta = fmaf(o.x, __uint_as_float(e.x << 16), delta);
          delta = fmaf(o.y, __uint_as_float(e.x & 0xFFFF0000u), delta);
          delta = fmaf(o.z, __uint_as_float(e.y << 16), delta);
          delta = fmaf(o.w, __uint_as_float(e.y & 0xFFFF0000u), delta);
        }
        st_row[2] = delta;
      }
      row_stat_s[(i & 1) * 256 + r_in] = m2l;
      row_stat_s[(i & 1) * 256 + 128 + r_in] = delta;
      __syncwarp();
      if (lane == 0) MbarArrive(&ctl->stat_full[i & 1]);
    };
    if constexpr (!kKV) row_stats(0);
    BwdTile tl;
    for (uint32_t i = 0; ok && BwdTileAt<kKV>(i, a.S, BH, &tl); ++i) {
      if constexpr (!kKV) {
        row_stats(i + 1);
        if (!ok) break;
      }
      const uint32_t ob = i % Sh::kOutBufs;
      if (!(ok = WarpWait(ctl, &ctl->out_full[ob], (i / Sh::kOutBufs) & 1))) break;
      TcFenceAfter();
      const uint32_t b = tl.bh / a.H, h = tl.bh - b * a.H;
      const uint32_t row0w = tl.row_tile * kTile + quarter * 32;
      const uint32_t rows_live = row0w < a.S ? (a.S - row0w < 32 ? a.S - row0w : 32) : 0;
      const size_t flat0 = (static_cast<size_t>(b) * a.S + row0w) * HD + static_cast<size_t>(h) * D;
      const uint32_t t_out = tmem + ((quarter * 32) << 16) + Sh::kOutCol + ob * Sh::kOutCols;
#pragma unroll 1
      for (uint32_t c = 0; c < D; c += 64) {
        StoreOutRows<64>(t_out + c, slab, lane, 1.0f, a.out + flat0 + c, HD, rows_live, a.shadow, flat0 + c, h * D + c);
        __syncwarp();   // the staging slab is reused
        if constexpr (kKV) {
          StoreOutRows<64>(t_out + D + c, slab, lane, 1.0f, a.out2 + flat0 + c, HD, rows_live, a.shadow2, flat0 + c,
                           h * D + c);
          __syncwarp();
        }
      }
      TcFenceBefore();
      __syncwarp();
      if (lane == 0) MbarArrive(&ctl->out_empty[ob]);
    }
  }
  __syncwarp();
  TcFenceBefore();
  __syncthreads();
  if (ctl->failed) {
    if (tid == 0) a.status->wait_timeout = 1;
    DrainDelay();
    __syncthreads();
  }
  if (warp == 12) {
    TcFenceAfter();
    TmemFree(ctl->tmem_base, 512);
  }
}

// ---- forward on dedicated warps ------------------------------------------------------------
// From two query tiles a sequence on.  One persistent CTA per SM works two neighbouring query tiles of a (sequence,
// head) at once, which share the keys' and values' steps of 64: a load warp, an issuing warp per tile, four warps per
// tile that turn scores into probabilities (a row per thread) and four that store finished tiles.  A tile has two
// score buffers, so the next step's scores are formed under this step's exponentials; P goes back to tensor memory as
// the second product's operand, and O, double-buffered for d = 64, leaves under the next tile's steps.  What is left
// is the exponentials: 8192 of them per step and tile on 16 lanes, 512 cycles, which the two tiles' warps keep busy
// in turn, where the one-CTA-per-tile kernel above spent 3100 cycles a step with four CTAs to an SM.  Measured: 8 x 2048
// positions of 16 heads 162 -> 115 us, 64 x 512 of 12 106 -> 83, 8 x 512 of 12 20.7 -> 15.4, 3 x 200 of 8 10.1 -> 9.7.  The row's
// reference exponent, its lazy rescaling and the statistics are that kernel's.
template <int D>
struct FwdShape {
  static constexpr uint32_t kQ = 128 * D * 2;                // one query tile
  static constexpr uint32_t kStep = 64 * D * 2;              // one step of keys, or of values
  static constexpr uint32_t kQBufs = D == 64 ? 2 : 1;        // of two tiles each
  static constexpr uint32_t kStages = D == 64 ? 5 : 3;
  static constexpr uint32_t kOutBufs = D == 64 ? 2 : 1;
  static constexpr uint32_t kOutCol = 128;                   // of a tile's 256 columns: after two score buffers
  static constexpr uint32_t kSlab = 32 * 64 * 4;
  static constexpr size_t kSmem = kQBufs * 2 * kQ + kStages * 2 * kStep + 4 * kSlab + 2 * 2 * 128 * 4 + 512 + 1024;
};
struct FwdCtl {
  uint64_t q_full[2], q_empty[2];
  uint64_t full[5], empty[5];
  uint64_t s_full[2][2], p_full[2][2], pv_done[2][2];   // [tile of the pair][score buffer]
  uint64_t out_full[2][2], out_empty[2][2], stat_full[2][2];
  uint32_t tmem_base;
  volatile uint32_t failed;
};
static_assert(sizeof(FwdCtl) <= 512, "control block");

// A CTA's pairs of tiles, heaviest first, dealt out in rounds that alternate direction.
struct FwdPair {
  uint32_t first_tile, bh, steps0, steps1, stream;
  __device__ __forceinline__ uint32_t Steps(uint32_t tile) const { return tile == 0 ? steps0 : steps1; }
};
__device__ __forceinline__ bool FwdPairAt(uint32_t round, uint32_t S, uint32_t BH, FwdPair* u) {
  const uint32_t n_t = (S + kTile - 1) / kTile, all_h = (S + kHalf - 1) / kHalf, n_u = (n_t + 1) / 2;
  const uint32_t at = round * gridDim.x + ((round & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
  if (at >= n_u * BH) return false;   // only in the last round
  const uint32_t rank = at / BH;
  u->bh = at - rank * BH;
  u->first_tile = 2 * (n_u - 1 - rank);
  auto steps = [&](uint32_t tile) { return tile >= n_t ? 0u : (2 * (tile + 1) < all_h ? 2 * (tile + 1) : all_h); };
  u->steps0 = steps(u->first_tile);
  u->steps1 = steps(u->first_tile + 1);
  u->stream = u->steps1 > u->steps0 ? u->steps1 : u->steps0;
  return true;
}

__device__ __forceinline__ float Max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

constexpr uint32_t kFwdThreads = 15 * 32;

template <int D>
__global__ void __launch_bounds__(kFwdThreads, 1)
AttnFwdPairKernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                  const __grid_constant__ CUtensorMap map_v, AttnUmmaArgs a) {
  using Sh = FwdShape<D>;
  extern __shared__ uint8_t smem_raw[];
  FwdCtl* ctl = reinterpret_cast<FwdCtl*>(smem_raw);
  uint8_t* q_s = AlignSmem(smem_raw + 512);
  uint8_t* ring_s = q_s + Sh::kQBufs * 2 * Sh::kQ;
  uint8_t* slab_s = ring_s + Sh::kStages * 2 * Sh::kStep;
  float* stat_s = reinterpret_cast<float*>(slab_s + 4 * Sh::kSlab);   // [tile of the pair][output buffer][128]: 1 / sum

  const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
  const uint32_t BH = a.B * a.H;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      MbarInit(&ctl->q_full[i], 1); MbarInit(&ctl->q_empty[i], 2);
      for (int j = 0; j < 2; ++j) {
        MbarInit(&ctl->s_full[i][j], 1); MbarInit(&ctl->p_full[i][j], 4); MbarInit(&ctl->pv_done[i][j], 1);
        MbarInit(&ctl->out_full[i][j], 1); MbarInit(&ctl->out_empty[i][j], 4); MbarInit(&ctl->stat_full[i][j], 4);
      }
    }
    for (int i = 0; i < 5; ++i) { MbarInit(&ctl->full[i], 1); MbarInit(&ctl->empty[i], 2); }
    ctl->failed = 0;
    MbarInitFence();
  }
  if (warp == 12) TmemAlloc(&ctl->tmem_base, 512);
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  AwaitPrevious();
  constexpr uint32_t tmem = 0;   // all 512 columns are this CTA's: 256 per tile of the pair

  if (warp == 14) {
    // ---- loads ----
    if (lane == 0) {
      uint32_t g = 0, i = 0;
      bool ok = true;
      FwdPair u;
      for (; ok && FwdPairAt(i, a.S, BH, &u); ++i) {
        const uint32_t b = u.bh / a.H, h = u.bh - b * a.H;
        const uint32_t qb = i % Sh::kQBufs;
        if (!(ok = RoleWait(ctl, &ctl->q_empty[qb], ((i / Sh::kQBufs) & 1) ^ 1))) break;
        uint8_t* q = q_s + qb * 2 * Sh::kQ;
        MbarExpectTx(&ctl->q_full[qb], (u.steps1 ? 2 : 1) * Sh::kQ);
        LoadRows<D, 128>(q, &map_q, &ctl->q_full[qb], u.first_tile * kTile, h, b);
        if (u.steps1) LoadRows<D, 128>(q + Sh::kQ, &map_q, &ctl->q_full[qb], (u.first_tile + 1) * kTile, h, b);
        for (uint32_t t = 0; t < u.stream; ++t, ++g) {
          const uint32_t s = g % Sh::kStages;
          if (!(ok = RoleWait(ctl, &ctl->empty[s], ((g / Sh::kStages) & 1) ^ 1))) break;
          uint8_t* st = ring_s + s * 2 * Sh::kStep;
          MbarExpectTx(&ctl->full[s], 2 * Sh::kStep);
          LoadRows<D, 64>(st, &map_k, &ctl->full[s], t * kHalf, h, b);
          LoadRows<D, 64>(st + Sh::kStep, &map_v, &ctl->full[s], t * kHalf, h, b);
        }
      }
      // Every slot's last release has arrived before the CTA may end.
      for (uint32_t k = 0; ok && k < Sh::kStages; ++k, ++g)
        ok = RoleWait(ctl, &ctl->empty[g % Sh::kStages], ((g / Sh::kStages) & 1) ^ 1);
      for (uint32_t k = 0; ok && k < Sh::kQBufs; ++k, ++i)
        ok = RoleWait(ctl, &ctl->q_empty[i % Sh::kQBufs], ((i / Sh::kQBufs) & 1) ^ 1);
    }
  } else if (warp >= 12) {
    // ---- products of one tile of the pair (the whole warp walks and waits; one elected lane issues) ----
    const uint32_t tile = warp - 12;
    const uint32_t base = tmem + tile * 256, idesc = MakeInstrDesc(128, D) | kInstrDescBMnMajor;
    FwdPair u;
    uint32_t g = 0, n = 0, j = 0;   // steps of the stream, of this tile's, finished tiles
    bool ok = true;
    for (uint32_t i = 0; ok && FwdPairAt(i, a.S, BH, &u); ++i) {
      const uint32_t qb = i % Sh::kQBufs, steps = u.Steps(tile), ob = j % Sh::kOutBufs;
      if (!(ok = WarpWait(ctl, &ctl->q_full[qb], (i / Sh::kQBufs) & 1))) break;
      const uint8_t* q = q_s + qb * 2 * Sh::kQ + tile * Sh::kQ;
      // The scores of step t (this tile's step m) into their buffer, whose last reader is P V two steps ago.  (A parity
      // tells one phase from the next only, so either buffer has a barrier of its own: its step m - 4 was waited for
      // before m - 2 was issued, also where a tile ended in between.)
      auto scores = [&](uint32_t t, uint32_t m) {
        const uint32_t at = g + t, s = at % Sh::kStages;
        if (!WarpWait(ctl, &ctl->full[s], (at / Sh::kStages) & 1)) return false;
        if (m >= 2 && !WarpWait(ctl, &ctl->pv_done[tile][m & 1], ((m >> 1) - 1) & 1)) return false;
        TcFenceAfter();
        if (ElectOne()) {
          MmaRowRow<D, 64>(base + (m & 1) * 64, q, ring_s + s * 2 * Sh::kStep);
          UmmaCommit(&ctl->s_full[tile][m & 1]);
          if (t + 1 == steps) UmmaCommit(&ctl->q_empty[qb]);
        }
        __syncwarp();
        return true;
      };
      if (steps == 0) {
        if (lane == 0) MbarArrive(&ctl->q_empty[qb]);
      } else {
        if (!(ok = scores(0, n))) break;
        if (!(ok = WarpWait(ctl, &ctl->out_empty[tile][ob], ((j / Sh::kOutBufs) & 1) ^ 1))) break;
        for (uint32_t t = 0; t < steps; ++t, ++n) {
          if (t + 1 < steps && !(ok = scores(t + 1, n + 1))) break;
          if (!(ok = WarpWait(ctl, &ctl->p_full[tile][n & 1], (n >> 1) & 1))) break;
          TcFenceAfter();
          const uint32_t s = (g + t) % Sh::kStages, v = SmemAddr(ring_s + s * 2 * Sh::kStep + Sh::kStep);
          if (ElectOne()) {
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
              UmmaBf16TmemA(base + Sh::kOutCol + ob * D, base + (n & 1) * 64 + k * 8, MakeSmemDescMn(v + k * 2048, 64 * 128),
                            idesc, (t | k) != 0 ? 1u : 0u);
            UmmaCommit(&ctl->pv_done[tile][n & 1]);
            UmmaCommit(&ctl->empty[s]);
            if (t + 1 == steps) UmmaCommit(&ctl->out_full[tile][ob]);
          }
          __syncwarp();
        }
        if (!ok) break;
        ++j;
      }
      for (uint32_t t = steps; t < u.stream; ++t) {   // steps that only the other tile takes
        const uint32_t s = (g + t) % Sh::kStages;
        if (!(ok = WarpWait(ctl, &ctl->full[s], ((g + t) / Sh::kStages) & 1))) break;
        if (lane == 0) MbarArrive(&ctl->empty[s]);
      }
      g += u.stream;
    }
  } else if (warp < 8) {
    // ---- probabilities ----
    const uint32_t tile = warp >> 2, quarter = warp & 3, r_in = quarter * 32 + lane;
    const uint32_t t_base = tmem + tile * 256 + ((quarter * 32) << 16);
    const float c1 = a.inv_sqrt_d * kLog2e;
    FwdPair u;
    uint32_t n = 0, j = 0;
    bool ok = true;
    for (uint32_t i = 0; ok && FwdPairAt(i, a.S, BH, &u); ++i) {
      const uint32_t steps = u.Steps(tile), ob = j % Sh::kOutBufs;
      if (steps == 0) continue;
      const uint32_t row0 = (u.first_tile + tile) * kTile, row = row0 + r_in;
      const uint32_t t_o = t_base + Sh::kOutCol + ob * D;
      float raw_max = -INFINITY;   // the row's true score maximum so far
      float ref = -INFINITY;       // the exponent (log2 units) its p, sum and O are relative to
      float l = 0.0f;              // the row's sum: one chain, the order of the kernel above
      for (uint32_t t = 0; t < steps; ++t, ++n) {
        if (!(ok = WarpWait(ctl, &ctl->s_full[tile][n & 1], (n >> 1) & 1))) break;
        TcFenceAfter();
        const uint32_t t_s = t_base + (n & 1) * 64, key0 = t * kHalf;
        uint32_t lo[32], hi[32];
        TmemLoad32(t_s, lo);
        TmemLoad32(t_s + 32, hi);
        TmemWaitLd();
        if (key0 + kHalf > row0) {   // some keys of this step lie above the diagonal
          constexpr uint32_t kMinusInf = 0xFF800000u;
#pragma unroll
          for (uint32_t e = 0; e < 32; ++e) {
            if (key0 + e > row) lo[e] = kMinusInf;
            if (key0 + 32 + e > row) hi[e] = kMinusInf;
          }
        }
        float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          m[0] = Max3(m[0], __uint_as_float(lo[e]), __uint_as_float(lo[e + 1]));
          m[1] = Max3(m[1], __uint_as_float(lo[e + 2]), __uint_as_float(lo[e + 3]));
          m[2] = Max3(m[2], __uint_as_float(hi[e]), __uint_as_float(hi[e + 1]));
          m[3] = Max3(m[3], __uint_as_float(hi[e + 2]), __uint_as_float(hi[e + 3]));
        }
        const float step_max = fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
        raw_max = fmaxf(raw_max, step_max);
        const float step_ref = step_max * c1;
        const bool moves = step_ref > ref + kRescaleSlack;   // always at a row's first live key (ref = -inf)
        float alpha = 1.0f;
        if (moves) {
          alpha = Exp2Approx(ref - step_ref);                // 0 the first time
          l *= alpha;
          ref = step_ref;
        }
        if (t > 0 && __any_sync(0xFFFFFFFFu, moves)) {       // the warp's rows rescale their O lanes together
          if (!(ok = WarpWait(ctl, &ctl->pv_done[tile][(n - 1) & 1], ((n - 1) >> 1) & 1))) break;
          TcFenceAfter();
#pragma unroll 1
          for (uint32_t c0 = 0; c0 < D; c0 += 16) {
            uint32_t o[16];
            TmemLoad16(t_o + c0, o);
            TmemWaitLd();
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
            TmemStore16(t_o + c0, o);
          }
          TmemWaitSt();
        }
        // p = 2^(s c1 - ref), packed over the scores' own registers.
        const F2 scale = Pair(c1, c1), shift = Pair(-ref, -ref);
        auto half = [&](uint32_t (&x)[32]) {
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const F2 y = Fma2(Pair(__uint_as_float(x[e]), __uint_as_float(x[e + 1])), scale, shift);
            const float p0 = Exp2Approx(Lo(y)), p1 = Exp2Approx(Hi(y));
            l += p0;
            l += p1;
            x[e / 2] = PackBf16x2(p0, p1);
          }
        };
        half(lo);
        half(hi);
        uint32_t w[32];
#pragma unroll
        for (int e = 0; e < 16; ++e) { w[e] = lo[e]; w[16 + e] = hi[e]; }
        TmemStore32(t_s, w);
        TmemWaitSt();
        TcFenceBefore();
        __syncwarp();
        if (lane == 0) MbarArrive(&ctl->p_full[tile][n & 1]);
      }
      if (!ok) break;
      if (row < a.S) {
        // The stats row speaks of the true maximum: the sum relative to it is l 2^(ref - max c).
        const float m = raw_max * a.inv_sqrt_d;
        const float inv_l_at_max = 1.0f / (l * Exp2Approx(ref - raw_max * c1));
        *reinterpret_cast<float4*>(a.stats + (static_cast<size_t>(u.bh) * a.S + row) * kAttnStatsWidth) =
            make_float4(m, inv_l_at_max, 0.0f, 0.0f);
      }
      if (!(ok = WarpWait(ctl, &ctl->out_empty[tile][ob], ((j / Sh::kOutBufs) & 1) ^ 1))) break;
      stat_s[(tile * 2 + ob) * 128 + r_in] = 1.0f / l;
      __syncwarp();
      if (lane == 0) MbarArrive(&ctl->stat_full[tile][ob]);
      ++j;
    }
  } else {
    // ---- outputs ----
    const uint32_t quarter = warp & 3, r_in = quarter * 32 + lane;
    float* slab = reinterpret_cast<float*>(slab_s + quarter * Sh::kSlab);
    const size_t HD = static_cast<size_t>(a.H) * D;
    uint32_t done0 = 0, done1 = 0;   // finished tiles of either place
    bool ok = true;
    FwdPair u;
    for (uint32_t i = 0; ok && FwdPairAt(i, a.S, BH, &u); ++i) {
      const uint32_t b = u.bh / a.H, h = u.bh - b * a.H;
#pragma unroll
      for (uint32_t tile = 0; tile < 2; ++tile) {
        if (!ok || u.Steps(tile) == 0) continue;
        uint32_t& j = tile == 0 ? done0 : done1;
        const uint32_t ob = j % Sh::kOutBufs, parity = (j / Sh::kOutBufs) & 1;
        if (!(ok = WarpWait(ctl, &ctl->out_full[tile][ob], parity) && WarpWait(ctl, &ctl->stat_full[tile][ob], parity))) break;
        TcFenceAfter();
        const float inv_l = stat_s[(tile * 2 + ob) * 128 + r_in];
        const uint32_t row0w = (u.first_tile + tile) * kTile + quarter * 32;
        const uint32_t rows_live = row0w < a.S ? (a.S - row0w < 32 ? a.S - row0w : 32) : 0;
        const size_t flat0 = (static_cast<size_t>(b) * a.S + row0w) * HD + static_cast<size_t>(h) * D;
        const uint32_t t_out = tmem + tile * 256 + ((quarter * 32) << 16) + Sh::kOutCol + ob * D;
#pragma unroll 1
        for (uint32_t c = 0; c < D; c += 64) {
          StoreOutRows<64>(t_out + c, slab, lane, inv_l, a.out + flat0 + c, HD, rows_live, a.shadow, flat0 + c, h * D + c,
                           a.keep);
          __syncwarp();   // the staging slab is reused
        }
        TcFenceBefore();
        __syncwarp();
        if (lane == 0) MbarArrive(&ctl->out_empty[tile][ob]);
        ++j;
      }
    }
  }
  __syncwarp();
  TcFenceBefore();
  __syncthreads();
  if (ctl->failed) {
    if (tid == 0) a.status->wait_timeout = 1;
    DrainDelay();
    __syncthreads();
  }
  if (warp == 12) {
    TcFenceAfter();
    TmemFree(ctl->tmem_base, 512);
  }
}

}  // namespace

size_t AttnFwdSmem(int d) { return 128 * d * 2 + 64 * d * 2 + d * 128 + kHalfTileBytes + 1152; }
size_t AttnDQSmem(int d) { return 2 * 128 * d * 2 + 3 * 64 * d * 2 + kHalfTileBytes + 1152; }
size_t AttnDKVSmem(int d, bool dk) {
  const size_t full = 128 * d * 2, half = 64 * d * 2;
  return (dk ? 2 : 1) * full + 4 * half + kHalfTileBytes + 2 * kHalf * 4 + 1152;
}

template <typename Kernel>
static cudaError_t Configure(Kernel kernel, size_t smem) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
}

void PackHeads(const float* x, uint16_t* rows, uint32_t B, uint32_t S, uint32_t H, uint32_t d, cudaStream_t s) {
  const size_t quads = static_cast<size_t>(B) * S * H * d / 4;
  const size_t blocks = (quads + 255) / 256;
  Next(PackRowsKernel, static_cast<unsigned>(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, s)(x, rows, quads);
}

template <int D>
static cudaError_t LaunchFwdPair(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const AttnUmmaArgs& a,
                                 cudaStream_t s) {
  const size_t smem = FwdShape<D>::kSmem;
  if (cudaError_t e = Configure(AttnFwdPairKernel<D>, smem); e != cudaSuccess) return e;
  const uint32_t pairs = ((a.S + kTile - 1) / kTile + 1) / 2 * a.B * a.H;
  Next(AttnFwdPairKernel<D>, pairs < a.sms ? pairs : a.sms, kFwdThreads, smem, s)(q, k, v, a);
  return cudaGetLastError();
}

// Which forward takes a geometry (both give the same bits).  Pairs share the keys' steps and keep the exponentials' pipe
// busy, but an SM works one pair at a time in whole rounds, and a short walk does not repay its longer set-up; the
// one-tile form has four CTAs to an SM (two for d = 128), started at once.  Measured on a B200, pairs / one tile, us, d = 64:
//   3 steps of keys: 24 heads of 192 positions 9.9 / 9.5, 192 of them (1.3 rounds) 15.2 / 12.1, 256 15.1 / 14.0; once the one-tile
//     CTAs are no longer all resident, 384, 18.6 / 19.4
//   4 steps: 48 of 256 10.2 / 11.2, 192 (1.3 rounds) 16.2 / 14.5, 256 (1.73) 16.0 / 16.9, 384 20.7 / 22.2
//   5 steps, three tiles, the last with a CTA of pairs to itself: 48 of 320 10.8 / 12.7, 96 (1.3 rounds) 15.6 / 14.0, 144 (1.95)
//     15.5 / 16.1, 192 (2.59) 19.5 / 18.0, 256 (3.46, not all resident) 24.1 / 24.8
//   6 steps: 96 of 384 15.5 / 15.6, 192 20.4 / 20.0, others 0.72 to 0.92; from 7 on pairs always
// and d = 128: 3 steps, 64 of 192 13.1 / 11.5, 128 15.1 / 13.5, 192 (not all resident) 21.3 / 21.2; 4 steps, 8 of 256 12.9 / 12.6,
// 128 15.3 / 15.9.
static bool PairsForward(const AttnUmmaArgs& a) {
  const uint64_t steps = (a.S + kHalf - 1) / kHalf, tiles = (a.S + kTile - 1) / kTile, heads = static_cast<uint64_t>(a.B) * a.H;
  const uint64_t ctas = tiles * heads, units = (tiles + 1) / 2 * heads, sms = a.sms;
  const bool resident = ctas <= (a.d == 64 ? 4u : 2u) * sms;
  if (steps <= 2) return false;   // a single tile has no neighbour to share its keys with
  if (steps == 3) return !resident;
  if (a.d == 128) return steps > 4 || ctas > sms;
  if (steps > 5 || !resident || units <= sms) return true;
  const uint64_t rounds = (units + sms - 1) / sms;
  return units * 10 >= rounds * sms * (steps == 4 ? 8 : 9);   // the last round is nearly full
}

cudaError_t AttnFwdUmma(const CUtensorMap& q, const CUtensorMap& k_half, const CUtensorMap& v_half,
                        const AttnUmmaArgs& a, cudaStream_t s) {
  if (PairsForward(a)) return a.d == 64 ? LaunchFwdPair<64>(q, k_half, v_half, a, s) : LaunchFwdPair<128>(q, k_half, v_half, a, s);
  dim3 grid((a.S + kTile - 1) / kTile, a.B * a.H);
  const size_t smem = AttnFwdSmem(a.d);
  cudaError_t e;
  if (a.d == 64) {
    if ((e = Configure(AttnFwdUmmaKernel<64>, smem)) != cudaSuccess) return e;
    Next(AttnFwdUmmaKernel<64>, grid, 128, smem, s)(q, k_half, v_half, a);
  } else {
    if ((e = Configure(AttnFwdUmmaKernel<128>, smem)) != cudaSuccess) return e;
    Next(AttnFwdUmmaKernel<128>, grid, 128, smem, s)(q, k_half, v_half, a);
  }
  return cudaGetLastError();
}

template <int D, bool kKV>
static cudaError_t LaunchBwd(const CUtensorMap& x, const CUtensorMap& y, const CUtensorMap& u, const CUtensorMap& w,
                             const AttnUmmaArgs& a, cudaStream_t s) {
  const size_t smem = BwdShape<D, kKV>::kSmem;
  if (cudaError_t e = Configure(AttnBwdKernel<D, kKV>, smem); e != cudaSuccess) return e;
  const uint32_t tiles = (a.S + kTile - 1) / kTile * a.B * a.H;
  Next(AttnBwdKernel<D, kKV>, tiles < a.sms ? tiles : a.sms, kBwdThreads, smem, s)(x, y, u, w, a);
  return cudaGetLastError();
}

cudaError_t AttnDQUmma(const CUtensorMap& q, const CUtensorMap& dout, const CUtensorMap& k_half,
                       const CUtensorMap& v_half, const AttnUmmaArgs& a, cudaStream_t s) {
  if (a.fwd_keep)
    return a.d == 64 ? LaunchBwd<64, false>(q, dout, k_half, v_half, a, s)
                     : LaunchBwd<128, false>(q, dout, k_half, v_half, a, s);
  dim3 grid((a.S + kTile - 1) / kTile, a.B * a.H);
  const size_t smem = AttnDQSmem(a.d);
  cudaError_t e;
  if (a.d == 64) {
    if ((e = Configure(AttnDQUmmaKernel<64>, smem)) != cudaSuccess) return e;
    Next(AttnDQUmmaKernel<64>, grid, 128, smem, s)(q, dout, k_half, v_half, a);
  } else {
    if ((e = Configure(AttnDQUmmaKernel<128>, smem)) != cudaSuccess) return e;
    Next(AttnDQUmmaKernel<128>, grid, 128, smem, s)(q, dout, k_half, v_half, a);
  }
  return cudaGetLastError();
}

cudaError_t AttnDKVUmma(int mode, const CUtensorMap& k, const CUtensorMap& v,
                        const CUtensorMap& q_half, const CUtensorMap& dout_half, const AttnUmmaArgs& a,
                        cudaStream_t s) {
  if (mode == 2)
    return a.d == 64 ? LaunchBwd<64, true>(k, v, q_half, dout_half, a, s)
                     : LaunchBwd<128, true>(k, v, q_half, dout_half, a, s);
  dim3 grid((a.S + kTile - 1) / kTile, a.B * a.H);
  cudaError_t e;
#define SEE_LAUNCH_DKV(D, DK)                                                                \
  do {                                                                                       \
    const size_t smem = AttnDKVSmem(D, DK);                                                  \
    if ((e = Configure(AttnDKVUmmaKernel<D, DK>, smem)) != cudaSuccess) return e;          \
    Next(AttnDKVUmmaKernel<D, DK>, grid, 128, smem, s)(k, v, q_half, dout_half, a);   \
  } while (0)
  if (a.d == 64) {
    if (mode == 1) SEE_LAUNCH_DKV(64, true); else SEE_LAUNCH_DKV(64, false);
  } else {
    if (mode == 1) SEE_LAUNCH_DKV(128, true); else SEE_LAUNCH_DKV(128, false);
  }
#undef SEE_LAUNCH_DKV
  return cudaGetLastError();
}

}  // namespace see::k
