// f32-accurate products of an f32 activation that lies row-major (A [M, K], K fastest) on the tensor cores, the
// activation cut into its three bf16 pieces on the way into shared memory:
//
//     C[M,N] = epilogue( A[M,K] . B[N,K]^T )      B: three bf16 pieces of an f32 weight, or one that is it exactly
//
// The same piece products in the same order as the piece form of k_gemm_umma.cu (UmmaEpilogue::seg_blocks): 64 k at a
// time in one accumulator, the blocks added in f32 registers.  There the pieces are a matrix of their own, made by a
// launch of its own (six bytes written for four read, read back twice over), and every piece product loads both its
// tiles anew: 6 x (16 + 32) KB per 64 k of a 128 x 256 tile.  Here 32 KB of f32 and each piece of B once: what a small
// product (4096 x 256 x 256 of an f32 decoder, 4096 x 768 x 768 of an int8 one) waited for.
//
// One CTA a tile (or a cluster of `splits`, each a part of K): warp 0 brings B by TMA, warp 1 issues tcgen05.mma.  An f32
// weight's few blocks of six products are cut and added by sixteen warps in turn, 64 k at a time: cut block k (its f32 already
// in registers) into the ring, ask for block k + 1, add the accumulator of block k - 1 into their registers while the tensor core
// multiplies block k.  An exact weight's blocks have three products and are many, so eight warps only cut and eight or, of wide tiles,
// sixteen only add: of a block of 128 x 192 cutting takes 1500 cycles, adding 1250 (tensor memory is read against the products
// that run), the products 1150; in turn that was 3000.  Then the tile goes through the ring's memory and leaves as whole rows.
// (4096 x 768 x 768 of int8 22.4 / 19.8 us, 4096 x 768 x 3072 61.7 / 56.0, 2048 x 512 x 2048 24.1 / 21.4, 600 x 2048 x 512 14.4 / 12.9; f32
// weights apart: 4096 x 256 x 256 9.2 / 9.0, 4096 x 256 x 1024 17.7 / 18.6, 300 x 5000 x 256 10.7 / 10.8.)
//
// Every wait on an mbarrier is bounded; one that runs out raises DeviceStatus::wait_timeout and the CTA stores nothing.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "launch.cuh"
#include "lora_split.cuh"
#include "umma_device.cuh"
#include "umma_epilogue.cuh"
#include "umma_kernel.h"

namespace see::k {

namespace {

using namespace umma_dev;
using namespace umma_epi;

constexpr uint32_t kBlockM = umma_cfg::kBlockM, kBlockK = umma_cfg::kBlockK;
constexpr uint32_t kPieceBytes = kBlockM * kBlockK * 2;   // one bf16 piece of a block of A
constexpr uint32_t kMaxStages = 3;

template <uint32_t kTN, uint32_t kBPieces>
struct CutShape {
  static constexpr uint32_t kBBytes = kTN * kBlockK * 2;   // one piece of a block of B
  static constexpr uint32_t kStageBytes = 3 * kPieceBytes + kBPieces * kBBytes;
  static constexpr uint32_t kFit = 216u * 1024u / kStageBytes;
  static constexpr uint32_t kStages = kFit < kMaxStages ? kFit : kMaxStages;
  static constexpr uint32_t kAccCols = kTN <= 64 ? 64 : (kTN <= 128 ? 128 : 256);
  // kApart (an exact weight: many blocks, of three products each): eight warps cut and eight or, of wide tiles, sixteen add.
  // Otherwise (an f32 weight: a few blocks of six) sixteen warps do both in turn.
  static constexpr bool kApart = kBPieces == 1;
  static constexpr uint32_t kCutWarps = kApart ? 8 : 16, kAddWarps = kApart && kTN <= 128 ? 8 : 16, kFirstAdd = kApart ? 2 + kCutWarps : 2;
  static constexpr uint32_t kColsPerWarp = kTN * 4 / kAddWarps;   // an adding warp has 32 rows of so many columns
  static constexpr uint32_t kWorkThreads = 32 * (kApart ? kCutWarps + kAddWarps : 16), kThreads = 64 + kWorkThreads;
  static constexpr size_t kSmem = kStages * kStageBytes + 512 + 1024;
  static_assert(kStages >= 1 && kStages * kStageBytes >= kBlockM * kTN * 4, "the epilogue stages the whole tile in the ring");
};

struct __align__(8) CutBarriers {
  uint64_t a_full[kMaxStages], b_full[kMaxStages], empty[kMaxStages];
  uint64_t tmem_full[2], tmem_empty[2];
  uint32_t tmem_base;
  volatile uint32_t abort;
  volatile uint32_t nonfinite;
};

// How a block of A comes: loads of 16 bytes alone (src_k % 4 == 0: four elements are all in or all out), the same with a scale
// along k, loaded likewise, or one element at a time.
enum class Loads { kPlain, kScaled, kAny };

// A thread's part of the 128 x 64 f32 elements of block kb: some of the warp's rows, four apart, eight columns of each.
template <uint32_t kWarps, Loads kLoads>
struct CutRegs {
  static constexpr uint32_t kRows = kBlockM / (4 * kWarps);
  float4 v[2 * kRows];
  float4 scale[kLoads == Loads::kScaled ? 2 : 1];   // (the columns', for when the elements are cut)
  static __device__ __forceinline__ uint32_t Row(uint32_t h) {
    return ((threadIdx.x >> 5) - 2) * (4 * kRows) + h * 4 + ((threadIdx.x & 31) >> 3);
  }
};
// The loads alone, so that the thread goes on while they fly; a choice between two ways of loading, or a product, would end in
// moves that wait for them (int8 products in exact arithmetic with a scale along k, us, one element at a time / so: 4096 x 768 x 768
// 38.8 / 21.7, 2048 x 512 x 2048 43.6 / 23.4, 4096 x 768 x 3072 126 / 62.9; without a scale 20.4, 21.5, 56.7).
template <Loads kLoads, uint32_t kWarps>
__device__ __forceinline__ void FetchBlock(CutRegs<kWarps, kLoads>* f, const UmmaEpilogue& ep, uint32_t m0, uint32_t kb) {
  const uint32_t k = kb * kBlockK + (threadIdx.x & 7) * 8;
  if constexpr (kLoads == Loads::kScaled) {
#pragma unroll
    for (uint32_t q = 0; q < 2; ++q)
      f->scale[q] = k + 4 * q < ep.src_k ? __ldg(reinterpret_cast<const float4*>(ep.src_a_scale + k + 4 * q)) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (uint32_t h = 0; h < f->kRows; ++h) {
    const uint32_t row = m0 + f->Row(h);
    const float* p = ep.src_a + static_cast<size_t>(row) * ep.src_k + k;
#pragma unroll
    for (uint32_t q = 0; q < 2; ++q) {
      const uint32_t c = k + 4 * q;
      float4& x = f->v[2 * h + q];
      x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row >= ep.M || c >= ep.src_k) continue;
      if constexpr (kLoads != Loads::kAny) {
        x = __ldg(reinterpret_cast<const float4*>(p + 4 * q));
      } else {
        auto at = [&](uint32_t e) {
          if (c + e >= ep.src_k) return 0.0f;
          return ep.src_a_scale ? p[4 * q + e] * ep.src_a_scale[c + e] : p[4 * q + e];
        };
        x = make_float4(at(0), at(1), at(2), at(3));
      }
    }
  }
}
// Two elements' pieces, packed (Split3's values).
__device__ __forceinline__ void CutPair(float lo, float hi, uint32_t (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    p[i] = PackBf16x2(lo, hi);
    lo = lo - __uint_as_float(p[i] << 16);
    hi = hi - __uint_as_float(p[i] & 0xFFFF0000u);
  }
}
template <uint32_t kWarps, Loads kLoads>
__device__ __forceinline__ void StoreBlock(uint8_t* pieces, const CutRegs<kWarps, kLoads>& f) {
#pragma unroll
  for (uint32_t h = 0; h < f.kRows; ++h) {
    uint32_t w[3][4];
#pragma unroll
    for (uint32_t q = 0; q < 2; ++q) {
      float4 x = f.v[2 * h + q];
      if constexpr (kLoads == Loads::kScaled) x = make_float4(x.x * f.scale[q].x, x.y * f.scale[q].y, x.z * f.scale[q].z, x.w * f.scale[q].w);
      uint32_t a[3], b[3];
      CutPair(x.x, x.y, a);
      CutPair(x.z, x.w, b);
#pragma unroll
      for (int i = 0; i < 3; ++i) { w[i][2 * q] = a[i]; w[i][2 * q + 1] = b[i]; }
    }
    const uint32_t at = Sw128Offset(f.Row(h), threadIdx.x & 7);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      *reinterpret_cast<uint4*>(pieces + i * kPieceBytes + at) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
  }
}

// kParts: a CTA's blocks are summed in several parts.
template <uint32_t kTN, uint32_t kBPieces, bool kParts>
__global__ void __launch_bounds__((CutShape<kTN, kBPieces>::kThreads), 1)
UmmaGemmCutKernel(const __grid_constant__ CUtensorMap map_b, const __grid_constant__ UmmaEpilogue ep, uint32_t splits,
                  uint32_t parts) {
  using Sh = CutShape<kTN, kBPieces>;
  constexpr uint32_t kTmemCols = (kParts ? 4 : 2) * Sh::kAccCols;   // two accumulators, and the parts so far
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (SmemAddr(smem_raw) & 1023u)) & 1023u);
  CutBarriers* bars = reinterpret_cast<CutBarriers*>(smem + Sh::kStages * Sh::kStageBytes);

  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t split = ClusterCtaRank();   // (a cluster is one tile's splits)
  const uint32_t tiles_n = (ep.N + kTN - 1) / kTN, tile = blockIdx.x / splits;
  const uint32_t mb = tile / tiles_n, nb = tile - mb * tiles_n;
  const uint32_t m0 = mb * kBlockM, n0 = nb * kTN;
  const uint32_t groups = (ep.src_k + kBlockK - 1) / kBlockK;   // an accumulator each
  const uint32_t g0 = groups * split / splits, g1 = groups * (split + 1) / splits;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < Sh::kStages; ++s) {
      MbarInit(&bars->a_full[s], Sh::kCutWarps);
      MbarInit(&bars->b_full[s], 1);
      MbarInit(&bars->empty[s], 1);
    }
    for (uint32_t b = 0; b < 2; ++b) {
      MbarInit(&bars->tmem_full[b], 1);
      MbarInit(&bars->tmem_empty[b], Sh::kAddWarps);
    }
    bars->abort = 0;
    bars->nonfinite = 0;
    MbarInitFence();
  }
  if (warp == 1) TmemAlloc(&bars->tmem_base, kTmemCols);
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  AwaitPrevious();
  const uint32_t tmem_base = bars->tmem_base;
  auto give_up = [&] { ep.status->wait_timeout = 1; bars->abort = 1; };

  const bool work = warp >= 2;
  const uint32_t wt = threadIdx.x - 64;
  constexpr uint32_t kChunks = kTN / 4;
  const uint32_t rows = kBlockM / splits, r0 = split * rows;   // the rows this CTA stores
  bool ok = true;
  if (warp == 0) {
    // ---- B ----
    if (lane == 0)
      for (uint32_t g = g0, it = 0; g < g1; ++g, ++it) {
        const uint32_t s = it % Sh::kStages, round = it / Sh::kStages;
        if (round > 0 && !MbarWait(&bars->empty[s], (round - 1) & 1)) { give_up(); break; }
        uint8_t* b = smem + s * Sh::kStageBytes + 3 * kPieceBytes;
        MbarExpectTx(&bars->b_full[s], kBPieces * Sh::kBBytes);
#pragma unroll
        for (uint32_t p = 0; p < kBPieces; ++p)
          TmaLoad2D(b + p * Sh::kBBytes, &map_b, &bars->b_full[s], static_cast<int32_t>((p * groups + g) * kBlockK),
                    static_cast<int32_t>(n0));
      }
  } else if (warp == 1) {
    // ---- products: small ones first, for the tensor core truncates toward zero at the accumulator's magnitude ----
    if (ElectOne()) {
      const uint32_t idesc = MakeInstrDesc(kBlockM, kTN);
      for (uint32_t g = g0, it = 0; g < g1; ++g, ++it) {
        const uint32_t s = it % Sh::kStages, parity = (it / Sh::kStages) & 1, buf = it & 1, use = it >> 1;
        if ((use > 0 && !MbarWait(&bars->tmem_empty[buf], (use - 1) & 1)) || !MbarWait(&bars->b_full[s], parity) ||
            !MbarWait(&bars->a_full[s], parity)) {
          give_up();
          break;
        }
        TcFenceAfter();
        const uint32_t acc = tmem_base + buf * Sh::kAccCols, a = SmemAddr(smem + s * Sh::kStageBytes), b = a + 3 * kPieceBytes;
        auto product = [&](uint32_t pa, uint32_t pb, bool first) {
          const uint64_t da = MakeSmemDesc(a + pa * kPieceBytes), db = MakeSmemDesc(b + pb * Sh::kBBytes);
#pragma unroll
          for (uint32_t k = 0; k < 4; ++k) UmmaBf16(acc, da + 2 * k, db + 2 * k, idesc, first && k == 0 ? 0u : 1u);
        };
        if constexpr (kBPieces == 3) {
          product(2, 0, true);
          product(1, 1, false);
          product(0, 2, false);
          product(1, 0, false);
          product(0, 1, false);
          product(0, 0, false);
        } else {
          product(2, 0, true);
          product(1, 0, false);
          product(0, 0, false);
        }
        UmmaCommit(&bars->empty[s]);
        UmmaCommit(&bars->tmem_full[buf]);
      }
    }
    __syncwarp();
  } else {
    // ---- cut, and add: the roles of this warp ----
    auto role = [&](auto cuts, auto adds) {
      constexpr bool kCuts = decltype(cuts)::value, kAdds = decltype(adds)::value;
      const uint32_t quarter = warp & 3, columns = kAdds ? ((warp - Sh::kFirstAdd) >> 2) * Sh::kColsPerWarp : 0;
      const uint32_t t_row = tmem_base + ((quarter * 32) << 16) + columns;
      // The blocks of a part of K are one chain of additions and the parts meet after that, as the piece form's CTAs do
      // where it cuts K more often than this kernel: no chain is longer than there.
      float sum[kAdds ? Sh::kColsPerWarp : 1];
#pragma unroll
      for (uint32_t j = 0; j < (kAdds ? Sh::kColsPerWarp : 1u); ++j) sum[j] = 0.0f;
      [[maybe_unused]] const uint32_t first_part = parts / splits * split;
      [[maybe_unused]] uint32_t part = first_part, part_end = groups * (part + 1) / parts;
      [[maybe_unused]] auto add = [&](uint32_t it) {   // the accumulator of this CTA's group number `it`
        const uint32_t buf = it & 1;
        bool there = MbarWait(&bars->tmem_full[buf], (it >> 1) & 1);
        if (!there && lane == 0) give_up();
        if (bars->abort) there = false;
        there = __all_sync(0xFFFFFFFFu, there);
        TcFenceAfter();
        if (!there) return false;
        constexpr uint32_t kChunk = kTN > 128 ? 8 : 16;   // (the registers of 26 warps hold 48 sums and no more than eight at once)
#pragma unroll
        for (uint32_t c = 0; c < Sh::kColsPerWarp; c += kChunk) {
          uint32_t r[kChunk];
          if constexpr (kChunk == 8) TmemLoad8(t_row + buf * Sh::kAccCols + c, r);
          else TmemLoad16(t_row + buf * Sh::kAccCols + c, r);
          TmemWaitLd();
#pragma unroll
          for (uint32_t j = 0; j < kChunk; ++j) sum[c + j] += __uint_as_float(r[j]);
        }
        TcFenceBefore();
        __syncwarp();
        if (lane == 0) MbarArrive(&bars->tmem_empty[buf]);
        if constexpr (kParts) {
          if (g0 + it + 1 == part_end) {   // the parts so far wait in tensor memory: the registers are full
#pragma unroll
            for (uint32_t c = 0; c < Sh::kColsPerWarp; c += 16) {
              uint32_t r[16];
              if (part > first_part) {
                TmemLoad16(t_row + 2 * Sh::kAccCols + c, r);
                TmemWaitLd();
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j) sum[c + j] = __uint_as_float(r[j]) + sum[c + j];
              }
              if (part_end < g1) {
#pragma unroll
                for (uint32_t j = 0; j < 16; ++j) {
                  r[j] = __float_as_uint(sum[c + j]);
                  sum[c + j] = 0.0f;
                }
                TmemStore16(t_row + 2 * Sh::kAccCols + c, r);
              }
            }
            TmemWaitSt();
            ++part;
            part_end = groups * (part + 1) / parts;
          }
        }
        return true;
      };
      // Cut block after block; where the same warps add, the one before while the products of this one run.
      [[maybe_unused]] auto walk = [&](auto loads) {
        constexpr Loads kLoads = decltype(loads)::value;
        CutRegs<Sh::kCutWarps, kLoads> f;
        FetchBlock<kLoads>(&f, ep, m0, g0);
        for (uint32_t g = g0, it = 0; g < g1 && ok; ++g, ++it) {
          const uint32_t s = it % Sh::kStages, round = it / Sh::kStages;
          bool free = round == 0 || MbarWait(&bars->empty[s], (round - 1) & 1);
          if (!free && lane == 0) give_up();
          if (bars->abort) free = false;
          if (!(ok = __all_sync(0xFFFFFFFFu, free))) break;
          StoreBlock(smem + s * Sh::kStageBytes, f);
          if (g + 1 < g1) FetchBlock<kLoads>(&f, ep, m0, g + 1);
          FenceProxyAsync();
          __syncwarp();
          if (lane == 0) MbarArrive(&bars->a_full[s]);
          if constexpr (kAdds)
            if (it > 0) ok = add(it - 1);
        }
      };
      if constexpr (kCuts) {
        const bool aligned = (ep.src_k & 3u) == 0 && ((reinterpret_cast<uintptr_t>(ep.src_a) | reinterpret_cast<uintptr_t>(ep.src_a_scale)) & 15) == 0;
        constexpr Loads kWithScale = Sh::kApart ? Loads::kScaled : Loads::kAny;   // (an f32 weight has no scales)
        if (aligned && !ep.src_a_scale) walk(std::integral_constant<Loads, Loads::kPlain>{});
        else if (aligned && kWithScale == Loads::kScaled) walk(std::integral_constant<Loads, kWithScale>{});
        else walk(std::integral_constant<Loads, Loads::kAny>{});
        if constexpr (kAdds)
          if (ok && g1 > g0) ok = add(g1 - g0 - 1);
      } else {
        for (uint32_t it = 0; it < g1 - g0 && ok; ++it) ok = add(it);
      }
      if constexpr (kAdds) {
        if (ok) {
          // All products are complete, so the ring is free: the tile goes there as [128][kTN] f32, 16-byte chunks XOR-ed
          // with the row so that neither side conflicts.
          if (!AllFinite(sum)) bars->nonfinite = 1;
          float* dump = reinterpret_cast<float*>(smem) + (quarter * 32 + lane) * kTN;
#pragma unroll
          for (uint32_t q = 0; q < Sh::kColsPerWarp / 4; ++q)
            *reinterpret_cast<float4*>(dump + (((columns >> 2) + q) ^ (lane & 7u)) * 4) =
                make_float4(sum[4 * q], sum[4 * q + 1], sum[4 * q + 2], sum[4 * q + 3]);
        }
        TcFenceBefore();
      }
    };
    if constexpr (!Sh::kApart) {
      role(std::true_type{}, std::true_type{});
    } else {
      if (warp < Sh::kFirstAdd) role(std::true_type{}, std::false_type{});
      else role(std::false_type{}, std::true_type{});
    }
  }
  __syncwarp();   // (one lane of the loading and of the issuing warp has walked the blocks: the barriers want whole warps)
  if (splits > 1) ClusterSync();
  else if (work) asm volatile("bar.sync 1, %0;" ::"n"(Sh::kWorkThreads) : "memory");
  if (bars->abort) ok = false;
  if (work && ok) {
    const uint32_t dump = SmemAddr(smem);
    auto element = [&](uint32_t lr, uint32_t chunk) {
      const uint32_t off = (lr * kTN + (chunk ^ (lr & 7u)) * 4) * 4;
      if (splits == 1) return *reinterpret_cast<const float4*>(smem + off);
      float4 acc = LoadClusterF4(MapToCta(dump + off, 0));
      for (uint32_t p = 1; p < splits; ++p) {
        const float4 v = LoadClusterF4(MapToCta(dump + off, p));
        acc = make_float4(acc.x + v.x, acc.y + v.y, acc.z + v.z, acc.w + v.w);
      }
      return acc;
    };
    bool remake = false;   // (an element's splits lie in several CTAs)
    for (uint32_t p = 0; p < splits; ++p)
      remake = remake || (splits == 1 ? bars->nonfinite : LoadClusterU32(MapToCta(SmemAddr(const_cast<uint32_t*>(&bars->nonfinite)), p))) != 0;
    const bool ragged = (ep.N & 3u) != 0, plain = IsPlainStore(ep);
    const bool sum_only = IsSum(ep);
    if (remake || ragged || !(plain || sum_only)) {
#pragma unroll 1
      for (uint32_t i = wt; i < rows * kChunks; i += Sh::kWorkThreads) {
        const uint32_t lr = r0 + i / kChunks, chunk = i % kChunks, row = m0 + lr, n = n0 + chunk * 4;
        if (row >= ep.M || n >= ep.N) continue;
        const float4 acc = element(lr, chunk);
        if (remake) { StoreRemade(ep, row, n, acc); continue; }
        if (ragged) { EpilogueStoreRagged(ep, row, n, acc, false); continue; }
        float4 scale = make_float4(ep.alpha, ep.alpha, ep.alpha, ep.alpha), bias = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ep.col_scale) scale = __ldg(reinterpret_cast<const float4*>(ep.col_scale + n));
        if (ep.bias) bias = __ldg(reinterpret_cast<const float4*>(ep.bias + n));
        EpilogueStore(ep, static_cast<size_t>(row) * ep.N + n, n, acc, scale, bias);
      }
    } else {   // the frequent forms: a few elements per thread at a time, what they need of global memory asked for first
      constexpr uint32_t kUnroll = kTN > 128 ? 2 : 4;
      for (uint32_t i0 = wt; i0 < rows * kChunks; i0 += Sh::kWorkThreads * kUnroll) {
        float4 side[kUnroll], scale[kUnroll];
        auto there = [&](uint32_t u, uint32_t* lr, uint32_t* chunk) {
          const uint32_t i = i0 + u * Sh::kWorkThreads;
          *lr = r0 + i / kChunks;
          *chunk = i % kChunks;
          return i < rows * kChunks && m0 + *lr < ep.M && n0 + *chunk * 4 < ep.N;
        };
#pragma unroll
        for (uint32_t u = 0; u < kUnroll; ++u) {
          uint32_t lr, chunk;
          scale[u] = make_float4(ep.alpha, ep.alpha, ep.alpha, ep.alpha);
          if (!there(u, &lr, &chunk)) continue;
          if (ep.col_scale) scale[u] = __ldg(reinterpret_cast<const float4*>(ep.col_scale + n0 + chunk * 4));
          if (!plain) side[u] = __ldg(reinterpret_cast<const float4*>(ep.addend + static_cast<size_t>(m0 + lr) * ep.N + n0 + chunk * 4));
        }
#pragma unroll
        for (uint32_t u = 0; u < kUnroll; ++u) {
          uint32_t lr, chunk;
          if (!there(u, &lr, &chunk)) continue;
          const uint32_t n = n0 + chunk * 4;
          const float4 acc = element(lr, chunk);
          const size_t at = static_cast<size_t>(m0 + lr) * ep.N + n;
          if (plain) {
            EpilogueStorePlain(ep, at, acc, scale[u]);
          } else {
            const float4 bias = ep.bias ? __ldg(reinterpret_cast<const float4*>(ep.bias + n)) : make_float4(0.f, 0.f, 0.f, 0.f);
            EpilogueStoreSum(ep, at, acc, scale[u], bias, side[u]);
          }
        }
      }
    }
  }

  TcFenceBefore();
  __syncthreads();
  if (bars->abort) DrainDelay();
  if (splits > 1) ClusterSync();   // no CTA leaves while another may still read its memories
  if (warp == 1) {
    TcFenceAfter();
    TmemFree(tmem_base, kTmemCols);
  }
}

template <uint32_t kTN, uint32_t kBPieces, bool kParts = false>
cudaError_t Launch(const UmmaCutPlan& plan, const CUtensorMap& map_b, const UmmaEpilogue& ep, cudaStream_t s) {
  auto kernel = UmmaGemmCutKernel<kTN, kBPieces, kParts>;
  constexpr size_t kSmem = CutShape<kTN, kBPieces>::kSmem;
  static std::atomic<bool> configured[64] = {};   // (a per-device setting of the function)
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
    if (cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem)); e != cudaSuccess)
      return e;
    if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
  }
  return Next(kernel, plan.grid, CutShape<kTN, kBPieces>::kThreads, kSmem, s, plan.splits)(map_b, ep, plan.splits, plan.parts);
}

}  // namespace

UmmaCutPlan UmmaPlanCut(uint32_t M, uint32_t N, uint32_t groups, bool exact_b, uint32_t sms) {
  // One round of CTAs only, and for an f32 weight at most sixteen blocks of 64 k: every further column tile cuts A again, and
  // the working warps, which take about 1 us for a block, fall behind the piece form's tensor time.  Measured on a B200, the
  // piece form's kernel (+ its cut of A) / this, us, f32 weights: 4096 x 256 x 256 13.3 (+2.5) / 8.9, 1024 x 256 x 256 8.0 (+1.6) / 7.8,
  // 600 x 512 x 512 11.3 (+1.8) / 10.6, 128 x 1024 x 1024 13.5 (+1.4) / 10.5, 300 x 5000 x 256 13.9 (+1.1) / 11.6, 4096 x 256 x 1024 20.3 (+5.8) /
  // 18.0, 4096 x 512 x 256 14.1 (+2.5) / 11.7; past the line 4096 x 768 x 256 16.1 (+2.8) / 21.9, 4096 x 1024 x 256 17.3 (+2.9) / 22.2, 4096 x 4096 x
  // 256 52.4 (+4.3) / 75.9; int8 weights: 4096 x 768 x 768 23.8 (+3.7) / 20.4, 4096 x 768 x 3072 64.5 (+20.7) / 56.6, 2048 x 512 x 2048 21.4 (+5.7) /
  // 21.8; past it 4096 x 3072 x 768 65.6 (+4.2) / 78.4, 2048 x 2304 x 768 24.4 (+3.4) / 31.9, 4096 x 1024 x 256 14.3 (+2.5) / 18.5.  Drawn when a
  // block took longer, the line is short of where both meet now: f32 2048 x 512 x 2048 28.9 (+6.8) / 27.4, and of exact weights in two
  // full rounds 4096 x 1536 x 768 44.8 (+4.0) / 39.3, 8192 x 768 x 768 44.7 (+9.2) / 39.3.
  UmmaCutPlan best;
  if (!exact_b && groups > 16) return best;
  double least = 1e30;
  const uint32_t tiles_m = (M + kBlockM - 1) / kBlockM;
  for (uint32_t tn : {64u, 128u, 192u}) {
    if (!exact_b && tn > 128) continue;   // (a block of three 192-wide pieces leaves room for one stage)
    for (uint32_t splits = 1; splits <= 4 && splits <= groups; splits *= 2) {
      const uint64_t ctas = static_cast<uint64_t>(tiles_m) * ((N + tn - 1) / tn) * splits;
      if (ctas > (splits <= 2 ? sms : sms * 9 / 10)) continue;   // clusters of four do not fill every GPC
      const double group = exact_b ? 1.1 + 0.001 * tn : 0.9 + 0.004 * tn;
      const double t = group * ((groups + splits - 1) / splits) + 0.015 * tn / splits + (splits > 1 ? 2.0 : 0.0);
      if (t < least) {
        least = t;
        best = {tn, splits, static_cast<uint32_t>(ctas)};
      }
    }
  }
  return best;
}

cudaError_t UmmaCutLaunch(const UmmaCutPlan& plan, bool exact_b, const CUtensorMap& map_b, const UmmaEpilogue& ep, cudaStream_t s) {
  if (plan.parts > plan.splits && plan.tn <= 128) {   // (192-wide tiles leave no tensor memory for it, and are cut at least as often)
    if (exact_b) return plan.tn == 64 ? Launch<64, 1, true>(plan, map_b, ep, s) : Launch<128, 1, true>(plan, map_b, ep, s);
    return plan.tn == 64 ? Launch<64, 3, true>(plan, map_b, ep, s) : Launch<128, 3, true>(plan, map_b, ep, s);
  }
  if (exact_b) {
    switch (plan.tn) {
      case 64: return Launch<64, 1>(plan, map_b, ep, s);
      case 128: return Launch<128, 1>(plan, map_b, ep, s);
      default: return Launch<192, 1>(plan, map_b, ep, s);
    }
  }
  return plan.tn == 64 ? Launch<64, 3>(plan, map_b, ep, s) : Launch<128, 3>(plan, map_b, ep, s);
}

}  // namespace see::k
