// The tensor-core GEMM for frozen-weight products that carry the relaxed
// permission (reference: source/plan/instruction.h:356-382; the reference's own
// relaxed kernels are runtime/executor/metal_backend.mm:1385-1449):
//
//     C[M,N] = epilogue( A_bf16[M,K] . B_bf16[N,K]^T )       f32 accumulate
//
// Blackwell-native: operands arrive by TMA (cp.async.bulk.tensor, 128-byte
// swizzle) into a shared-memory ring, one elected thread issues tcgen05.mma
// (kind::f16) with the accumulator in tensor memory, tcgen05.commit hands ring
// slots back to the producer, and the epilogue warps read the accumulator with
// tcgen05.ld and apply scale / addend / bias / activation on the way to HBM.
// Two kernels: UmmaGemmTileKernel for products of about one tile per SM, whose
// time is latency and operand delivery, and UmmaGemmPersistentKernel for those
// with several tiles per SM.  The operands may also be bf16 pieces side by side
// (UmmaEpilogue::seg_blocks), which makes either an f32-accurate product: 64 k of
// piece products per accumulator, the accumulators added in registers.
//
// Every wait on an mbarrier is bounded; a wait that runs out raises
// DeviceStatus::wait_timeout, the CTA stops issuing work, frees its tensor
// memory and returns, and the host reports the condition at its next flush.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <type_traits>
#include <utility>

#include "act_expr.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "shadow.cuh"
#include "umma_device.cuh"
#include "umma_epilogue.cuh"
#include "umma_kernel.h"

namespace see::k {

namespace {

constexpr uint32_t kBlockM = umma_cfg::kBlockM;
constexpr uint32_t kBlockN = umma_cfg::kBlockN;
constexpr uint32_t kBlockK = umma_cfg::kBlockK;   // 64 bf16 = one 128-byte swizzle row
constexpr uint32_t kUmmaK = 16;
constexpr uint32_t kATileBytes = kBlockM * kBlockK * 2;

using namespace umma_epi;
using namespace umma_dev;   // mbarriers with bounded waits, TMA loads, descriptors, MMA issue, TMEM loads

// A wait for a part of the CTA that may be in there: as bounded as the others, only longer.
template <bool kSeg>
__device__ __forceinline__ bool PartnerWait(uint64_t* bar, uint32_t parity) {
  for (int i = 0; i < (kSeg ? 64 : 1); ++i)
    if (MbarWait(bar, parity)) return true;
  return false;
}

// What a launch's accumulators are.
//   kPlain  one per tile (of one product, or of each of several side by side)
//   kPieces piece products (UmmaEpilogue::seg_blocks): one per block of K
//   kChain  the products of a chain: one each
enum class Sums { kPlain, kPieces, kChain };

// Element offsets along K of reduction block kb's tiles of A and B of a product.
struct BlockAt { int32_t a, b; bool aux; };
__device__ __forceinline__ BlockAt BlockCoord(const UmmaEpilogue& ep, uint32_t kb, uint32_t main_blocks) {
  if (kb >= main_blocks) {
    const int32_t x = static_cast<int32_t>((kb - main_blocks) * kBlockK);
    return {x, x, true};
  }
  if (ep.seg_blocks == 0) return {static_cast<int32_t>(kb * kBlockK), static_cast<int32_t>(kb * kBlockK), false};
  const uint32_t w = kb / ep.segs, seg = kb - w * ep.segs;
  return {static_cast<int32_t>((((ep.seg_a >> (4 * seg)) & 15u) * ep.seg_blocks + w) * kBlockK),
          static_cast<int32_t>((((ep.seg_b >> (4 * seg)) & 15u) * ep.seg_blocks + w) * kBlockK), false};
}
// Blocks of a product's whole reduction.
__device__ __forceinline__ uint32_t ReductionBlocks(const UmmaEpilogue& ep, uint32_t main_blocks, uint32_t product) {
  return main_blocks + ep.product[product].aux_k_blocks;
}

// ---- about one tile per SM --------------------------------------------------------------
// Such a product (a data-parallel rank's 4096 rows, a few hundred rows of a short fine-tune, a
// 256-wide f32 decoder) is bound by operand latency and by the fixed cost of a launch, not by the
// tensor pipe.  Hence
//  * a ring as deep as shared memory is large (4 to 8 stages): the tile's epilogue has nothing to
//    overlap with, so it takes the ring's memory for its staging;
//  * a tile width from 64 to 256 and a reduction cut over `splits` CTAs of a cluster, so that the
//    grid comes near 148 CTAs whatever the shape.  The partial tiles meet in distributed shared
//    memory: each CTA dumps its accumulator, and after a cluster barrier each takes 1 / splits of
//    the rows, adds the partials in split order (a fixed order) and stores them;
//  * the second operand of the epilogue (an addend, an activation's input) asked into L2 at the
//    start: from HBM, a round trip per group of rows was 12-17 us of such a launch.
// CTA pairs (cta_group::2, a third fewer operand bytes) were slower here at every shape: the two
// CTAs' operands must both be there before either SM's tensor core starts.
// Measured on a B200 (weights from HBM, plain epilogue), one-tile kernel of three stages or the
// persistent kernel / this one, us: 4096 x 256 x 1536 16.0 / 10.8; 4096 x 256 x 6144 42 / 18.9;
// 4096 x 768 x 3072 28.5 / 22.0; 600 x 512 x 2048 18.7 / 9.2; 600 x 512 x 8000 66 / 16.3.
constexpr uint32_t kTThreads = 320;      // warp 0 TMA, warp 1 MMA, eight epilogue warps
constexpr uint32_t kTEpiThreads = 256;
constexpr uint32_t kTMaxStages = 8;
template <uint32_t kTN>
struct TTile {
  static constexpr uint32_t kStageBytes = kATileBytes + kTN * kBlockK * 2;
  static constexpr uint32_t kFit = 208u * 1024u / kStageBytes;
  static constexpr uint32_t kStages = kFit < kTMaxStages ? kFit : kTMaxStages;
  static constexpr uint32_t kTmemCols = kTN <= 64 ? 64 : (kTN <= 128 ? 128 : 256);
  static_assert(kStages * kStageBytes >= kBlockM * kTN * 4, "the epilogue stages the whole tile in the ring");
};

struct __align__(8) TBarriers {
  uint64_t full[kTMaxStages];
  uint64_t empty[kTMaxStages];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];   // where accumulators take turns (piece products, wide chains)
  uint32_t tmem_base;
  volatile uint32_t abort;      // set by a role whose wait ran out; the epilogue then stores nothing
  volatile uint32_t nonfinite;  // piece products: some sum of this CTA is not finite
};

// A chain (kChain) is the sum of its products as separate launches would leave it, bit for bit: every product has an
// accumulator of its own, cut over the same splits, and their scaled sums meet in f32 in the products' order.  (One
// accumulator for all truncates at the sum's magnitude: rms error 3.2e-6 at K = 3072 where 768 at a time leave 7.3e-7.)
// Up to 128 columns all accumulators stay in tensor memory until the end (3 x 128 of 512 columns); wider tiles, never cut,
// take turns in two buffers and are added in registers.
template <uint32_t kTN, Sums kSums>
__global__ void __launch_bounds__(kTThreads, 1)
UmmaGemmTileKernel(const __grid_constant__ UmmaMaps maps, const __grid_constant__ UmmaEpilogue ep, uint32_t splits) {
  using T = TTile<kTN>;
  constexpr bool kSeg = kSums == Sums::kPieces, kChain = kSums == Sums::kChain;
  constexpr bool kResident = kChain && kTN <= 128;       // the accumulators lie side by side until the end
  constexpr bool kTurns = (kSeg || kChain) && !kResident; // ... take turns and are added in registers
  static_assert(!kResident || T::kStages * T::kStageBytes >= kUmmaProducts * kBlockM * kTN * 4, "a chain's tiles are staged together");
  constexpr uint32_t kStages = T::kStages, kStageBytes = T::kStageBytes;
  extern __shared__ uint8_t smem_raw[];
  // 1024-byte alignment: the swizzle pattern and the descriptors' base offset assume it.
  uint8_t* smem = smem_raw + ((1024u - (SmemAddr(smem_raw) & 1023u)) & 1023u);
  TBarriers* bars = reinterpret_cast<TBarriers*>(smem + kStages * kStageBytes);

  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t split = ClusterCtaRank();   // (a cluster is one tile's splits)
  const uint32_t tiles_n = (ep.N + kTN - 1) / kTN, all_n = kSums == Sums::kPlain ? tiles_n * ep.products : tiles_n, tile = blockIdx.x / splits;
  const uint32_t mb = tile / all_n, product = kSums == Sums::kPlain ? tile % all_n / tiles_n : 0, nb = tile % all_n % tiles_n;
  const uint32_t m0 = mb * kBlockM, n0 = nb * kTN;
  // The reduction runs over the main operands' K and then over aux_k_blocks more
  // 64-wide blocks taken from the second pair of maps (a low-rank term T . B'^T
  // accumulated into the same tile; see UmmaEpilogue::Product).
  const uint32_t main_blocks = (ep.K + kBlockK - 1) / kBlockK;
  // This CTA's accumulators: of one product, of each block of K of piece products, of each product of a chain.
  const uint32_t part0 = kSeg ? ep.seg_blocks * split / splits : 0, part1 = kSeg ? ep.seg_blocks * (split + 1) / splits : 0;
  const uint32_t groups = kSeg ? part1 - part0 : (kChain ? ep.products : 1u);
  struct Blocks { uint32_t product, begin, end; };
  auto blocks_of = [&](uint32_t g) -> Blocks {
    if (kSeg) return {0, (part0 + g) * ep.segs, (part0 + g + 1) * ep.segs};
    const uint32_t p = kChain ? g : product, all = ReductionBlocks(ep, main_blocks, p);
    return {p, all * split / splits, all * (split + 1) / splits};
  };
  constexpr uint32_t kTmemCols = kTurns ? 2 * T::kTmemCols : (kResident ? 4 * T::kTmemCols : T::kTmemCols);

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < kStages; ++s) {
      MbarInit(&bars->full[s], 1);
      MbarInit(&bars->empty[s], 1);
    }
    for (uint32_t b = 0; b < 2; ++b) {
      MbarInit(&bars->tmem_full[b], 1);
      MbarInit(&bars->tmem_empty[b], kTEpiThreads / 32);
    }
    bars->abort = 0;
    bars->nonfinite = 0;
    MbarInitFence();
  }
  if (warp == 1) {
    TmemAlloc(&bars->tmem_base, kTmemCols);
  }
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  AwaitPrevious();
  const uint32_t tmem_base = bars->tmem_base;

  if (warp == 0) {
    // ---- TMA producer ----
    if (lane == 0) {
      bool going = true;
      for (uint32_t g = 0, it = 0; g < groups && going; ++g) {
        const Blocks part = blocks_of(g);
        for (uint32_t kb = part.begin; kb < part.end; ++kb, ++it) {
          const uint32_t s = it % kStages, round = it / kStages;
          if (round > 0 && !MbarWait(&bars->empty[s], (round - 1) & 1)) {
            ep.status->wait_timeout = 1;
            bars->abort = 1;
            going = false;
            break;
          }
          uint8_t* a_dst = smem + s * kStageBytes;
          const BlockAt at = BlockCoord(ep, kb, main_blocks);
          const CUtensorMap* ma = at.aux ? &maps.a2[part.product] : &maps.a[part.product];
          const CUtensorMap* mb_ = at.aux ? &maps.b2[part.product] : &maps.b[part.product];
          MbarExpectTx(&bars->full[s], kStageBytes);
          TmaLoad2D(a_dst, ma, &bars->full[s], at.a, static_cast<int32_t>(m0));
          TmaLoad2D(a_dst + kATileBytes, mb_, &bars->full[s], at.b, static_cast<int32_t>(n0));
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer ----
    if (ElectOne()) {
      const uint32_t idesc = MakeInstrDesc(kBlockM, kTN);
      bool going = true;
      for (uint32_t g = 0, it = 0; g < groups && going; ++g) {
        const uint32_t buf = kTurns ? g & 1 : (kResident ? g : 0), use = g >> 1;
        if (kTurns && use > 0 && !MbarWait(&bars->tmem_empty[buf], (use - 1) & 1)) {
          ep.status->wait_timeout = 1;
          bars->abort = 1;
          break;
        }
        const uint32_t acc = tmem_base + buf * T::kTmemCols;
        const Blocks part = blocks_of(g);
        for (uint32_t b = 0; b < part.end - part.begin; ++b, ++it) {
          const uint32_t s = it % kStages, round = it / kStages;
          if (!MbarWait(&bars->full[s], round & 1)) {
            ep.status->wait_timeout = 1;
            bars->abort = 1;
            going = false;
            break;
          }
          TcFenceAfter();
          const uint32_t a_addr = SmemAddr(smem + s * kStageBytes);
          const uint64_t desc_a = MakeSmemDesc(a_addr), desc_b = MakeSmemDesc(a_addr + kATileBytes);
#pragma unroll
          for (uint32_t k = 0; k < kBlockK / kUmmaK; ++k) {
            // advance 16 bf16 = 32 bytes inside the 128-byte swizzle row: +2 in >>4 units
            UmmaBf16(acc, desc_a + 2 * k, desc_b + 2 * k, idesc, (b | k) != 0 ? 1u : 0u);
          }
          UmmaCommit(&bars->empty[s]);      // the slot is free once these MMAs have read it
        }
        // accumulator complete (or abandoned on timeout); of resident ones the last, with all before it
        if (kTurns) UmmaCommit(&bars->tmem_full[buf]);
        else if (g + 1 == groups || !going) UmmaCommit(&bars->tmem_full[0]);
      }
    }
  }
  __syncwarp();
  const bool epilogue = warp >= 2;
  const uint32_t et = threadIdx.x - 64;   // thread of the epilogue
  const float* side_ptr = ep.fuse_mode == kFuseActBwd ? ep.fuse_x : ep.addend;
  const bool ragged = (ep.N & 3u) != 0;
  constexpr uint32_t kChunks = kTN / 4;
  const uint32_t rows = kBlockM / splits, r0 = split * rows;   // the rows this CTA stores
  bool ok = true;
  if (epilogue) {
    // The second operand of the epilogue is asked into L2 while the products run.
    if (side_ptr && !ragged)
      for (uint32_t i = et; i < rows * (kTN / 32); i += kTEpiThreads) {
        const uint32_t row = m0 + r0 + i / (kTN / 32), n = n0 + i % (kTN / 32) * 32;
        if (row < ep.M && n < ep.N)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(side_ptr + static_cast<size_t>(row) * ep.N + n));
      }
    const uint32_t quarter = warp & 3, columns = ((warp - 2) >> 2) * (kTN / 2);
    const uint32_t t_row = tmem_base + ((quarter * 32) << 16) + columns;
    auto await = [&](uint32_t buf, uint32_t parity) {
      bool there = MbarWait(&bars->tmem_full[buf], parity);
      if (!there && lane == 0) ep.status->wait_timeout = 1;
      if (bars->abort) there = false;
      there = __all_sync(0xFFFFFFFFu, there);
      TcFenceAfter();
      return there;
    };
    // Accumulators that take turns are added with f32's rounding while the next one's products run.
    [[maybe_unused]] float sum[kTurns ? kTN / 2 : 1];
    if constexpr (kTurns) {
#pragma unroll
      for (uint32_t j = 0; j < kTN / 2; ++j) sum[j] = kChain ? -0.0f : 0.0f;   // (-0 + x is x, -0 included)
      for (uint32_t g = 0; g < groups && ok; ++g) {
        const uint32_t buf = g & 1;
        if (!(ok = await(buf, (g >> 1) & 1))) break;
#pragma unroll
        for (uint32_t c0 = 0; c0 < kTN / 2; c0 += 16) {
          uint32_t r[16];
          TmemLoad16(t_row + buf * T::kTmemCols + c0, r);
          TmemWaitLd();
#pragma unroll
          for (uint32_t j = 0; j < 16; ++j) sum[c0 + j] += kChain ? __uint_as_float(r[j]) * ep.alpha : __uint_as_float(r[j]);
        }
        TcFenceBefore();
        __syncwarp();
        if (lane == 0) MbarArrive(&bars->tmem_empty[buf]);
      }
    } else {
      ok = await(0, 0);
    }
    if (ok) {
      // The accumulator arrives one row per thread; HBM wants whole rows.  All MMAs are complete, so
      // the ring is free: the tile goes there as [128][kTN] f32, 16-byte chunks XOR-ed with the
      // row so that neither side conflicts.
      float* dump = reinterpret_cast<float*>(smem) + (quarter * 32 + lane) * kTN;
      if constexpr (kTurns) {
        if (kSeg && !AllFinite(sum)) bars->nonfinite = 1;
#pragma unroll
        for (uint32_t q = 0; q < kTN / 8; ++q)
          *reinterpret_cast<float4*>(dump + (((columns >> 2) + q) ^ (lane & 7u)) * 4) =
              make_float4(sum[4 * q], sum[4 * q + 1], sum[4 * q + 2], sum[4 * q + 3]);
      } else {
        for (uint32_t g = 0; g < (kResident ? groups : 1u); ++g) {   // (a chain's tiles one behind the other)
#pragma unroll 1
          for (uint32_t c0 = 0; c0 < kTN / 2; c0 += 32) {
            uint32_t r[32];
            TmemLoad32(t_row + g * T::kTmemCols + c0, r);
            TmemWaitLd();
#pragma unroll
            for (uint32_t q = 0; q < 8; ++q)
              *reinterpret_cast<uint4*>(dump + g * (kBlockM * kTN) + ((((columns + c0) >> 2) + q) ^ (lane & 7u)) * 4) =
                  make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
          }
        }
      }
    }
    TcFenceBefore();
  }
  if (splits > 1) ClusterSync();
  else if (epilogue) asm volatile("bar.sync 1, %0;" ::"n"(kTEpiThreads) : "memory");
  if (epilogue && ok) {
    const uint32_t dump = SmemAddr(smem);
    // The tile's element of row r0 + lr, chunk: this CTA's, or the sum of the splits' partials.
    auto partials = [&](uint32_t off) {
      if (splits == 1) return *reinterpret_cast<const float4*>(smem + off);
      float4 acc = LoadClusterF4(MapToCta(dump + off, 0));
      for (uint32_t p = 1; p < splits; ++p) {
        const float4 v = LoadClusterF4(MapToCta(dump + off, p));
        acc = make_float4(acc.x + v.x, acc.y + v.y, acc.z + v.z, acc.w + v.w);
      }
      return acc;
    };
    auto element = [&](uint32_t lr, uint32_t chunk) {
      const uint32_t off = (lr * kTN + (chunk ^ (lr & 7u)) * 4) * 4;
      float4 acc = partials(off);
      if constexpr (kResident) {   // the products' scaled sums, in order
        const float s = ep.alpha;
        acc = make_float4(acc.x * s, acc.y * s, acc.z * s, acc.w * s);
        for (uint32_t g = 1; g < groups; ++g) {
          const float4 v = partials(off + g * (kBlockM * kTN * 4));
          acc = make_float4(acc.x + v.x * s, acc.y + v.y * s, acc.z + v.z * s, acc.w + v.w * s);
        }
      }
      return acc;
    };
    // Four elements per thread at a time, their operands loaded before the first is stored.  `store` is one form of
    // the epilogue, chosen once: tests per element would cost more than the stores.
    constexpr uint32_t kUnroll = 4;
    const bool side_by_side = kSums == Sums::kPlain && ep.products > 1;
    const float alpha = kChain ? 1.0f : (side_by_side ? ep.product[product].alpha : ep.alpha);
    const float* col_scale = side_by_side ? ep.product[product].col_scale : ep.col_scale;
    uint16_t* pack_dst = side_by_side ? ep.product[product].pack_dst : ep.pack_dst;
    auto each = [&](auto has_side, auto store) {
      for (uint32_t i0 = et; i0 < rows * kChunks; i0 += kTEpiThreads * kUnroll) {
        float4 acc[kUnroll], side[kUnroll];
#pragma unroll
        for (uint32_t u = 0; u < kUnroll; ++u) {
          const uint32_t i = i0 + u * kTEpiThreads, lr = r0 + i / kChunks, chunk = i % kChunks;
          const uint32_t row = m0 + lr, n = n0 + chunk * 4;
          if (i >= rows * kChunks || row >= ep.M || n >= ep.N) continue;
          if constexpr (decltype(has_side)::value)
            side[u] = __ldg(reinterpret_cast<const float4*>(side_ptr + static_cast<size_t>(row) * ep.N + n));
          acc[u] = element(lr, chunk);
        }
#pragma unroll
        for (uint32_t u = 0; u < kUnroll; ++u) {
          const uint32_t i = i0 + u * kTEpiThreads, lr = r0 + i / kChunks, chunk = i % kChunks;
          const uint32_t row = m0 + lr, n = n0 + chunk * 4;
          if (i >= rows * kChunks || row >= ep.M || n >= ep.N) continue;
          float4 scale = make_float4(alpha, alpha, alpha, alpha);
          if (col_scale) scale = __ldg(reinterpret_cast<const float4*>(col_scale + n));
          store(static_cast<size_t>(row) * ep.N + n, row, n, acc[u], scale, side[u]);
        }
      }
    };
    const float4 one = make_float4(1.f, 1.f, 1.f, 1.f), none = make_float4(0.f, 0.f, 0.f, 0.f);
    auto bias_at = [&](uint32_t n) { return ep.bias ? __ldg(reinterpret_cast<const float4*>(ep.bias + n)) : none; };
    using Side = std::true_type;
    using NoSide = std::false_type;
    bool remake = false;   // (an element's splits lie in several CTAs)
    if constexpr (kSeg)
      for (uint32_t p = 0; p < splits; ++p)
        remake = remake || (splits == 1 ? bars->nonfinite : LoadClusterU32(MapToCta(SmemAddr(const_cast<uint32_t*>(&bars->nonfinite)), p))) != 0;
    if (kChain) {   // (stored as it is: nothing else is part of a chain)
      each(NoSide{}, [&](size_t at, uint32_t, uint32_t, const float4& acc, const float4& scale, const float4&) {
        EpilogueStorePlain(ep, at, acc, scale);
      });
    } else if (remake) {
      for (uint32_t i = et; i < rows * kChunks; i += kTEpiThreads) {
        const uint32_t lr = r0 + i / kChunks, row = m0 + lr, n = n0 + i % kChunks * 4;
        if (row < ep.M && n < ep.N) StoreRemade(ep, row, n, element(lr, i % kChunks));
      }
    } else if (ragged) {
      for (uint32_t i = et; i < rows * kChunks; i += kTEpiThreads) {
        const uint32_t lr = r0 + i / kChunks, row = m0 + lr, n = n0 + i % kChunks * 4;
        if (row < ep.M && n < ep.N) EpilogueStoreRagged(ep, row, n, element(lr, i % kChunks), false);
      }
    } else if (IsPlainStore(ep)) {
      each(NoSide{}, [&](size_t at, uint32_t, uint32_t, const float4& acc, const float4& scale, const float4&) {
        EpilogueStorePlain(ep, at, acc, scale);
      });
    } else if (IsAddendOnly(ep)) {
      each(Side{}, [&](size_t at, uint32_t, uint32_t, const float4& acc, const float4& scale, const float4& side) {
        EpilogueStoreAddend(ep, at, acc, scale, side);
      });
    } else if (IsCopyOnly(ep)) {
      each(NoSide{}, [&](size_t at, uint32_t, uint32_t, const float4& acc, const float4& scale, const float4&) {
        EpilogueStoreCopy(pack_dst, at, acc, scale);
      });
    } else if (IsBiasGeluOnly(ep) && !ep.shadow_k_scale) {
      each(NoSide{}, [&](size_t at, uint32_t, uint32_t n, const float4& acc, const float4& scale, const float4&) {
        EpilogueStoreBiasGelu(ep, at, acc, scale, bias_at(n), one);
      });
    } else if (kSeg && IsBiasStored(ep, kActNone)) {
      each(NoSide{}, [&](size_t at, uint32_t, uint32_t n, const float4& acc, const float4& scale, const float4&) {
        EpilogueStoreBias<kActNone>(ep, at, acc, scale, bias_at(n));
      });
    } else if (kSeg && IsBiasStored(ep, kActGelu)) {
      each(NoSide{}, [&](size_t at, uint32_t, uint32_t n, const float4& acc, const float4& scale, const float4&) {
        EpilogueStoreBias<kActGelu>(ep, at, acc, scale, bias_at(n));
      });
    } else if (kSeg && IsSum(ep)) {
      each(Side{}, [&](size_t at, uint32_t, uint32_t n, const float4& acc, const float4& scale, const float4& side) {
        EpilogueStoreSum(ep, at, acc, scale, bias_at(n), side);
      });
    } else if (IsGeluGradOnly(ep) && !ep.shadow_k_scale) {
      each(Side{}, [&](size_t at, uint32_t, uint32_t, const float4& acc, const float4& scale, const float4& side) {
        EpilogueStoreGeluGrad(ep, at, acc, scale, one, side);
      });
    } else if (side_ptr) {
      each(Side{}, [&](size_t at, uint32_t, uint32_t n, const float4& acc, const float4& scale, const float4& side) {
        EpilogueStore(ep, at, n, acc, scale, bias_at(n), false, one, true, side);
      });
    } else {
      each(NoSide{}, [&](size_t at, uint32_t, uint32_t n, const float4& acc, const float4& scale, const float4&) {
        EpilogueStore(ep, at, n, acc, scale, bias_at(n));
      });
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

// ---- persistent form -------------------------------------------------------------------
// One CTA per SM walks 128 x 256 output tiles t = blockIdx.x, blockIdx.x +
// gridDim.x, ... (tiles of one row block are neighbours, so concurrent CTAs
// share A in L2).  The wider tile is what the shared-memory fill rate asks for:
// a 128 x 128 tile moves 32 KB per 128x128x64 block of math (64 FLOP per byte
// from L2), which tops out near 12-13 TB/s of L2 traffic well below the tensor
// peak; 128 x 256 moves 48 KB per twice the math (85 FLOP per byte).  The
// operand ring keeps flowing across tile boundaries, the accumulator is
// double-buffered in tensor memory (2 x 256 columns: all of it), and the
// epilogue warps own a small staging slab, so tile i's epilogue (128 KB of f32) runs
// under tile i+1's main loop.  What the one-tile kernel pays per tile — barrier
// set-up, tensor-memory allocation, the first TMA round trip, CTA launch and
// retirement — is paid once per SM.
constexpr uint32_t kPBlockN = 256;
constexpr uint32_t kPMaxStages = 5;
constexpr uint32_t kPEpiWarps = 16;
constexpr uint32_t kPThreads = 64 + 32 * kPEpiWarps;   // warp 0 TMA, warp 1 MMA, then the epilogue warps
constexpr uint32_t kSlabCols = 32;
constexpr uint32_t kSlabBytes = 32 * kSlabCols * 4;   // one epilogue warp's 32 x 32 f32
// kPair: two CTAs of a cluster work one 256 x 256 tile (cta_group::2): each loads
// its own 128 rows of A and its own 128 of B's 256 rows (32 KB per k block instead
// of 48 KB for the same 128 x 256 of output per CTA), the even CTA issues one
// 256-row MMA that reads both shared memories, and each CTA's tensor memory
// receives its own 128 rows.  A third less operand traffic from L2 per flop, and
// the smaller stage leaves room for five ring slots: the K = 768 shapes of the
// step were bound by bytes in flight per SM, not by the tensor pipe.
template <bool kPair>
struct PTile {
  static constexpr uint32_t kStages = kPair ? 5 : 3;
  static constexpr uint32_t kBRows = kPair ? kPBlockN / 2 : kPBlockN;      // rows of B this CTA loads per k block
  static constexpr uint32_t kBTileBytes = kBRows * kBlockK * 2;
  static constexpr uint32_t kStageBytes = kATileBytes + kBTileBytes;
  static constexpr uint32_t kTmemCols = 2 * kPBlockN;
  static constexpr uint32_t kColsPerEpiWarp = kPBlockN / (kPEpiWarps / 4);
  static constexpr uint32_t kEpiPasses = kColsPerEpiWarp / kSlabCols;
  static constexpr uint32_t kRowsPerTile = kPair ? 2 * kBlockM : kBlockM;
};

// Tile order of the persistent kernel.  Bands of band_blocks row blocks; inside a
// band the row block runs fastest.  With band_blocks = 1 the column tile runs
// fastest: the CTAs of a wave share W (small) and each row block of A is used
// by neighbouring CTAs.  A vocabulary-wide W (dozens of column tiles) does not
// stay in L2 next to the C it produces; with a band of 64 row blocks the CTAs of
// one wave share the band's rows of A and two or three column tiles, and W is
// streamed from HBM once per band rather than once per row block (measured at
// 32768 x 32000 x 768: 1.93 ms -> 1.70 ms; bands of 16 / 32 / 128: 1.83 / 1.76 / 1.82).
constexpr uint32_t kWideBandBlocks = 64;
constexpr uint32_t kWideTilesN = 32;
__device__ __forceinline__ void TileCoord(uint32_t t, uint32_t tiles_m, uint32_t tiles_n, uint32_t band_blocks,
                                          uint32_t* m_block, uint32_t* n_block) {
  const uint32_t per_band = band_blocks * tiles_n;
  const uint32_t band = t / per_band, within = t - band * per_band;
  const uint32_t first = band * band_blocks;
  const uint32_t height = tiles_m - first < band_blocks ? tiles_m - first : band_blocks;
  const uint32_t nb = within / height;
  *m_block = first + (within - nb * height);
  *n_block = nb;
}

struct __align__(8) PBarriers {
  uint64_t full[kPMaxStages];
  uint64_t empty[kPMaxStages];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  volatile uint32_t abort;
};

// kSideLoads: the epilogue reads a second [M, N] f32 operand beside every output
// (an addend, or the x of an absorbed backward activation).  Those loads are
// then software-pipelined: the four of the NEXT group of rows are in flight
// while this group is converted and stored, across passes and from before the
// wait for the accumulator, so a memory round trip is not paid per group with
// every warp of the CTA waiting on it.
// Piece products and chains: an accumulator buffer holds one block of K, or one product, and the epilogue warps add them
// in registers, 64 outputs a thread, one buffer behind the products.
template <bool kSideLoads, bool kPair, Sums kSums>
__global__ void __launch_bounds__(kPThreads, 1)
UmmaGemmPersistentKernel(const __grid_constant__ UmmaMaps maps, const __grid_constant__ UmmaEpilogue ep,
                         uint32_t band_blocks) {
  constexpr bool kSeg = kSums == Sums::kPieces, kChain = kSums == Sums::kChain, kAdds = kSeg || kChain;
  static_assert(!(kSideLoads && kAdds), "the sums take the registers of the loads in flight");
  using T = PTile<kPair>;
  constexpr uint32_t kTN = kPBlockN;
  constexpr uint32_t kPStages = T::kStages, kPStageBytes = T::kStageBytes, kPTmemCols = T::kTmemCols;
  constexpr uint32_t kColsPerEpiWarp = T::kColsPerEpiWarp, kEpiPasses = T::kEpiPasses;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (SmemAddr(smem_raw) & 1023u)) & 1023u);
  uint8_t* slabs = smem + kPStages * kPStageBytes;
  PBarriers* bars = reinterpret_cast<PBarriers*>(slabs + kPEpiWarps * kSlabBytes);

  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t main_blocks = (ep.K + kBlockK - 1) / kBlockK;
  constexpr bool kSeveral = !kAdds && !kSideLoads;   // products side by side
  const uint32_t tiles_n = (ep.N + kTN - 1) / kTN, all_n = kSeveral ? tiles_n * ep.products : tiles_n;
  const uint32_t tiles_m = (ep.M + T::kRowsPerTile - 1) / T::kRowsPerTile;
  const uint32_t total_tiles = tiles_m * all_n;
  const uint32_t groups = kSeg ? ep.seg_blocks : (kChain ? ep.products : 1u);   // accumulators per tile
  // A work unit is a CTA, or a CTA pair: `unit` walks the tiles, `cta_rank` is this CTA's half of a pair's tile.
  const uint32_t cta_rank = kPair ? ClusterCtaRank() : 0u;
  const uint32_t unit = kPair ? blockIdx.x >> 1 : blockIdx.x, units = kPair ? gridDim.x >> 1 : gridDim.x;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < kPStages; ++s) {
      MbarInit(&bars->full[s], 1);
      MbarInit(&bars->empty[s], 1);
    }
    for (uint32_t b = 0; b < 2; ++b) {
      MbarInit(&bars->tmem_full[b], 1);
      // one arrival per epilogue warp (of both CTAs of a pair: the even CTA's barrier counts them all)
      MbarInit(&bars->tmem_empty[b], kPair ? 2 * kPEpiWarps : kPEpiWarps);
    }
    bars->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if constexpr (kPair) {
      TmemAllocPair(const_cast<uint32_t*>(&bars->tmem_base), kPTmemCols);
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                   ::"r"(SmemAddr(&bars->tmem_base)), "r"(kPTmemCols)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if constexpr (kPair) ClusterSync();   // the peer's barriers exist before anything signals them
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  AwaitPrevious();
  const uint32_t tmem_base = bars->tmem_base;

  if (warp == 0) {
    // ---- TMA producer ----
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (uint32_t t = unit; t < total_tiles && ok; t += units) {
        uint32_t mb, nb;
        TileCoord(t, tiles_m, all_n, band_blocks, &mb, &nb);
        const uint32_t product = kSeveral ? nb / tiles_n : 0;
        nb -= product * tiles_n;
        const uint32_t m0 = mb * T::kRowsPerTile + cta_rank * kBlockM, n0 = nb * kTN;
        // Ask L2 for the A rows of this CTA's next tile now, so that its loads
        // find them there instead of paying an HBM round trip inside the ring.
        uint32_t ahead = 0;   // blocks of a tile
        for (uint32_t p = kChain ? 0 : product; p <= (kChain ? groups - 1 : product); ++p) ahead += ReductionBlocks(ep, main_blocks, p);
        if (t + units < total_tiles && ahead <= 64 && !kSeg) {   // (a long K would only thrash L2)
          uint32_t next_mb, next_nb;
          TileCoord(t + units, tiles_m, all_n, band_blocks, &next_mb, &next_nb);
          const uint32_t next_m0 = next_mb * T::kRowsPerTile + cta_rank * kBlockM;
          if (next_m0 != m0)
            for (uint32_t p = 0; p < (kChain ? groups : 1u); ++p)   // (side by side: they share A)
              for (uint32_t kb = 0; kb < main_blocks; ++kb)
                asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];"
                             ::"l"(reinterpret_cast<uint64_t>(&maps.a[p])),
                               "r"(static_cast<int32_t>(kb * kBlockK)), "r"(static_cast<int32_t>(next_m0))
                             : "memory");
        }
        for (uint32_t g = 0; g < (kChain ? groups : 1u) && ok; ++g) {
          const uint32_t p = kChain ? g : product;
          const uint32_t k_blocks = kSeg ? groups * ep.segs : ReductionBlocks(ep, main_blocks, p);
          for (uint32_t kb = 0; kb < k_blocks; ++kb, ++it) {
            const uint32_t s = it % kPStages, round = it / kPStages;
            if (round > 0 && !PartnerWait<kSeg>(&bars->empty[s], (round - 1) & 1)) {
              ep.status->wait_timeout = 1;
              bars->abort = 1;
              ok = false;
              break;
            }
            uint8_t* a_dst = smem + s * kPStageBytes;
            const BlockAt at = BlockCoord(ep, kb, main_blocks);
            const CUtensorMap* ma = at.aux ? &maps.a2[p] : &maps.a[p];
            const CUtensorMap* mb_ = at.aux ? &maps.b2[p] : &maps.b[p];
            if constexpr (kPair) {
              // Both CTAs' bytes are counted on the even CTA's barrier, which alone expects them.
              if (cta_rank == 0) MbarExpectTx(&bars->full[s], 2 * kPStageBytes);
              const uint32_t full_bar = MapToCta(SmemAddr(&bars->full[s]), 0);
              TmaLoad2DPair(a_dst, ma, full_bar, at.a, static_cast<int32_t>(m0));
              TmaLoad2DPair(a_dst + kATileBytes, mb_, full_bar, at.b, static_cast<int32_t>(n0 + cta_rank * kBlockN));
            } else {
              MbarExpectTx(&bars->full[s], kPStageBytes);
              TmaLoad2D(a_dst, ma, &bars->full[s], at.a, static_cast<int32_t>(m0));
              // B's rows as 128-row boxes, back to back: one [256][64] tile.
              TmaLoad2D(a_dst + kATileBytes, mb_, &bars->full[s], at.b, static_cast<int32_t>(n0));
              TmaLoad2D(a_dst + kATileBytes + kBlockN * kBlockK * 2, mb_, &bars->full[s], at.b,
                        static_cast<int32_t>(n0 + kBlockN));
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer ----
    if (ElectOne() && cta_rank == 0) {   // (a pair's odd CTA issues nothing: its memories are read by the even one's MMAs)
      const uint32_t idesc = MakeInstrDesc(T::kRowsPerTile, kTN);
      uint32_t it = 0, lt = 0;   // lt: accumulators so far
      bool ok = true;
      for (uint32_t t = unit, g = 0; t < total_tiles && ok; ++lt, g = g + 1 < groups ? g + 1 : (t += units, 0u)) {
        const uint32_t buf = lt & 1, use = lt >> 1;
        if (use > 0 && !PartnerWait<kSeg>(&bars->tmem_empty[buf], (use - 1) & 1)) {
          ep.status->wait_timeout = 1;
          bars->abort = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem_base + buf * kTN;
        uint32_t group;   // blocks of this accumulator
        if constexpr (kSeg) {
          group = ep.segs;
        } else if constexpr (kChain) {
          group = ReductionBlocks(ep, main_blocks, g);
        } else {
          uint32_t mb, nb;
          TileCoord(t, tiles_m, all_n, band_blocks, &mb, &nb);
          group = ReductionBlocks(ep, main_blocks, kSeveral ? nb / tiles_n : 0);
        }
        for (uint32_t kb = 0; kb < group; ++kb, ++it) {
          const uint32_t s = it % kPStages, round = it / kPStages;
          if (!PartnerWait<kSeg && kPair>(&bars->full[s], round & 1)) {
            ep.status->wait_timeout = 1;
            bars->abort = 1;
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_addr = SmemAddr(smem + s * kPStageBytes);
          const uint64_t desc_a = MakeSmemDesc(a_addr);
          const uint64_t desc_b = MakeSmemDesc(a_addr + kATileBytes);
#pragma unroll
          for (uint32_t k = 0; k < kBlockK / kUmmaK; ++k) {
            if constexpr (kPair) UmmaBf16Pair(acc, desc_a + 2 * k, desc_b + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
            else UmmaBf16(acc, desc_a + 2 * k, desc_b + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
          }
          if constexpr (kPair) UmmaCommitPair(&bars->empty[s], 0);
          else UmmaCommit(&bars->empty[s]);
        }
        // accumulator complete (or abandoned on timeout)
        if constexpr (kPair) UmmaCommitPair(&bars->tmem_full[buf], 0);
        else UmmaCommit(&bars->tmem_full[buf]);
      }
    }
  } else {
    // ---- epilogue warps.  TMEM lane quarter = warp % 4 (the hardware's rule);
    // the warps of a quarter split the tile's 256 columns between them.
    const uint32_t quarter = warp & 3, col_group = (warp - 2) >> 2;
    float* slab = reinterpret_cast<float*>(slabs + (warp - 2) * kSlabBytes);
    constexpr uint32_t kChunks = kSlabCols / 4;          // 16-byte chunks per slab row
    constexpr uint32_t kRowsPerInstr = 32 / kChunks;     // rows one store instruction covers
    const uint32_t sub = lane / kChunks, cl = lane % kChunks;
    uint32_t lt = 0;   // accumulators so far
    for (uint32_t t = unit; t < total_tiles; t += units, ++lt) {
      uint32_t buf = lt & 1, use = lt >> 1;
      uint32_t mb, nb;
      TileCoord(t, tiles_m, all_n, band_blocks, &mb, &nb);
      const uint32_t product = kSeveral ? nb / tiles_n : 0;
      nb -= product * tiles_n;
      const uint32_t m0 = mb * T::kRowsPerTile + cta_rank * kBlockM, n0 = nb * kTN;
      if (ep.fuse_mode == kFuseActBwd) {
        // The absorbed backward activation reads x[m, n] next to every output:
        // ask L2 for this warp's lines of the NEXT tile now (one 128-byte line per
        // lane and pass), a whole tile ahead of the loads that use them.
        auto prefetch_x = [&](uint32_t tile) {
          uint32_t pmb, pnb;
          TileCoord(tile, tiles_m, all_n, band_blocks, &pmb, &pnb);   // (one product: nothing side by side has an x)
          const uint32_t prow = pmb * T::kRowsPerTile + cta_rank * kBlockM + quarter * 32 + lane;
          if (prow >= ep.M) return;
#pragma unroll
          for (uint32_t pass = 0; pass < kEpiPasses; ++pass) {
            const uint32_t pcol = pnb * kTN + col_group * kColsPerEpiWarp + pass * kSlabCols;
            if (pcol < ep.N)
              asm volatile("prefetch.global.L2 [%0];" ::"l"(ep.fuse_x + static_cast<size_t>(prow) * ep.N + pcol));
          }
        };
        if (lt == 0) prefetch_x(t);
        if (t + units < total_tiles) prefetch_x(t + units);
      }
      const uint32_t row0 = m0 + quarter * 32;
      const uint32_t rows = row0 < ep.M ? (ep.M - row0 < 32 ? ep.M - row0 : 32) : 0;
      [[maybe_unused]] const float* side_ptr = ep.fuse_mode == kFuseActBwd ? ep.fuse_x : ep.addend;
      [[maybe_unused]] const bool gelu_grad_only = IsGeluGradOnly(ep);
      [[maybe_unused]] const bool addend_only = IsAddendOnly(ep);
      [[maybe_unused]] const bool bias_gelu_only = IsBiasGeluOnly(ep);
      [[maybe_unused]] const bool copy_only = IsCopyOnly(ep);
      [[maybe_unused]] const bool plain_store = IsPlainStore(ep);
      [[maybe_unused]] const bool bias_stored = kSeg && IsBiasStored(ep, kActNone), bias_gelu_stored = kSeg && IsBiasStored(ep, kActGelu);
      [[maybe_unused]] const bool sum_stored = kSeg && IsSum(ep);
      const bool side_by_side = kSeveral && ep.products > 1;
      [[maybe_unused]] const float alpha = side_by_side ? ep.product[product].alpha : ep.alpha;
      [[maybe_unused]] const float* col_scale = side_by_side ? ep.product[product].col_scale : ep.col_scale;
      [[maybe_unused]] uint16_t* pack_dst = side_by_side ? ep.product[product].pack_dst : ep.pack_dst;
      [[maybe_unused]] const bool ragged = (ep.N & 3u) != 0;   // (never with kSideLoads)
      [[maybe_unused]] float4 side_a[4], side_b[4];
      if constexpr (kSideLoads) {   // the first group's loads fly during the wait for the accumulator
        const uint32_t n_g = n0 + col_group * kColsPerEpiWarp + cl * 4;
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
          const uint32_t rr = sub + u * kRowsPerInstr;
          side_a[u] = rr < rows && n_g < ep.N
                          ? __ldg(reinterpret_cast<const float4*>(side_ptr + static_cast<size_t>(row0 + rr) * ep.N + n_g))
                          : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      auto await = [&] {
        bool there = PartnerWait<kSeg>(&bars->tmem_full[buf], use & 1);
        if (!there && lane == 0) { ep.status->wait_timeout = 1; bars->abort = 1; }
        if (bars->abort) there = false;
        there = __all_sync(0xFFFFFFFFu, there);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return there;
      };
      auto hand_back = [&] {   // the accumulator buffer is read out
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          if constexpr (kPair) MbarArriveCluster(MapToCta(SmemAddr(&bars->tmem_empty[buf]), 0));
          else MbarArrive(&bars->tmem_empty[buf]);
        }
      };
      [[maybe_unused]] float sum[kAdds ? kEpiPasses : 1][kAdds ? kSlabCols : 1];
      [[maybe_unused]] bool remake = false;   // some sum of this warp's is not finite
      if constexpr (kAdds) {
#pragma unroll
        for (uint32_t p = 0; p < kEpiPasses; ++p)
#pragma unroll
          for (uint32_t j = 0; j < kSlabCols; ++j) sum[p][j] = kChain ? -0.0f : 0.0f;   // (-0 + x is x, -0 included)
        bool ok = true;
        for (uint32_t g = 0; g < groups; ++g) {
          if (g > 0) { ++lt; buf = lt & 1; use = lt >> 1; }
          if (!(ok = await())) break;
          const uint32_t t_row = tmem_base + ((quarter * 32) << 16) + buf * kTN + col_group * kColsPerEpiWarp;
#pragma unroll
          for (uint32_t c = 0; c < kColsPerEpiWarp; c += 16) {   // (all 64 at once do not fit the registers)
            uint32_t ra[16];
            TmemLoad16(t_row + c, ra);
            TmemWaitLd();
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j) {
              float& to = sum[c / kSlabCols][c % kSlabCols + j];
              if constexpr (kChain) to += __uint_as_float(ra[j]) * alpha;   // as the products' own epilogues, one after the other
              else to += __uint_as_float(ra[j]);
            }
          }
          hand_back();
        }
        if (!ok) break;
        if constexpr (kSeg) {
#pragma unroll
          for (uint32_t p = 0; p < kEpiPasses; ++p) remake = remake || !AllFinite(sum[p]);
          remake = __any_sync(0xFFFFFFFFu, remake);
        }
      } else {
        if (!await()) break;
      }
      // 32 columns at a time through the slab.  A thread writes its accumulator
      // row as eight 16-byte chunks, chunk index XOR-ed with the row; the warp
      // then reads four rows per instruction (eight lanes each): whole 128-byte
      // lines of C per store instruction.  Conflict-free both ways.
      const uint32_t t_row = tmem_base + ((quarter * 32) << 16) + buf * kTN + col_group * kColsPerEpiWarp;
      if constexpr (!kSideLoads) {
        auto store_pass = [&](uint32_t pass, const uint32_t (&ra)[32]) {
  #pragma unroll
          for (uint32_t q = 0; q < kChunks; ++q)
            *reinterpret_cast<uint4*>(slab + lane * kSlabCols + ((q ^ (lane & (kChunks - 1))) * 4)) =
                make_uint4(ra[4 * q], ra[4 * q + 1], ra[4 * q + 2], ra[4 * q + 3]);
          __syncwarp();
          const uint32_t n = n0 + col_group * kColsPerEpiWarp + pass * kSlabCols + cl * 4;
          auto staged = [&](uint32_t rr) {
            return *reinterpret_cast<const float4*>(slab + rr * kSlabCols + ((cl ^ (rr & (kChunks - 1))) * 4));
          };
          if constexpr (kChain) {   // scaled already, and nothing else is part of a chain
  #pragma unroll 4
            for (uint32_t rr = sub; rr < rows && n < ep.N; rr += kRowsPerInstr)
              *reinterpret_cast<float4*>(ep.C + static_cast<size_t>(row0 + rr) * ep.N + n) = staged(rr);
          } else if (kSeg && remake) {
            for (uint32_t rr = sub; rr < rows && n < ep.N; rr += kRowsPerInstr) StoreRemade(ep, row0 + rr, n, staged(rr));
          } else if (ragged) {
            for (uint32_t rr = sub; rr < rows && n < ep.N; rr += kRowsPerInstr)
              EpilogueStoreRagged(ep, row0 + rr, n, staged(rr), false);
          } else if (n < ep.N) {   // N % 4 == 0: a float4 is all in or all out
            float4 scale = make_float4(alpha, alpha, alpha, alpha);
            if (col_scale) scale = __ldg(reinterpret_cast<const float4*>(col_scale + n));
            float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
            if (ep.bias) bias = __ldg(reinterpret_cast<const float4*>(ep.bias + n));
            float4 kscale = make_float4(1.f, 1.f, 1.f, 1.f);   // the consumer's per-column factor (x * 1 == x)
            if (ep.fuse_mode != kFuseNone && ep.shadow_k_scale)
              kscale = __ldg(reinterpret_cast<const float4*>(ep.shadow_k_scale + n));
            if (kSeg && sum_stored) {   // two addends in flight at a time: more do not fit the registers
  #pragma unroll 1
              for (uint32_t rr = sub; rr < rows; rr += 2 * kRowsPerInstr) {
                const bool both = rr + kRowsPerInstr < rows;
                const size_t at = static_cast<size_t>(row0 + rr) * ep.N + n, next = at + static_cast<size_t>(kRowsPerInstr) * ep.N;
                const float4 d = __ldg(reinterpret_cast<const float4*>(ep.addend + at));
                const float4 e = __ldg(reinterpret_cast<const float4*>(ep.addend + (both ? next : at)));
                EpilogueStoreSum(ep, at, staged(rr), scale, bias, d);
                if (both) EpilogueStoreSum(ep, next, staged(rr + kRowsPerInstr), scale, bias, e);
              }
            } else
  #pragma unroll 4
            for (uint32_t rr = sub; rr < rows; rr += kRowsPerInstr) {
              const float4 acc = staged(rr);
              const size_t at = static_cast<size_t>(row0 + rr) * ep.N + n;
              if (plain_store)
                EpilogueStorePlain(ep, at, acc, scale);
              else if (copy_only)
                EpilogueStoreCopy(pack_dst, at, acc, scale);
              else if (kSeg && bias_stored)
                EpilogueStoreBias<kActNone>(ep, at, acc, scale, bias);
              else if (kSeg && bias_gelu_stored)
                EpilogueStoreBias<kActGelu>(ep, at, acc, scale, bias);
              else if (bias_gelu_only)
                EpilogueStoreBiasGelu(ep, at, acc, scale, bias, kscale);
              else
                EpilogueStore(ep, at, n, acc, scale, bias, true, kscale);
            }
          }
          __syncwarp();   // the slab is rewritten next
        };
        if constexpr (kAdds) {
#pragma unroll
          for (uint32_t pass = 0; pass < kEpiPasses; ++pass) {
            uint32_t ra[32];
#pragma unroll
            for (uint32_t j = 0; j < kSlabCols; ++j) ra[j] = __float_as_uint(sum[pass][j]);
            store_pass(pass, ra);
          }
        } else {
  #pragma unroll 1
          for (uint32_t pass = 0; pass < kEpiPasses; ++pass) {
            uint32_t ra[32];
            TmemLoad32(t_row + pass * kSlabCols, ra);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (pass == kEpiPasses - 1) hand_back();   // before the slow part
            store_pass(pass, ra);
          }
        }
      } else {
        // Groups of four row steps (two per pass); group g + 1's side operands are
        // loaded while group g is converted and stored.
        auto load_group = [&](float4 (&dst)[4], uint32_t grp) {
          const uint32_t n_g = n0 + col_group * kColsPerEpiWarp + (grp >> 1) * kSlabCols + cl * 4;
#pragma unroll
          for (uint32_t u = 0; u < 4; ++u) {
            const uint32_t rr = sub + ((grp & 1) * 4 + u) * kRowsPerInstr;
            dst[u] = rr < rows && n_g < ep.N
                         ? __ldg(reinterpret_cast<const float4*>(side_ptr + static_cast<size_t>(row0 + rr) * ep.N + n_g))
                         : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        };
#pragma unroll
        for (uint32_t pass = 0; pass < kEpiPasses; ++pass) {
          uint32_t ra[32];
          TmemLoad32(t_row + pass * kSlabCols, ra);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (pass == kEpiPasses - 1) hand_back();
#pragma unroll
          for (uint32_t q = 0; q < kChunks; ++q)
            *reinterpret_cast<uint4*>(slab + lane * kSlabCols + ((q ^ (lane & (kChunks - 1))) * 4)) =
                make_uint4(ra[4 * q], ra[4 * q + 1], ra[4 * q + 2], ra[4 * q + 3]);
          __syncwarp();
          const uint32_t n = n0 + col_group * kColsPerEpiWarp + pass * kSlabCols + cl * 4;
          float4 scale = make_float4(ep.alpha, ep.alpha, ep.alpha, ep.alpha);
          float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
          float4 kscale = make_float4(1.f, 1.f, 1.f, 1.f);
          if (n < ep.N) {
            if (ep.col_scale) scale = __ldg(reinterpret_cast<const float4*>(ep.col_scale + n));
            if (ep.bias) bias = __ldg(reinterpret_cast<const float4*>(ep.bias + n));
            if (ep.fuse_mode != kFuseNone && ep.shadow_k_scale)
              kscale = __ldg(reinterpret_cast<const float4*>(ep.shadow_k_scale + n));
          }
          auto process = [&](const float4 (&sv)[4], uint32_t half) {
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
              const uint32_t rr = sub + (half * 4 + u) * kRowsPerInstr;
              if (rr < rows && n < ep.N) {
                const float4 acc = *reinterpret_cast<const float4*>(
                    slab + rr * kSlabCols + ((cl ^ (rr & (kChunks - 1))) * 4));
                const size_t at = static_cast<size_t>(row0 + rr) * ep.N + n;
                if (gelu_grad_only)
                  EpilogueStoreGeluGrad(ep, at, acc, scale, kscale, sv[u]);
                else if (addend_only)
                  EpilogueStoreAddend(ep, at, acc, scale, sv[u]);
                else
                  EpilogueStore(ep, at, n, acc, scale, bias, true, kscale, true, sv[u]);
              }
            }
          };
          load_group(side_b, 2 * pass + 1);
          process(side_a, 0);
          if (pass + 1 < kEpiPasses) load_group(side_a, 2 * pass + 2);
          process(side_b, 1);
          __syncwarp();   // the slab is rewritten next
        }
      }
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (bars->abort) DrainDelay();
  if constexpr (kPair) ClusterSync();   // neither CTA leaves while the other may still read its memories
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if constexpr (kPair) {
      TmemFreePair(tmem_base, kPTmemCols);
    } else {
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                   "r"(kPTmemCols)
                   : "memory");
    }
  }
}

// Weight conversion to the K-major bf16 layout [N][K] the kernel consumes.
// transpose = true: src is [K][N] (the NN forms); false: src is [N][K].
template <typename T> __device__ __forceinline__ uint16_t ToBf16Bits(T v);
template <> __device__ __forceinline__ uint16_t ToBf16Bits<int8_t>(int8_t v) {
  return static_cast<uint16_t>(__float_as_uint(static_cast<float>(v)) >> 16);  // exact
}
template <> __device__ __forceinline__ uint16_t ToBf16Bits<uint16_t>(uint16_t v) { return v; }
template <> __device__ __forceinline__ uint16_t ToBf16Bits<float>(float f) {
  uint32_t b = __float_as_uint(f);
  if ((b & 0x7FFFFFFFu) > 0x7F800000u) return static_cast<uint16_t>((b >> 16) | 0x0040u);
  b += 0x7FFFu + ((b >> 16) & 1u);
  return static_cast<uint16_t>(b >> 16);
}

template <typename T> __device__ __forceinline__ float WidenWeight(T v);
template <> __device__ __forceinline__ float WidenWeight<int8_t>(int8_t v) { return static_cast<float>(v); }
template <> __device__ __forceinline__ float WidenWeight<uint16_t>(uint16_t v) {
  return __uint_as_float(static_cast<uint32_t>(v) << 16);
}
template <> __device__ __forceinline__ float WidenWeight<float>(float v) { return v; }
template <typename T>
__device__ __forceinline__ uint16_t WeightBits(T v, const float* k_scale, uint32_t k) {
  return k_scale ? ToBf16Bits<float>(WidenWeight<T>(v) * k_scale[k]) : ToBf16Bits<T>(v);
}

template <typename T>
__global__ void WeightToBf16Kernel(const T* __restrict__ src, uint16_t* __restrict__ dst, uint32_t N,
                                   uint32_t K, bool transpose, const float* __restrict__ k_scale) {
  AwaitPrevious();
  __shared__ uint16_t tile[32][33];
  const uint32_t bx = blockIdx.x * 32, by = blockIdx.y * 32;
  if (!transpose) {  // src [N][K] -> dst [N][K]
    for (uint32_t i = threadIdx.y; i < 32; i += blockDim.y) {
      const uint32_t n = by + i, k = bx + threadIdx.x;
      if (n < N && k < K)
        dst[static_cast<size_t>(n) * K + k] = WeightBits<T>(src[static_cast<size_t>(n) * K + k], k_scale, k);
    }
    return;
  }
  // src [K][N]: bx indexes n, by indexes k
  for (uint32_t i = threadIdx.y; i < 32; i += blockDim.y) {
    const uint32_t k = by + i, n = bx + threadIdx.x;
    if (k < K && n < N) tile[i][threadIdx.x] = WeightBits<T>(src[static_cast<size_t>(k) * N + n], k_scale, k);
  }
  __syncthreads();
  for (uint32_t i = threadIdx.y; i < 32; i += blockDim.y) {
    const uint32_t n = bx + i, k = by + threadIdx.x;
    if (k < K && n < N) dst[static_cast<size_t>(n) * K + k] = tile[threadIdx.x][i];
  }
}

}  // namespace

template <bool kPair>
static size_t UmmaPersistentSmemBytes() {
  using T = PTile<kPair>;
  return T::kStages * T::kStageBytes + kPEpiWarps * kSlabBytes + sizeof(PBarriers) + 1024;
}
template <uint32_t kTN>
static size_t UmmaTileSmemBytes() {
  using T = TTile<kTN>;
  return T::kStages * T::kStageBytes + sizeof(TBarriers) + 1024;
}

// Calls f(kernel, shared-memory bytes) with the tile kernel of this width.
template <Sums kSums, typename F>
static cudaError_t WithTileKernel(uint32_t tn, F f) {
  switch (tn) {
    case 64: return f(UmmaGemmTileKernel<64, kSums>, UmmaTileSmemBytes<64>());
    case 128: return f(UmmaGemmTileKernel<128, kSums>, UmmaTileSmemBytes<128>());
    case 192: return f(UmmaGemmTileKernel<192, kSums>, UmmaTileSmemBytes<192>());
    default: return f(UmmaGemmTileKernel<256, kSums>, UmmaTileSmemBytes<256>());
  }
}
template <typename F>
static cudaError_t WithTileKernel(Sums sums, uint32_t tn, F f) {
  return sums == Sums::kPieces  ? WithTileKernel<Sums::kPieces>(tn, f)
         : sums == Sums::kChain ? WithTileKernel<Sums::kChain>(tn, f)
                                : WithTileKernel<Sums::kPlain>(tn, f);
}
// ... with the persistent one.  (Only a plain product has side loads.)
template <typename F>
static cudaError_t WithPersistentKernel(Sums sums, bool side_loads, bool pair, F f) {
  const size_t bytes = pair ? UmmaPersistentSmemBytes<true>() : UmmaPersistentSmemBytes<false>();
  if (sums == Sums::kPieces)
    return pair ? f(UmmaGemmPersistentKernel<false, true, Sums::kPieces>, bytes)
                : f(UmmaGemmPersistentKernel<false, false, Sums::kPieces>, bytes);
  if (sums == Sums::kChain)
    return pair ? f(UmmaGemmPersistentKernel<false, true, Sums::kChain>, bytes)
                : f(UmmaGemmPersistentKernel<false, false, Sums::kChain>, bytes);
  if (side_loads)
    return pair ? f(UmmaGemmPersistentKernel<true, true, Sums::kPlain>, bytes)
                : f(UmmaGemmPersistentKernel<true, false, Sums::kPlain>, bytes);
  return pair ? f(UmmaGemmPersistentKernel<false, true, Sums::kPlain>, bytes)
              : f(UmmaGemmPersistentKernel<false, false, Sums::kPlain>, bytes);
}

static std::atomic<bool> g_cta_pairs{true};
void UmmaSetCtaPairs(bool on) { g_cta_pairs.store(on, std::memory_order_relaxed); }

static cudaError_t Configure() {
  auto allow = [](auto kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  };
  cudaError_t e = cudaSuccess;
  for (Sums sums : {Sums::kPlain, Sums::kPieces, Sums::kChain}) {
    for (uint32_t tn : {64u, 128u, 192u, 256u})
      if ((e = WithTileKernel(sums, tn, allow)) != cudaSuccess) return e;
    for (bool pair : {false, true})
      for (bool side_loads : {false, true})
        if ((e = WithPersistentKernel(sums, side_loads, pair, allow)) != cudaSuccess) return e;
  }
  return e;
}

UmmaGemmPlan UmmaPlanGemm(uint32_t M, uint32_t N, uint32_t k_blocks, uint32_t group, bool light, uint32_t sms,
                          uint32_t side_by_side, uint32_t only_splits, bool chained) {
  UmmaGemmPlan p;
  const uint32_t ptiles_n = (N + kPBlockN - 1) / kPBlockN * side_by_side, tiles_m = (M + kBlockM - 1) / kBlockM;
  const uint64_t wide = static_cast<uint64_t>(ptiles_n) * tiles_m;
  const bool pairs_on = g_cta_pairs.load(std::memory_order_relaxed) && sms >= 2;
  // The tile kernel, on the width and split of least estimated time (us): waves of CTAs, each a fixed part, its
  // reduction blocks, its epilogue and, when the reduction is cut, the exchange.  The constants are a fit (10 %
  // standard error) to a sweep of 32 to 4096 rows, widths 256 to 32000 and K 512 to 32000 on a B200; the persistent
  // kernel's likewise.
  double best = 1e30;
  for (uint32_t tn : {64u, 128u, 192u, 256u})
    for (uint32_t splits = 1; splits <= 4 && splits * group <= k_blocks; splits *= 2) {
      if ((only_splits != 0 && splits != only_splits) || (chained && splits > 1 && tn > 128)) continue;
      const uint64_t ctas = static_cast<uint64_t>(tiles_m) * ((N + tn - 1) / tn) * side_by_side * splits;
      const uint64_t room = splits <= 2 ? sms : sms * 9 / 10;   // clusters of four do not fill every GPC
      const double waves = static_cast<double>((ctas + room - 1) / room);
      const double block = std::max(0.165 + 0.00087 * tn, 0.267);
      const double t = 0.8 + waves * (2.0 + block * ((k_blocks + splits - 1) / splits) + 0.02 * tn / splits + (splits > 1 ? 3.0 : 0.0));
      if (t < best) {
        best = t;
        p.tn = tn;
        p.splits = splits;
        p.grid = static_cast<uint32_t>(ctas);
        p.b_box = tn;
      }
    }
  if (wide > sms && only_splits <= 1) {
    // Enough tiles for every SM to amortise its set-up over several: a round of the persistent kernel is its main
    // loop (0.53 us per reduction block, 0.43 in CTA pairs, which load a third fewer bytes per flop) or its
    // epilogue, whichever is longer.  At 32768 rows the epilogue is HBM's: plain and copy-only ones take 8.3 us a tile
    // and 7.3 in pairs, those with a second operand or an activation about 10.5 and 11.5, for a pair's two epilogues
    // must both finish before the accumulator is free again.  An output that stays in L2 takes about 2 us less.
    const uint64_t pair_tiles = static_cast<uint64_t>(ptiles_n) * ((M + 2 * kBlockM - 1) / (2 * kBlockM));
    const uint64_t pairs = sms / 2;
    const double l2 = static_cast<uint64_t>(M) * N * side_by_side <= (1ull << 24) ? 2.0 : 0.0;
    const double single = 7.0 + static_cast<double>((wide + sms - 1) / sms) * std::max(0.53 * k_blocks, (light ? 8.3 : 10.5) - l2);
    const double paired = pairs_on && wide > 2ull * sms
                              ? 7.5 + static_cast<double>((pair_tiles + pairs - 1) / pairs) *
                                          std::max(0.43 * k_blocks, (light ? 7.3 : 11.5) - l2)
                              : 1e30;
    if (std::min(single, paired) < best) {
      best = std::min(single, paired);
      p = UmmaGemmPlan{};
      p.persistent = true;
      p.pair = paired < single;
      p.tn = kPBlockN;
      p.grid = p.pair ? sms & ~1u : sms;
      const uint32_t band = ptiles_n >= kWideTilesN ? kWideBandBlocks : 1u;
      p.band = p.pair && band > 1 ? band / 2 : band;
      p.b_box = kBlockN;
    }
  }
  p.us = best;
  return p;
}

cudaError_t UmmaGemmLaunch(const UmmaGemmPlan& plan, const UmmaMaps& maps, const UmmaEpilogue& ep, cudaStream_t s) {
  // The shared-memory limit of a kernel is a per-device attribute: one flag per
  // device, so a second backend on another GPU of the same process configures its own.
  static std::atomic<bool> configured_on[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  const bool tracked = dev >= 0 && dev < 64;
  if (!tracked || !configured_on[dev].load(std::memory_order_acquire)) {
    if (cudaError_t e = Configure(); e != cudaSuccess) return e;
    if (tracked) configured_on[dev].store(true, std::memory_order_release);
  }
  const Sums sums = ep.seg_blocks != 0 ? Sums::kPieces : ep.chained ? Sums::kChain : Sums::kPlain;
  if (!plan.persistent)
    return WithTileKernel(sums, plan.tn, [&](auto kernel, size_t bytes) {
      return Next(kernel, plan.grid, kTThreads, bytes, s, plan.splits)(maps, ep, plan.splits);
    });
  // An addend or the x of an absorbed backward activation is software-pipelined (16 bytes at a time).
  const bool side_loads = (ep.addend != nullptr || ep.fuse_mode == kFuseActBwd) && (ep.N & 3) == 0;
  return WithPersistentKernel(sums, side_loads, plan.pair, [&](auto kernel, size_t bytes) {
    return Next(kernel, plan.grid, kPThreads, bytes, s, plan.pair ? 2u : 1u)(maps, ep, plan.band);
  });
}

void WeightToBf16(const void* src, BType type, uint16_t* dst, uint32_t N, uint32_t K,
                  bool transpose, const float* k_scale, cudaStream_t s) {
  dim3 block(32, 8);
  dim3 grid = transpose ? dim3((N + 31) / 32, (K + 31) / 32) : dim3((K + 31) / 32, (N + 31) / 32);
  switch (type) {
    case BType::kI8:
      Next(WeightToBf16Kernel<int8_t>, grid, block, 0, s)(static_cast<const int8_t*>(src), dst, N, K, transpose, k_scale);
      break;
    case BType::kBf16:
      Next(WeightToBf16Kernel<uint16_t>, grid, block, 0, s)(static_cast<const uint16_t*>(src), dst, N, K, transpose, k_scale);
      break;
    case BType::kF32:
      Next(WeightToBf16Kernel<float>, grid, block, 0, s)(static_cast<const float*>(src), dst, N, K, transpose, k_scale);
      break;
  }
}

}  // namespace see::k
