// Interface between the tensor-core GEMM kernel (k_gemm_umma.cu) and its host
// planner (umma_gemm.cc).
#ifndef SEE_CUDA_UMMA_KERNEL_H_
#define SEE_CUDA_UMMA_KERNEL_H_

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "kernels.h"

namespace see::k {

namespace umma_cfg {
constexpr uint32_t kBlockM = 128, kBlockN = 128, kBlockK = 64;
}

struct UmmaEpilogue {
  float* C;                 // [M, N] f32
  const float* addend;      // [M, N] or null:  v = d + v (before the bias, or after it when addend_last)
  const float* bias;        // [N] or null:     v = v + bias[n]
  const float* col_scale;   // [N] or null:     v = acc * col_scale[n]   (else acc * alpha)
  float alpha;
  int act;
  uint32_t M, N, K;
  DeviceStatus* status;
  // A following activation instruction absorbed into this epilogue.  With v the
  // value above (after scale, addend, bias, act):
  //   kFuseActFwd: g = act(v);          kFuseActBwd: g = act'(dy = v, x = fuse_x[m, n]).
  // g leaves only as the bf16 operand copy of the GEMM that consumes it
  // (shadow_dst, [M, N], times shadow_k_scale[n] when set); v itself is stored to
  // C only when store_c is set.
  int fuse_mode = 0;
  int fuse_act = 0;
  const float* fuse_x = nullptr;
  uint16_t* shadow_dst = nullptr;
  const float* shadow_k_scale = nullptr;
  int store_c = 1;
  int addend_last = 0;
  // Up to kUmmaProducts products of one shape in one launch.  chained = 0: side by side, each with its own output
  // (`products` > 1: they share A, and every one leaves as its attention copy alone, product[p].pack_dst).
  // chained = 1: one output, the sum of the products: an accumulator each, scaled and added in f32 in the products' order,
  // what launches one after the other leave.
  // Each may carry a low-rank term: after the main operands' K the reduction continues over aux_k_blocks blocks of
  // 64 from a second operand pair, T' [M, 64 * aux_k_blocks] and B' [N, 64 * aux_k_blocks] (bf16, K-major),
  // so the tile holds A W^T + T' B'^T before the epilogue scales it.  With T' and
  // B' the three-way bf16 splits of f32 factors (LoraSplit* in kernels.h) the
  // added term is the f32 product t . b to about 2^-23 of |t| |b|.
  uint32_t products = 1;
  int chained = 0;
  struct Product {
    uint32_t aux_k_blocks = 0;
    uint16_t* pack_dst = nullptr;      // side by side
    const float* col_scale = nullptr;  // side by side: [N], or null and alpha
    float alpha = 1.0f;
  } product[kUmmaProducts];
  // The stored value also as bf16 [M, N] (GemmArgs::pack_dst).
  uint16_t* pack_dst = nullptr;
  // An f32-accurate product out of bf16 pieces: the operands hold pieces side by side along K, each
  // seg_blocks * 64 wide (zero-padded).  64 wide block by block, piece product s = 0 .. segs - 1 multiplies A's
  // piece number (seg_a >> 4s) & 15 by B's piece number (seg_b >> 4s) & 15; a block's products meet in one
  // accumulator, the blocks' accumulators in f32 registers.  K = 64 * seg_blocks * segs.  0: a plain product.
  uint32_t seg_blocks = 0, segs = 0, seg_a = 0, seg_b = 0;
  // The operands the pieces were cut from.  Pieces of a value that is not finite, or larger than the largest bf16,
  // do not add up to it; an output that is not finite is therefore made again from these, one multiply-add after
  // the other.
  const float* src_a = nullptr;        // [M, src_k], or [src_k, M] (src_a_t)
  const void* src_b = nullptr;         // [src_k, N], or [N, src_k] (src_b_t)
  const float* src_a_scale = nullptr;  // of column k of A, or null
  uint32_t src_k = 0;
  int src_a_t = 0, src_b_t = 0;
  BType src_b_type = BType::kF32;
};

// The operands of a launch, per product: a, a2: bf16 [M, K] row-major, box {64, 128}, 128-byte swizzle; b, b2: bf16
// [N, K], box {64, plan.b_box}; a2 and b2 the low-rank term's (any valid map where there is none).
struct UmmaMaps { CUtensorMap a[kUmmaProducts], b[kUmmaProducts], a2[kUmmaProducts], b2[kUmmaProducts]; };

// Which kernel takes a product, on which tiles (k_gemm_umma.cu).
struct UmmaGemmPlan {
  bool persistent = false, pair = false;
  uint32_t tn = 0;          // tile width
  uint32_t splits = 1;      // tile kernel: CTAs that share a tile's reduction
  uint32_t grid = 0, band = 1;
  uint32_t b_box = 0;       // rows of B one TMA load brings: the box height of map_b and aux_b
  double us = 0.0;          // the estimate it was chosen by
};
// k_blocks: 64-wide blocks of the whole reduction, a low-rank term's included; `group` of them in a row (1: any) are
// not cut.  light: the epilogue only stores (f32 or a bf16 copy), without a second operand, bias or activation.
// side_by_side: outputs of this shape in the launch.  only_splits != 0: with the reduction cut that often.  chained: k_blocks are
// a chain's, whose reductions are each cut (tn up to 128 only where they are).  No such plan: us = 1e30.
UmmaGemmPlan UmmaPlanGemm(uint32_t M, uint32_t N, uint32_t k_blocks, uint32_t group, bool light, uint32_t sms,
                          uint32_t side_by_side = 1, uint32_t only_splits = 0, bool chained = false);
cudaError_t UmmaGemmLaunch(const UmmaGemmPlan& plan, const UmmaMaps& maps, const UmmaEpilogue& ep, cudaStream_t s);
// Piece products of an f32 activation that the kernel cuts itself (k_gemm_cut.cu; UmmaEpilogue::src_a, src_k and
// src_a_scale are its operand): groups = blocks of 64 k.  grid == 0: the piece form is the faster one.
// parts: chains of additions that K is summed in (a multiple of splits, or fewer).
struct UmmaCutPlan { uint32_t tn = 64, splits = 1, grid = 0, parts = 1; };
UmmaCutPlan UmmaPlanCut(uint32_t M, uint32_t N, uint32_t groups, bool exact_b, uint32_t sms);
// map_b: bf16 [N, 3 Kp] or, exact, [N, K], box {64, plan.tn}.
cudaError_t UmmaCutLaunch(const UmmaCutPlan& plan, bool exact_b, const CUtensorMap& map_b, const UmmaEpilogue& ep, cudaStream_t s);
// Large products run on CTA pairs (cta_group::2) by default; off = one CTA per tile.  Process-wide.
void UmmaSetCtaPairs(bool on);
// dst[N][K] (bf16 bits) from src [K][N] (transpose) or [N][K]; int8 and bf16 widen exactly.
// k_scale (or null): dst[n][k] = bf16(src * k_scale[k]).
void WeightToBf16(const void* src, BType type, uint16_t* dst, uint32_t N, uint32_t K,
                  bool transpose, const float* k_scale, cudaStream_t s);

}  // namespace see::k

#endif  // SEE_CUDA_UMMA_KERNEL_H_
