// What a tensor-core GEMM does with its accumulators on the way out: scale, addend, bias, activation, absorbed
// activations and operand copies, and the products of operands whose pieces do not add up to them.  Shared by the
// kernels on bf16 operands (k_gemm_umma.cu) and the ones that cut f32 operands themselves (k_gemm_cut.cu); both are
// compiled without fused multiply-add contraction.
#ifndef SEE_CUDA_UMMA_EPILOGUE_CUH_
#define SEE_CUDA_UMMA_EPILOGUE_CUH_

#include "act_expr.cuh"
#include "kernels.h"
#include "shadow.cuh"
#include "umma_kernel.h"

namespace see::k::umma_epi {

__device__ __forceinline__ float ApplyAct(float v, int act) { return ActFwdExpr(act, v); }

// The tail of both epilogues: four neighbouring columns n.. of row (at / N).
__device__ __forceinline__ void EpilogueStore(const UmmaEpilogue& ep, size_t at, uint32_t n, const float4& acc,
                                              const float4& scale, const float4& bias,
                                              bool has_kscale = false,
                                              float4 kscale = make_float4(1.f, 1.f, 1.f, 1.f),
                                              bool has_side = false,   // the addend / x element, already loaded
                                              float4 side = make_float4(0.f, 0.f, 0.f, 0.f)) {
  float4 v = make_float4(acc.x * scale.x, acc.y * scale.y, acc.z * scale.z, acc.w * scale.w);
  if (ep.addend && !ep.addend_last) {
    const float4 d = has_side ? side : __ldg(reinterpret_cast<const float4*>(ep.addend + at));
    v = make_float4(d.x + v.x, d.y + v.y, d.z + v.z, d.w + v.w);
  }
  if (ep.bias) v = make_float4(v.x + bias.x, v.y + bias.y, v.z + bias.z, v.w + bias.w);
  if (ep.addend && ep.addend_last) {   // an absorbed kAddEW that followed the kAddBias
    const float4 d = has_side ? side : __ldg(reinterpret_cast<const float4*>(ep.addend + at));
    v = make_float4(d.x + v.x, d.y + v.y, d.z + v.z, d.w + v.w);
  }
  if (ep.act != kActNone)
    v = make_float4(ApplyAct(v.x, ep.act), ApplyAct(v.y, ep.act), ApplyAct(v.z, ep.act),
                    ApplyAct(v.w, ep.act));
  if (ep.store_c) *reinterpret_cast<float4*>(ep.C + at) = v;
  if (ep.pack_dst) {   // the bf16 operand copy a tiled attention instruction reads this tensor through
    uint32_t lo, hi;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(v.y), "f"(v.x));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(v.w), "f"(v.z));
    *reinterpret_cast<uint2*>(ep.pack_dst + at) = make_uint2(lo, hi);
  }
  if (ep.fuse_mode != kFuseNone) {
    float4 g;
    if (ep.fuse_mode == kFuseActFwd) {
      if (ep.fuse_act == kActGelu) {   // two elements per instruction; the bits of GeluExpr
        UnpackF2(GeluExpr2(PackF2(v.x, v.y)), &g.x, &g.y);
        UnpackF2(GeluExpr2(PackF2(v.z, v.w)), &g.z, &g.w);
      } else {
        g = make_float4(ActFwdExpr(ep.fuse_act, v.x), ActFwdExpr(ep.fuse_act, v.y),
                        ActFwdExpr(ep.fuse_act, v.z), ActFwdExpr(ep.fuse_act, v.w));
      }
    } else {
      const float4 x = has_side ? side : __ldg(reinterpret_cast<const float4*>(ep.fuse_x + at));
      if (ep.fuse_act == kActGelu) {   // likewise, the bits of GeluGrad
        UnpackF2(GeluGrad2(PackF2(v.x, v.y), PackF2(x.x, x.y)), &g.x, &g.y);
        UnpackF2(GeluGrad2(PackF2(v.z, v.w), PackF2(x.z, x.w)), &g.z, &g.w);
      } else {
        g = make_float4(ActBwdExpr(ep.fuse_act, v.x, x.x), ActBwdExpr(ep.fuse_act, v.y, x.y),
                        ActBwdExpr(ep.fuse_act, v.z, x.z), ActBwdExpr(ep.fuse_act, v.w, x.w));
      }
    }
    Shadow sh;
    sh.dst = ep.shadow_dst;
    sh.k_scale = has_kscale ? nullptr : ep.shadow_k_scale;
    sh.cols = ep.N;
    if (has_kscale) g = make_float4(g.x * kscale.x, g.y * kscale.y, g.z * kscale.z, g.w * kscale.w);
    ShadowStore4(sh, at / 4, n, g);
  }
}

// EpilogueStore for the one form in which instruction count bounds the whole kernel: an absorbed GELU
// gradient and nothing else (no addend, bias, activation or attention copy).  The same values, without
// the per-element tests of the general form.
__device__ __forceinline__ bool IsGeluGradOnly(const UmmaEpilogue& ep) {
  return ep.fuse_mode == kFuseActBwd && ep.fuse_act == kActGelu && ep.addend == nullptr && ep.bias == nullptr &&
         ep.act == kActNone && ep.pack_dst == nullptr;
}
__device__ __forceinline__ void EpilogueStoreGeluGrad(const UmmaEpilogue& ep, size_t at, const float4& acc,
                                                      const float4& scale, const float4& kscale, const float4& x) {
  const float4 v = make_float4(acc.x * scale.x, acc.y * scale.y, acc.z * scale.z, acc.w * scale.w);
  if (ep.store_c) *reinterpret_cast<float4*>(ep.C + at) = v;
  float4 g;
  UnpackF2(GeluGrad2(PackF2(v.x, v.y), PackF2(x.x, x.y)), &g.x, &g.y);
  UnpackF2(GeluGrad2(PackF2(v.z, v.w), PackF2(x.z, x.w)), &g.z, &g.w);
  uint2 r;
  r.x = ShadowBf16x2(g.x * kscale.x, g.y * kscale.y);
  r.y = ShadowBf16x2(g.z * kscale.z, g.w * kscale.w);
  reinterpret_cast<uint2*>(ep.shadow_dst)[at >> 2] = r;
}

// Likewise for an addend and nothing else (the accumulating gradient products): C = addend + acc * scale.
__device__ __forceinline__ bool IsAddendOnly(const UmmaEpilogue& ep) {
  return ep.addend != nullptr && ep.bias == nullptr && ep.act == kActNone && ep.pack_dst == nullptr &&
         ep.fuse_mode == kFuseNone && ep.store_c;
}
__device__ __forceinline__ void EpilogueStoreAddend(const UmmaEpilogue& ep, size_t at, const float4& acc,
                                                    const float4& scale, const float4& d) {
  *reinterpret_cast<float4*>(ep.C + at) =
      make_float4(d.x + acc.x * scale.x, d.y + acc.y * scale.y, d.z + acc.z * scale.z, d.w + acc.w * scale.w);
}
// ... for a product that leaves only as the bf16 copy a tiled attention instruction reads (Q, K, V) ...
__device__ __forceinline__ bool IsCopyOnly(const UmmaEpilogue& ep) {
  return ep.addend == nullptr && ep.bias == nullptr && ep.act == kActNone && ep.pack_dst != nullptr &&
         ep.fuse_mode == kFuseNone && !ep.store_c;
}
__device__ __forceinline__ void EpilogueStoreCopy(uint16_t* pack_dst, size_t at, const float4& acc,
                                                  const float4& scale) {
  uint32_t lo, hi;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(lo) : "f"(acc.y * scale.y), "f"(acc.x * scale.x));
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(acc.w * scale.w), "f"(acc.z * scale.z));
  *reinterpret_cast<uint2*>(pack_dst + at) = make_uint2(lo, hi);
}
// ... for a product stored as it is (the vocabulary head, the gradient products that carry nothing else) ...
__device__ __forceinline__ bool IsPlainStore(const UmmaEpilogue& ep) {
  return ep.addend == nullptr && ep.bias == nullptr && ep.act == kActNone && ep.pack_dst == nullptr &&
         ep.fuse_mode == kFuseNone && ep.store_c;
}
__device__ __forceinline__ void EpilogueStorePlain(const UmmaEpilogue& ep, size_t at, const float4& acc,
                                                   const float4& scale) {
  *reinterpret_cast<float4*>(ep.C + at) =
      make_float4(acc.x * scale.x, acc.y * scale.y, acc.z * scale.z, acc.w * scale.w);
}
// ... and for a bias followed by an absorbed GELU (the feed-forward up product): C = acc * scale + bias,
// the bf16 operand copy of gelu(C) beside it.
__device__ __forceinline__ bool IsBiasGeluOnly(const UmmaEpilogue& ep) {
  return ep.addend == nullptr && ep.bias != nullptr && ep.act == kActNone && ep.pack_dst == nullptr &&
         ep.fuse_mode == kFuseActFwd && ep.fuse_act == kActGelu && ep.store_c;
}
__device__ __forceinline__ void EpilogueStoreBiasGelu(const UmmaEpilogue& ep, size_t at, const float4& acc,
                                                      const float4& scale, const float4& bias, const float4& kscale) {
  float4 v = make_float4(acc.x * scale.x, acc.y * scale.y, acc.z * scale.z, acc.w * scale.w);
  v = make_float4(v.x + bias.x, v.y + bias.y, v.z + bias.z, v.w + bias.w);
  *reinterpret_cast<float4*>(ep.C + at) = v;
  float4 g;
  UnpackF2(GeluExpr2(PackF2(v.x, v.y)), &g.x, &g.y);
  UnpackF2(GeluExpr2(PackF2(v.z, v.w)), &g.z, &g.w);
  uint2 r;
  r.x = ShadowBf16x2(g.x * kscale.x, g.y * kscale.y);
  r.y = ShadowBf16x2(g.z * kscale.z, g.w * kscale.w);
  reinterpret_cast<uint2*>(ep.shadow_dst)[at >> 2] = r;
}

// Exact products that absorbed what follows them: C = acc * scale + bias, or the GELU of that.  Their sums leave the epilogue
// warps no time under the next tile's products, so the general form's tests per element were the whole tail (4096 x 3072 x 768 of
// an int8 weight, plain 63 us: a bias 68.0 / 63.8, with a GELU 80.1 / 68.0; 4096 x 1024 x 256 of f32, plain 17.1: 22.8 / 18.8, 29.9 / 22.0).
__device__ __forceinline__ bool IsBiasStored(const UmmaEpilogue& ep, int act) {
  return ep.addend == nullptr && ep.bias != nullptr && ep.act == act && ep.pack_dst == nullptr && ep.fuse_mode == kFuseNone &&
         ep.store_c;
}
template <int kAct>
__device__ __forceinline__ void EpilogueStoreBias(const UmmaEpilogue& ep, size_t at, const float4& acc, const float4& scale,
                                                  const float4& bias) {
  float4 v = make_float4(acc.x * scale.x, acc.y * scale.y, acc.z * scale.z, acc.w * scale.w);
  v = make_float4(v.x + bias.x, v.y + bias.y, v.z + bias.z, v.w + bias.w);
  if constexpr (kAct == kActGelu) {   // (the bits of GeluExpr)
    UnpackF2(GeluExpr2(PackF2(v.x, v.y)), &v.x, &v.y);
    UnpackF2(GeluExpr2(PackF2(v.z, v.w)), &v.z, &v.w);
  }
  *reinterpret_cast<float4*>(ep.C + at) = v;
}

// ... or an addition, before a bias or after it (the same shapes: 98.3 / 95.7, 23.5 / 20.9).
__device__ __forceinline__ bool IsSum(const UmmaEpilogue& ep) {
  return ep.addend != nullptr && ep.act == kActNone && ep.pack_dst == nullptr && ep.fuse_mode == kFuseNone && ep.store_c;
}
__device__ __forceinline__ void EpilogueStoreSum(const UmmaEpilogue& ep, size_t at, const float4& acc, const float4& scale,
                                                 const float4& bias, const float4& d) {
  float4 v = make_float4(acc.x * scale.x, acc.y * scale.y, acc.z * scale.z, acc.w * scale.w);
  if (!ep.addend_last) v = make_float4(d.x + v.x, d.y + v.y, d.z + v.z, d.w + v.w);
  if (ep.bias) v = make_float4(v.x + bias.x, v.y + bias.y, v.z + bias.z, v.w + bias.w);
  if (ep.addend_last) v = make_float4(d.x + v.x, d.y + v.y, d.z + v.z, d.w + v.w);
  *reinterpret_cast<float4*>(ep.C + at) = v;
}

// Four neighbouring columns of one row of an output whose width is no multiple of four (an odd vocabulary): rows
// start at any 4-byte boundary, so everything moves one element at a time.  No absorbed activation, no copy.
__device__ __forceinline__ void EpilogueStoreRagged(const UmmaEpilogue& ep, size_t row, uint32_t n, const float4& acc,
                                                    bool scaled) {
  const float a[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
  for (uint32_t e = 0; e < 4; ++e) {
    if (n + e >= ep.N) continue;
    const size_t at = row * ep.N + n + e;
    float v = scaled ? a[e] : a[e] * (ep.col_scale ? ep.col_scale[n + e] : ep.alpha);
    if (ep.addend && !ep.addend_last) v = ep.addend[at] + v;
    if (ep.bias) v = v + ep.bias[n + e];
    if (ep.addend && ep.addend_last) v = ep.addend[at] + v;
    if (ep.act != kActNone) v = ApplyAct(v, ep.act);
    ep.C[at] = v;
  }
}

// Piece products whose sum is not finite (UmmaEpilogue::src_a), scaled where the CUDA-core kernels scale: alpha on A's
// elements and col_scale on B's, or alpha on the sum where B is [N, K].  A warp's lanes ask for neighbouring columns of a row,
// so this walks A by broadcasts and B, stored [K, N], by whole lines; nothing calls it while all values are finite.
__device__ __forceinline__ float4 DotsFromSource(const UmmaEpilogue& ep, size_t row, uint32_t n) {
  const size_t K = ep.src_k, N = ep.N;
  float v[4];
#pragma unroll
  for (uint32_t e = 0; e < 4; ++e) v[e] = n + e < ep.N ? 0.0f : __uint_as_float(0x7FC00000u);
  for (size_t k = 0; k < K; ++k) {
    float a = ep.src_a[ep.src_a_t ? k * ep.M + row : row * K + k];
    if (ep.src_a_scale) a = a * ep.src_a_scale[k];
    if (!ep.src_b_t && !ep.col_scale) a = ep.alpha * a;
#pragma unroll
    for (uint32_t e = 0; e < 4; ++e) {
      if (n + e >= ep.N) continue;
      const size_t at = ep.src_b_t ? (n + e) * K + k : k * N + n + e;
      float b = ep.src_b_type == BType::kF32   ? static_cast<const float*>(ep.src_b)[at]
                : ep.src_b_type == BType::kI8 ? static_cast<float>(static_cast<const int8_t*>(ep.src_b)[at])
                                              : __uint_as_float(static_cast<uint32_t>(static_cast<const uint16_t*>(ep.src_b)[at]) << 16);
      if (ep.col_scale) b = b * ep.col_scale[n + e];
      v[e] = v[e] + a * b;
    }
    if (v[0] != v[0] && v[1] != v[1] && v[2] != v[2] && v[3] != v[3]) break;   // NaN for good: a diverged run's rows end at once
  }
  const float after = ep.src_b_t && !ep.col_scale ? ep.alpha : 1.0f;
  return make_float4(after * v[0], after * v[1], after * v[2], after * v[3]);
}
// True: *acc held a value that is not finite and now holds the scaled products.
__device__ __forceinline__ bool Remade(const UmmaEpilogue& ep, size_t row, uint32_t n, float4* acc) {
  const float zero = (acc->x * 0.0f + acc->y * 0.0f) + (acc->z * 0.0f + acc->w * 0.0f);   // NaN unless all are finite
  if (zero == 0.0f) return false;
  *acc = DotsFromSource(ep, row, n);
  return true;
}
// Four outputs of a tile in which some sum is not finite: made again where they are the ones.
static __device__ __noinline__ void StoreRemade(const UmmaEpilogue& ep, size_t row, uint32_t n, float4 acc) {
  const bool made = Remade(ep, row, n, &acc);
  if ((ep.N & 3u) != 0) { EpilogueStoreRagged(ep, row, n, acc, made); return; }
  float4 scale = make_float4(ep.alpha, ep.alpha, ep.alpha, ep.alpha), bias = make_float4(0.f, 0.f, 0.f, 0.f);
  if (ep.col_scale) scale = __ldg(reinterpret_cast<const float4*>(ep.col_scale + n));
  if (made) scale = make_float4(1.f, 1.f, 1.f, 1.f);
  if (ep.bias) bias = __ldg(reinterpret_cast<const float4*>(ep.bias + n));
  EpilogueStore(ep, row * ep.N + n, n, acc, scale, bias);
}
template <uint32_t kCount>
__device__ __forceinline__ bool AllFinite(const float (&v)[kCount]) {
  float zero[4] = {0.0f, 0.0f, 0.0f, 0.0f};   // NaN once something is not
#pragma unroll
  for (uint32_t j = 0; j < kCount; ++j) zero[j & 3] = fmaf(v[j], 0.0f, zero[j & 3]);
  return (zero[0] + zero[1]) + (zero[2] + zero[3]) == 0.0f;
}
__device__ __forceinline__ uint32_t LoadClusterU32(uint32_t cluster_addr) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cluster_addr));
  return v;
}
__device__ __forceinline__ float4 LoadClusterF4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr));
  return v;
}

}  // namespace see::k::umma_epi

#endif  // SEE_CUDA_UMMA_EPILOGUE_CUH_
