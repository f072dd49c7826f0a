// f32 products too small or too narrow for the tensor cores, where the plan does
// not observe the bits (engine mode): the rank-r products of an adapter at any
// width, the layers of a feed-forward plan at a batch of a few dozen.
//
//     C = act(addend + alpha op(A) op(B) + bias)
//
// Fused multiply-adds in f32, in an order that is a function of the shape alone.
//
// What bounds such a product is latency: a few thousand outputs, each a reduction
// of hundreds to thousands of terms.  So the reduction is cut twice: over the CTAs
// of a cluster (up to eight, as many as bring the grid to one CTA per SM), and
// inside a CTA over its eight warps.  A CTA's operand slices arrive by cp.async, 128 k
// at a time in two buffers, in the layout they have in memory; each warp holds the
// whole output tile in registers (RM x RN per lane) for its eighth of the chunk's
// k.  The eight partial tiles are added in warp order through shared memory, the
// CTAs' in rank order through distributed shared memory.
// Wide activations streamed through a narrow product (t = x A at thousands of rows)
// are HBM-bound on the same kernel: one pass over x.
//
// Measured on a B200, us, before (one 64 x 64 or 256 x 16 tile per CTA, K serial) / now:
// 32 x 1024 x 256 24.6 / 4; 32 x 64 x 1024 88.8 / 5.2; 600 x 8 x 512 70 / 4.3; 4096 x 8 x
// 4096 944 / 26.  (Gradients of a rank-r factor over many rows stream: cuda_backend.cc.)
#include <algorithm>
#include <atomic>

#include "gemm_exact_common.cuh"
#include "launch.cuh"
#include "umma_device.cuh"

namespace see::k {

namespace {

using exact::ApplyAct;

constexpr int kThreads = 256;
constexpr int kWarps = 8;
constexpr int kChunk = 128;   // k per buffer

struct FastParams {
  const float* A; const float* B; float* C;
  int M, N, K;
  float alpha;
  const float* bias; const float* addend;
  int act;
  int per_split;   // k of one CTA of the cluster, a multiple of 4
};

__device__ __forceinline__ void CpAsync16(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
               ::"r"(umma_dev::SmemAddr(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void CpAsync4(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;"
               ::"r"(umma_dev::SmemAddr(dst)), "l"(src), "r"(bytes) : "memory");
}

// Rows [r0, r0 + kRows) x columns [c0, c0 + kCols) of a row-major [rows][cols] matrix into dst[kRows][kLd];
// what lies outside (columns past c_end too) is zero.
template <int kRows, int kCols, int kLd>
__device__ __forceinline__ void CopyTile(float* dst, const float* src, int rows, int cols, int r0, int c0, int r_end,
                                         int c_end, bool vec) {
  if (vec) {   // cols % 4 == 0 and c_end % 4 == 0: four columns are all in or all out
    for (int i = threadIdx.x; i < kRows * (kCols / 4); i += kThreads) {
      const int r = i / (kCols / 4), c = i % (kCols / 4) * 4;
      const bool in = r0 + r < r_end && c0 + c < c_end;
      CpAsync16(dst + r * kLd + c, in ? src + static_cast<size_t>(r0 + r) * cols + c0 + c : src, in ? 16 : 0);
    }
  } else {
    for (int i = threadIdx.x; i < kRows * kCols; i += kThreads) {
      const int r = i / kCols, c = i % kCols;
      const bool in = r0 + r < r_end && c0 + c < c_end;
      CpAsync4(dst + r * kLd + c, in ? src + static_cast<size_t>(r0 + r) * cols + c0 + c : src, in ? 4 : 0);
    }
  }
}

enum FastMode { kNN = 0, kNT = 1, kTN = 2 };

// LM x LN lanes, RM x RN outputs each.  Lane rows are lm + LM i (so that a quarter warp's 16-byte reads along k hit
// different banks), lane columns ln RN + j.
template <int kMode, int LM, int LN, int RM, int RN>
struct FastTile {
  static constexpr int TM = LM * RM, TN = LN * RN;
  // natural layouts: A [m][k] or [k][m]; B [k][n] or [n][k]
  static constexpr int kALd = kMode == kTN ? TM + 4 : kChunk + 4;
  static constexpr int kARows = kMode == kTN ? kChunk : TM;
  static constexpr int kBLd = kMode == kNT ? kChunk + 4 : TN + 4;
  static constexpr int kBRows = kMode == kNT ? TN : kChunk;
  static constexpr int kBuffer = kARows * kALd + kBRows * kBLd;   // floats
  static constexpr int kOut = TM * TN;
  static constexpr int kFloats = 2 * kBuffer > kWarps * kOut + kOut ? 2 * kBuffer : kWarps * kOut + kOut;
};

template <int kMode, int LM, int LN, int RM, int RN>
__global__ void __launch_bounds__(kThreads) FastGemmKernel(FastParams p) {
  AwaitPrevious();
  using T = FastTile<kMode, LM, LN, RM, RN>;
  constexpr int TM = T::TM, TN = T::TN;
  extern __shared__ __align__(16) float smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lm = lane % LM, ln = lane / LM;
  const uint32_t rank = umma_dev::ClusterCtaRank();
  uint32_t splits;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(splits));
  const int tiles_n = (p.N + TN - 1) / TN, tile = static_cast<int>(blockIdx.x / splits);
  const int m0 = tile / tiles_n * TM, n0 = tile % tiles_n * TN;
  const int kb = static_cast<int>(rank) * p.per_split, ke = min(p.K, kb + p.per_split);
  const bool a_vec = (((kMode == kTN ? p.M : p.K) & 3) == 0) && (reinterpret_cast<uintptr_t>(p.A) & 15) == 0;
  const bool b_vec = (((kMode == kNT ? p.K : p.N) & 3) == 0) && (reinterpret_cast<uintptr_t>(p.B) & 15) == 0;

  auto load = [&](int k0, int buf) {
    float* as = smem + buf * T::kBuffer;
    float* bs = as + T::kARows * T::kALd;
    // (a k range ends at a multiple of 4 or at K)
    if (kMode == kTN) CopyTile<kChunk, TM, T::kALd>(as, p.A, p.K, p.M, k0, m0, ke, p.M, a_vec);
    else CopyTile<TM, kChunk, T::kALd>(as, p.A, p.M, p.K, m0, k0, p.M, ke, a_vec);
    if (kMode == kNT) CopyTile<TN, kChunk, T::kBLd>(bs, p.B, p.N, p.K, n0, k0, p.N, ke, b_vec);
    else CopyTile<kChunk, TN, T::kBLd>(bs, p.B, p.K, p.N, k0, n0, ke, p.N, b_vec);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float acc[RM][RN];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; ++j) acc[i][j] = 0.0f;

  int buf = 0;
  if (kb < ke) load(kb, 0);
  for (int k0 = kb; k0 < ke; k0 += kChunk, buf ^= 1) {
    if (k0 + kChunk < ke) {
      load(k0 + kChunk, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const float* as = smem + buf * T::kBuffer;
    const float* bs = as + T::kARows * T::kALd;
    // This warp's slice of the chunk, a multiple of 4 (zeros past the end of k).
    const int len = min(kChunk, ke - k0), slice = (len + 4 * kWarps - 1) / (4 * kWarps) * 4;
    const int s0 = warp * slice, s1 = min(len, s0 + slice);
    for (int k = s0; k < s1; k += 4) {
      float a[RM][4], b[4][RN];
      if (kMode == kTN) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int i = 0; i < RM; ++i) a[i][q] = as[(k + q) * T::kALd + lm + LM * i];
      } else {
#pragma unroll
        for (int i = 0; i < RM; ++i) {
          const float4 v = *reinterpret_cast<const float4*>(as + (lm + LM * i) * T::kALd + k);
          a[i][0] = v.x; a[i][1] = v.y; a[i][2] = v.z; a[i][3] = v.w;
        }
      }
      if (kMode == kNT) {
#pragma unroll
        for (int j = 0; j < RN; ++j) {
          const float4 v = *reinterpret_cast<const float4*>(bs + (ln * RN + j) * T::kBLd + k);
          b[0][j] = v.x; b[1][j] = v.y; b[2][j] = v.z; b[3][j] = v.w;
        }
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int j = 0; j < RN; j += 4) {
            const float4 v = *reinterpret_cast<const float4*>(bs + (k + q) * T::kBLd + ln * RN + j);
            b[q][j] = v.x; b[q][j + 1] = v.y; b[q][j + 2] = v.z; b[q][j + 3] = v.w;
          }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
          for (int j = 0; j < RN; ++j) acc[i][j] = fmaf(a[i][q], b[q][j], acc[i][j]);
    }
    __syncthreads();   // the buffer is refilled two chunks on
  }

  // The eight warps' partial tiles, added in warp order into out[].
  float* red = smem;
  float* out = smem + kWarps * T::kOut;
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN; j += 4)
      *reinterpret_cast<float4*>(red + warp * T::kOut + (lm + LM * i) * TN + ln * RN + j) =
          make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
  __syncthreads();
  for (int i = threadIdx.x; i < T::kOut; i += kThreads) {
    float s = red[i];
#pragma unroll
    for (int w = 1; w < kWarps; ++w) s += red[w * T::kOut + i];
    out[i] = s;
  }
  if (splits > 1) umma_dev::ClusterSync();
  else __syncthreads();
  // Each CTA finishes its share of the tile's outputs.
  const int share = (T::kOut + static_cast<int>(splits) - 1) / static_cast<int>(splits);
  const int o_begin = static_cast<int>(rank) * share, o_end = min(T::kOut, o_begin + share);
  const uint32_t out_addr = umma_dev::SmemAddr(out);
  for (int i = o_begin + static_cast<int>(threadIdx.x); i < o_end; i += kThreads) {
    const int m = m0 + i / TN, n = n0 + i % TN;
    if (m >= p.M || n >= p.N) continue;
    float v;
    if (splits == 1) {
      v = out[i];
    } else {
      float part[8];
#pragma unroll
      for (uint32_t r = 0; r < 8; ++r)
        if (r < splits)
          asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(part[r]) : "r"(umma_dev::MapToCta(out_addr + i * 4, r)));
      v = part[0];
#pragma unroll
      for (uint32_t r = 1; r < 8; ++r)
        if (r < splits) v += part[r];
    }
    v *= p.alpha;
    const size_t at = static_cast<size_t>(m) * p.N + n;
    if (p.addend) v = p.addend[at] + v;
    if (p.bias) v = v + p.bias[n];
    p.C[at] = ApplyAct(v, static_cast<Act>(p.act));
  }
  if (splits > 1) umma_dev::ClusterSync();   // no CTA leaves while another may still read its sums
}

template <int kMode, int LM, int LN, int RM, int RN>
bool Launch(FastParams p, cudaStream_t s) {
  using T = FastTile<kMode, LM, LN, RM, RN>;
  constexpr size_t smem = sizeof(float) * T::kFloats;
  static std::atomic<bool> configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  const bool tracked = dev >= 0 && dev < 64;
  if (!tracked || !configured[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(FastGemmKernel<kMode, LM, LN, RM, RN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(smem)) != cudaSuccess)
      return false;
    if (tracked) configured[dev].store(true, std::memory_order_release);
  }
  const long tiles = static_cast<long>((p.M + T::TM - 1) / T::TM) * ((p.N + T::TN - 1) / T::TN);
  // As many CTAs per tile as bring the grid to one per SM, at least 32 k each; a whole number of k quads.
  int splits = 1;
  while (splits < 8 && tiles * splits * 2 <= 148 + 74 && p.K >= splits * 2 * 32) splits *= 2;
  p.per_split = ((p.K + splits - 1) / splits + 3) / 4 * 4;
  return Next(FastGemmKernel<kMode, LM, LN, RM, RN>, static_cast<unsigned>(tiles * splits), kThreads, smem, s, static_cast<unsigned>(splits))(p) == cudaSuccess;
}

// The tile whose narrow side fits the output's: 64 x 8 and 64 x 16 for rank-wide results, 8 x 64 and 16 x 64 for
// rank-tall ones, 32 x 32 otherwise.
template <int kMode>
bool LaunchMode(const FastParams& p, cudaStream_t s) {
  if (p.N <= 8) return Launch<kMode, 16, 2, 4, 4>(p, s);
  if (p.N <= 16) return Launch<kMode, 16, 2, 4, 8>(p, s);
  if (p.M <= 8) return Launch<kMode, 2, 16, 4, 4>(p, s);
  if (p.M <= 16) return Launch<kMode, 4, 8, 4, 8>(p, s);
  return Launch<kMode, 8, 4, 4, 8>(p, s);
}

}  // namespace

bool FastGemm(const GemmArgs& a, cudaStream_t s) {
  if (a.b_type != BType::kF32 || a.accumulate || a.b_col_scale || a.a_k_scale || a.M == 0 || a.N == 0 || a.K == 0) return false;
  if (a.M > 0x3FFFFFFF || a.N > 0x3FFFFFFF || a.K > 0x3FFFFFFF) return false;
  if ((a.M + 7) / 8 * ((a.N + 7) / 8) > 0x7FFFFFF) return false;
  const FastParams p{a.A, static_cast<const float*>(a.B), a.C, static_cast<int>(a.M), static_cast<int>(a.N),
                     static_cast<int>(a.K), a.alpha, a.bias, a.addend, static_cast<int>(a.act), 0};
  if (a.a_transposed) return LaunchMode<kTN>(p, s);
  if (a.b_transposed) return LaunchMode<kNT>(p, s);
  return LaunchMode<kNN>(p, s);
}

}  // namespace see::k
