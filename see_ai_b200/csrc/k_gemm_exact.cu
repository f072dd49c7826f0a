// The exact GEMM family on CUDA cores: reproduces the CPU executor's two
// reduction contracts bit for bit, for f32, int8 and bf16 weights.
//
//   quad order (NN, TN, AccNN and their narrow-weight forms; reference:
//     runtime/executor/gemm.cc:73-187): per element, from c = 0 (or the
//     existing C for the accumulate form),
//         c += ((a0*b0 + a1*b1) + a2*b2) + a3*b3
//     over consecutive k-quads aligned to k = 0, then one term at a time for
//     the K % 4 tail; alpha (or the per-tensor dequant scale) is multiplied
//     into each A element first, a per-column scale into each widened B element.
//   lane order (NT forms; reference: runtime/executor/gemm.cc:346-527): eight
//     accumulators, product k into lane k mod 8, lanes summed 0..7, the result
//     times alpha; a reduction-axis scale is multiplied into A first.
//
// Epilogue order matches the reference (gemm.cc:536-578): addend `d + s` on
// the finished sum, then bias, then the activation expression.  Compiled with
// -fmad=false; no multiply is ever fused into an add.  This family is the
// parity anchor and the path for the rank-r adapter products, whose outputs are
// 8-16 wide (or tall): the block tile comes in three shapes (64x64, 256x16,
// 16x256 for the quad order; 64x32, 128x16, 16x128 for the lane order) picked
// from the output shape, so a skinny product wastes no lanes, and a flat form
// (GemmFlatKernel) for outputs of too few tiles.  A tile shape
// changes which thread owns an element, never the element's arithmetic.
// Large frozen-weight products carrying the relaxed permission go to the
// tensor cores instead.
#include <algorithm>

#include "gemm_exact_common.cuh"
#include "launch.cuh"

namespace see::k {

namespace {

using namespace exact;

constexpr int BK = 16;
constexpr int kThreads = 256;

template <bool TA>
__device__ __forceinline__ float LoadA(const Params& p, size_t m, size_t k) {
  if (m >= p.M || k >= p.K) return 0.0f;
  return TA ? p.A[k * p.M + m] : p.A[m * p.K + k];
}
template <bool TB, typename BT>
__device__ __forceinline__ float LoadB(const Params& p, size_t k, size_t n) {
  if (n >= p.N || k >= p.K) return 0.0f;
  const BT* B = static_cast<const BT*>(p.B);
  return Widen<BT>(TB ? B[n * p.K + k] : B[k * p.N + n]);
}

// ---- quad order: BM x BN tile (BM * BN = 4096), 256 threads, 4x4 outputs per thread ----
template <bool TA, typename BT, int BM, int BN>
__global__ void __launch_bounds__(kThreads) GemmQuadKernel(Params p) {
  AwaitPrevious();
  static_assert(BM * BN == 16 * kThreads, "4x4 outputs per thread");
  __shared__ __align__(16) float As[BK][BM + 4];
  __shared__ __align__(16) float Bs[BK][BN + 4];
  const int tx = threadIdx.x % (BN / 4), ty = threadIdx.x / (BN / 4);
  const size_t m0 = static_cast<size_t>(blockIdx.y) * BM, n0 = static_cast<size_t>(blockIdx.x) * BN;
  float c[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const size_t m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
      c[i][j] = (p.accumulate && m < p.M && n < p.N) ? p.C[m * p.N + n] : 0.0f;
    }
  const bool a_vec = (reinterpret_cast<uintptr_t>(p.A) & 15) == 0 && ((TA ? p.M : p.K) & 3) == 0;
  const size_t k_begin = p.k_chunk ? static_cast<size_t>(blockIdx.z) * p.k_chunk : 0;
  const size_t k_end = p.k_chunk ? (k_begin + p.k_chunk < p.K ? k_begin + p.k_chunk : p.K) : p.K;
  for (size_t k0 = k_begin; k0 < k_end; k0 += BK) {
    // Stage the tiles; alpha and the column scale are applied here, once per
    // element, as the reference applies them when an element enters the product.
    if (a_vec) {  // 16-byte global loads along A's contiguous axis
#pragma unroll
      for (int idx = threadIdx.x; idx < BM * BK / 4; idx += kThreads) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (TA) {
          const int kk = idx / (BM / 4), mm = (idx % (BM / 4)) * 4;
          if (m0 + mm < p.M && k0 + kk < p.K)
            v = *reinterpret_cast<const float4*>(p.A + (k0 + kk) * p.M + m0 + mm);
          *reinterpret_cast<float4*>(&As[kk][mm]) =
              make_float4(p.alpha * v.x, p.alpha * v.y, p.alpha * v.z, p.alpha * v.w);
        } else {
          const int mm = idx / (BK / 4), kk = (idx % (BK / 4)) * 4;
          if (m0 + mm < p.M && k0 + kk < p.K)
            v = *reinterpret_cast<const float4*>(p.A + (m0 + mm) * p.K + k0 + kk);
          As[kk][mm] = p.alpha * v.x; As[kk + 1][mm] = p.alpha * v.y;
          As[kk + 2][mm] = p.alpha * v.z; As[kk + 3][mm] = p.alpha * v.w;
        }
      }
    } else {
#pragma unroll
      for (int idx = threadIdx.x; idx < BM * BK; idx += kThreads) {
        int mm, kk;
        if (TA) { kk = idx / BM; mm = idx % BM; } else { mm = idx / BK; kk = idx % BK; }
        As[kk][mm] = p.alpha * LoadA<TA>(p, m0 + mm, k0 + kk);
      }
    }
#pragma unroll
    for (int idx = threadIdx.x; idx < BK * BN; idx += kThreads) {
      const int kb = idx / BN, nb = idx % BN;
      float b = LoadB<false, BT>(p, k0 + kb, n0 + nb);
      if (p.b_col_scale && n0 + nb < p.N) b = b * p.b_col_scale[n0 + nb];
      Bs[kb][nb] = b;
    }
    __syncthreads();
    const int kmax = k_end - k0 < static_cast<size_t>(BK) ? static_cast<int>(k_end - k0) : BK;
    int kk = 0;
    for (; kk + 4 <= kmax; kk += 4) {
      float a[4][4], b[4][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // one 16-byte shared load per operand row
        const float4 av = *reinterpret_cast<const float4*>(&As[kk + q][ty * 4]);
        const float4 bv = *reinterpret_cast<const float4*>(&Bs[kk + q][tx * 4]);
        a[q][0] = av.x; a[q][1] = av.y; a[q][2] = av.z; a[q][3] = av.w;
        b[q][0] = bv.x; b[q][1] = bv.y; b[q][2] = bv.z; b[q][3] = bv.w;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float t = a[0][i] * b[0][j];
          t = t + a[1][i] * b[1][j];
          t = t + a[2][i] * b[2][j];
          t = t + a[3][i] * b[3][j];
          c[i][j] = c[i][j] + t;
        }
    }
    for (; kk < kmax; ++kk) {  // the K % 4 tail, one term at a time
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          c[i][j] = c[i][j] + As[kk][ty * 4 + i] * Bs[kk][tx * 4 + j];
    }
    __syncthreads();
  }
  // Whole 16-byte rows of the thread's 4x4 block when the layout allows it.
  const size_t nq = n0 + tx * 4;
  const bool vec = !p.partials && (p.N & 3) == 0 && nq + 3 < p.N &&
                   (reinterpret_cast<uintptr_t>(p.C) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(p.addend) & 15) == 0;
  if (vec) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const size_t m = m0 + ty * 4 + i;
      if (m >= p.M) continue;
      float v[4] = {c[i][0], c[i][1], c[i][2], c[i][3]};
      if (p.addend) {
        const float4 d = *reinterpret_cast<const float4*>(p.addend + m * p.N + nq);
        v[0] = d.x + v[0]; v[1] = d.y + v[1]; v[2] = d.z + v[2]; v[3] = d.w + v[3];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (p.bias) v[j] = v[j] + p.bias[nq + j];
        v[j] = ApplyAct(v[j], p.act);
      }
      *reinterpret_cast<float4*>(p.C + m * p.N + nq) = make_float4(v[0], v[1], v[2], v[3]);
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const size_t m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
      if (m >= p.M || n >= p.N) continue;
      float v = c[i][j];
      if (p.partials) {
        p.partials[(static_cast<size_t>(blockIdx.z) * p.M + m) * p.N + n] = v;
        continue;
      }
      if (p.addend) v = p.addend[m * p.N + n] + v;
      if (p.bias) v = v + p.bias[n];
      p.C[m * p.N + n] = ApplyAct(v, p.act);
    }
}

// Folds split-K partials, then the epilogue.  Fixed two-level order: the chunks
// are cut into eight consecutive groups; warp w of a block sums group w in chunk
// order (for 32 neighbouring outputs, one per lane, so every load is a full
// 128-byte line), and the eight group sums are then added in group order.  The
// grouping is a function of the chunk count alone.
constexpr int kFoldGroups = 8;
__global__ void __launch_bounds__(32 * kFoldGroups) SplitKFoldKernel(Params p, size_t chunks) {
  AwaitPrevious();
  __shared__ float group_sum[kFoldGroups][32];
  const size_t total = p.M * p.N;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const size_t i = static_cast<size_t>(blockIdx.x) * 32 + lane;
  const size_t per = (chunks + kFoldGroups - 1) / kFoldGroups;
  const size_t z_begin = w * per, z_end = z_begin + per < chunks ? z_begin + per : chunks;
  float v = 0.0f;
  if (i < total) {
    for (size_t z0 = z_begin; z0 < z_end; z0 += 16) {   // sixteen independent loads at a time
      float part[16];
#pragma unroll
      for (int u = 0; u < 16; ++u)
        part[u] = z0 + u < z_end ? p.partials[(z0 + u) * total + i] : 0.0f;
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        if (z0 + u == z_begin) v = part[u];
        else if (z0 + u < z_end) v = v + part[u];
      }
    }
  }
  group_sum[w][lane] = v;
  __syncthreads();
  if (w != 0 || i >= total) return;
  v = group_sum[0][lane];
  for (int gi = 1; gi < kFoldGroups; ++gi)
    if (static_cast<size_t>(gi) * per < chunks) v = v + group_sum[gi][lane];
  if (p.addend) v = p.addend[i] + v;
  if (p.bias) v = v + p.bias[i % p.N];
  p.C[i] = ApplyAct(v, p.act);
}

// ---- lane order: BM x BN tile (BM * BN = 2048), 256 threads, 4x2 outputs x 8 lanes -----
template <typename BT, int BM, int BN>
__global__ void __launch_bounds__(kThreads) GemmLaneKernel(Params p) {
  AwaitPrevious();
  static_assert(BM * BN == 8 * kThreads, "4x2 outputs per thread");
  __shared__ __align__(16) float As[BK][BM + 4];
  __shared__ __align__(16) float Bs[BK][BN + 4];
  const int tx = threadIdx.x % (BN / 2), ty = threadIdx.x / (BN / 2);
  const size_t m0 = static_cast<size_t>(blockIdx.y) * BM, n0 = static_cast<size_t>(blockIdx.x) * BN;
  float acc[4][2][8];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int l = 0; l < 8; ++l) acc[i][j][l] = 0.0f;
  const bool a_vec = (p.K & 3) == 0 && (reinterpret_cast<uintptr_t>(p.A) & 15) == 0 &&
                     (reinterpret_cast<uintptr_t>(p.a_k_scale) & 15) == 0;
  for (size_t k0 = 0; k0 < p.K; k0 += BK) {
    if (a_vec) {  // 16-byte global loads along k
#pragma unroll
      for (int idx = threadIdx.x; idx < BM * BK / 4; idx += kThreads) {
        const int mm = idx / (BK / 4), kk = (idx % (BK / 4)) * 4;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (m0 + mm < p.M && k0 + kk < p.K) {
          v = *reinterpret_cast<const float4*>(p.A + (m0 + mm) * p.K + k0 + kk);
          if (p.a_k_scale) {
            const float4 sc = *reinterpret_cast<const float4*>(p.a_k_scale + k0 + kk);
            v.x = v.x * sc.x; v.y = v.y * sc.y; v.z = v.z * sc.z; v.w = v.w * sc.w;
          }
        }
        As[kk][mm] = v.x; As[kk + 1][mm] = v.y; As[kk + 2][mm] = v.z; As[kk + 3][mm] = v.w;
      }
    } else {
#pragma unroll
      for (int idx = threadIdx.x; idx < BM * BK; idx += kThreads) {
        const int mm = idx / BK, kk = idx % BK;
        float a = LoadA<false>(p, m0 + mm, k0 + kk);
        if (p.a_k_scale && k0 + kk < p.K) a = a * p.a_k_scale[k0 + kk];
        As[kk][mm] = a;
      }
    }
#pragma unroll
    for (int idx = threadIdx.x; idx < BN * BK; idx += kThreads) {
      const int nn = idx / BK, kk = idx % BK;
      Bs[kk][nn] = LoadB<true, BT>(p, k0 + kk, n0 + nn);
    }
    __syncthreads();
    const int kmax = p.K - k0 < static_cast<size_t>(BK) ? static_cast<int>(p.K - k0) : BK;
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      if (kk < kmax) {
        const int l = kk & 7;  // k0 is a multiple of 16, so k mod 8 == kk mod 8
        const float4 av = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
        const float2 bv = *reinterpret_cast<const float2*>(&Bs[kk][tx * 2]);
        const float a[4] = {av.x, av.y, av.z, av.w};
        const float b[2] = {bv.x, bv.y};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) acc[i][j][l] = acc[i][j][l] + a[i] * b[j];
      }
    }
    __syncthreads();
  }
  const size_t np = n0 + tx * 2;
  if ((p.N & 1) == 0 && np + 1 < p.N && (reinterpret_cast<uintptr_t>(p.C) & 7) == 0 &&
      (reinterpret_cast<uintptr_t>(p.addend) & 7) == 0) {  // 8-byte pairs
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const size_t m = m0 + ty * 4 + i;
      if (m >= p.M) continue;
      float v[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float s = acc[i][j][0];
#pragma unroll
        for (int l = 1; l < 8; ++l) s = s + acc[i][j][l];
        v[j] = p.alpha * s;
      }
      if (p.addend) {
        const float2 d = *reinterpret_cast<const float2*>(p.addend + m * p.N + np);
        v[0] = d.x + v[0]; v[1] = d.y + v[1];
      }
      *reinterpret_cast<float2*>(p.C + m * p.N + np) = make_float2(v[0], v[1]);
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const size_t m = m0 + ty * 4 + i, n = n0 + tx * 2 + j;
      if (m >= p.M || n >= p.N) continue;
      float s = acc[i][j][0];
#pragma unroll
      for (int l = 1; l < 8; ++l) s = s + acc[i][j][l];
      float v = p.alpha * s;
      if (p.addend) v = p.addend[m * p.N + n] + v;
      p.C[m * p.N + n] = v;
    }
}

// ---- merge: a run of deltas, each alpha A B from zero, in one launch -----------------------
// delta [M, N] = 0 + (alpha A) B in the quad order, K = rank: what a kFill with zero followed by a kGemmAccNN leaves,
// bit for bit, without the filled tensor's round trip through memory.  A block owns 64 rows x 256 columns of one
// delta: two columns per thread with their K x 2 slice of B in registers (asked for before A's rows are waited for),
// 32 rows one after the other, A's rows broadcast from shared memory.  Bound by the f32 pipe: without fused
// multiply-adds an output is 2 K operations, 25 us for the 113 MB (48 deltas of 768 x 768, rank 16) that take 17 us to
// write.  Measured for those: 58.7 us with blocks of 32 rows and four columns a thread, whose B and A round trips lay
// eight rows apart under sixteen warps to an SM; 42.5 so (0.86 instructions issued per cycle and scheduler); 45.8 with the operations as f32x2 pairs.
// `nonfinite` (or null) counts the values that are not finite on their way out.
constexpr int kMergeRows = 64;
template <int K>
__global__ void __launch_bounds__(kThreads) MergeDeltasKernel(const __grid_constant__ MergeTable table,
                                                              unsigned long long* __restrict__ nonfinite) {
  AwaitPrevious();
  __shared__ __align__(16) float As[kMergeRows][K];
  const MergeEntry& e = table.entry[blockIdx.y];
  const int tiles_n = static_cast<int>((e.N + 255) / 256);
  const size_t m0 = static_cast<size_t>(blockIdx.x / tiles_n) * kMergeRows;
  if (m0 >= e.M) return;
  const size_t n = static_cast<size_t>(blockIdx.x % tiles_n) * 256 + (threadIdx.x & 127) * 2;
  const size_t rows = e.M - m0 < kMergeRows ? e.M - m0 : kMergeRows;
  float2 b[K];
#pragma unroll
  for (int k = 0; k < K; ++k)
    b[k] = n < e.N ? *reinterpret_cast<const float2*>(e.B + k * e.N + n) : make_float2(0.0f, 0.0f);   // N % 4 == 0
  for (size_t i = threadIdx.x; i < rows * K; i += kThreads) As[i / K][i % K] = e.alpha * e.A[m0 * K + i];
  __syncthreads();
  unsigned bad = 0;
  if (n < e.N) {
    float zero = 0.0f;   // NaN once a value is not finite
    const size_t step = 2 * static_cast<size_t>(e.N);
    float* const c_first = e.C + (m0 + (threadIdx.x >> 7)) * e.N + n;
    float* at = c_first;
    const float* a_row = As[threadIdx.x >> 7];
#pragma unroll 4
    for (int left = (static_cast<int>(rows) + 1 - static_cast<int>(threadIdx.x >> 7)) / 2; left > 0; --left, at += step, a_row += 2 * K) {
      float2 c = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int k = 0; k < K; k += 4) {
        const float4 a = *reinterpret_cast<const float4*>(a_row + k);
        float tx = a.x * b[k].x, ty = a.x * b[k].y;
        tx = tx + a.y * b[k + 1].x; ty = ty + a.y * b[k + 1].y;
        tx = tx + a.z * b[k + 2].x; ty = ty + a.z * b[k + 2].y;
        tx = tx + a.w * b[k + 3].x; ty = ty + a.w * b[k + 3].y;
        c.x = c.x + tx;
        c.y = c.y + ty;
      }
      *reinterpret_cast<float2*>(at) = c;
      zero = fmaf(c.x, 0.0f, zero);
      zero = fmaf(c.y, 0.0f, zero);
    }
    if (!(zero == 0.0f))   // count them, on what was written
      for (const float* p = c_first; p < at; p += step) bad += !isfinite(p[0]) + !isfinite(p[1]);
  }
  if (!nonfinite) return;
  bad = __reduce_add_sync(0xFFFFFFFFu, bad);
  if ((threadIdx.x & 31) == 0 && bad) atomicAdd(nonfinite, static_cast<unsigned long long>(bad));
}

// ---- both orders, few outputs --------------------------------------------------------------
// With fewer 64 x 64 (or skinny) tiles than SMs the kernels above are a serial chain of global loads: K / 16 steps of
// about 1.4 us in one or two blocks.  Here a block owns 16 R x 16 R outputs, R x R per thread, so that there are blocks
// to go round, and takes K 128 at a time with the next 128 already on their way in registers while these are
// multiplied.  The same operations per output in the same order (57 x 8 x 784: 81.5 -> 8.1 us; 57 x 128 x 784: 76 -> 8.4 us).
constexpr int kFlatK = 128;
// T x T outputs of a block, R x R of a thread.
template <int T> struct FlatShape { static constexpr int R = T > 16 ? 2 : 1, kSide = T / R, kThreads = kSide * kSide; };
template <bool TA, bool TB, typename BT, int T>
struct FlatLoader {
  static constexpr int kThreads = FlatShape<T>::kThreads, kPer = T * kFlatK / kThreads;   // elements per thread and operand
  float a[kPer], b[kPer];
  // Where an operand's first element of this thread lies, how far its elements and the blocks of K are apart: lanes along
  // the operand's contiguous axis.  (Addresses made anew for every element, 64-bit products and two bounds each, took as long as the
  // arithmetic: 57 x 128 x 784 11.4 / 10.3 us, transposed 15.7 / 10.8 and 15.4 / 10.2.)
  const float* pa;
  const BT* pb;
  size_t a_step, b_step, a_chunk, b_chunk;
  static constexpr int kKStep = kThreads / T;                                   // (k apart, along rows)
  static constexpr int kLanes = kThreads < kFlatK ? kThreads : kFlatK, kRun = kFlatK / kLanes, kRowStep = kThreads / kLanes;
  // Which (row, k) element i of this thread is.
  static __device__ __forceinline__ void At(int i, bool k_contiguous, int* row, int* k) {
    const int t = static_cast<int>(threadIdx.x);
    if (k_contiguous) { *row = t / kLanes + i / kRun * kRowStep; *k = t % kLanes + i % kRun * kLanes; }
    else { *row = t % T; *k = t / T + i * kKStep; }
  }
  // ... and how far from element 0.
  static __device__ __forceinline__ size_t Distance(int i, bool k_contiguous, size_t step) {
    return k_contiguous ? i / kRun * step + i % kRun * kLanes : i * step;
  }
  __device__ __forceinline__ FlatLoader(const Params& p, size_t m0, size_t n0) {
    int r, k;
    At(0, !TA, &r, &k);
    pa = TA ? p.A + k * p.M + m0 + r : p.A + (m0 + r) * p.K + k;
    a_step = TA ? kKStep * p.M : kRowStep * p.K;
    a_chunk = TA ? kFlatK * p.M : kFlatK;
    At(0, TB, &r, &k);
    pb = static_cast<const BT*>(p.B) + (TB ? (n0 + r) * p.K + k : k * p.N + n0 + r);
    b_step = TB ? kRowStep * p.K : kKStep * p.N;
    b_chunk = TB ? kFlatK : kFlatK * p.N;
  }
  // The block at k0, which follows the one loaded before.
  __device__ __forceinline__ void Load(const Params& p, size_t m0, size_t n0, size_t k0) {
    auto clamp = [](size_t left) { return left < static_cast<size_t>(kFlatK) ? static_cast<int>(left) : kFlatK; };
    const int left = clamp(p.K - k0), rows = clamp(p.M - m0), cols = clamp(p.N - n0);
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      int r, k;
      At(i, !TA, &r, &k);
      a[i] = r < rows && k < left ? pa[Distance(i, !TA, a_step)] : 0.0f;
      At(i, TB, &r, &k);
      b[i] = r < cols && k < left ? Widen<BT>(pb[Distance(i, TB, b_step)]) : 0.0f;
    }
    pa += a_chunk;
    pb += b_chunk;
    if (p.a_k_scale) {
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        int r, k;
        At(i, !TA, &r, &k);
        if (k < left) a[i] = a[i] * p.a_k_scale[k0 + k];
      }
    }
    if (p.b_col_scale) {
#pragma unroll
      for (int i = 0; i < kPer; ++i) {
        int r, k;
        At(i, TB, &r, &k);
        if (r < cols) b[i] = b[i] * p.b_col_scale[n0 + r];
      }
    }
  }
  // As [row][k] (a row's quads are 16-byte reads), Bs [row][k] likewise.
  __device__ __forceinline__ void Store(float (*As)[kFlatK + 4], float (*Bs)[kFlatK + 4], float alpha) {
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
      int r, k;
      At(i, !TA, &r, &k);
      As[r][k] = alpha * a[i];
      At(i, TB, &r, &k);
      Bs[r][k] = b[i];
    }
  }
};

// Lane order when kLane, quad order otherwise.
template <bool kLane, bool TA, bool TB, typename BT, int T>
__global__ void __launch_bounds__(FlatShape<T>::kThreads) GemmFlatKernel(Params p) {
  AwaitPrevious();
  constexpr int R = FlatShape<T>::R, kSide = FlatShape<T>::kSide;
  __shared__ __align__(16) float As[T][kFlatK + 4];
  __shared__ __align__(16) float Bs[T][kFlatK + 4];
  const int tx = threadIdx.x % kSide, ty = threadIdx.x / kSide;   // outputs (ty + kSide i, tx + kSide j)
  const size_t m0 = static_cast<size_t>(blockIdx.y) * T, n0 = static_cast<size_t>(blockIdx.x) * T;
  float c[R][R][kLane ? 8 : 1];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < R; ++j) {
#pragma unroll
      for (int l = 0; l < (kLane ? 8 : 1); ++l) c[i][j][l] = 0.0f;
      const size_t m = m0 + ty + kSide * i, n = n0 + tx + kSide * j;
      if (!kLane && p.accumulate && m < p.M && n < p.N) c[i][j][0] = p.C[m * p.N + n];
    }
  const float alpha_a = kLane ? 1.0f : p.alpha;   // (x * 1 == x)
  FlatLoader<TA, TB, BT, T> next(p, m0, n0);
  next.Load(p, m0, n0, 0);
  for (size_t k0 = 0; k0 < p.K; k0 += kFlatK) {
    next.Store(As, Bs, alpha_a);
    __syncthreads();
    if (k0 + kFlatK < p.K) next.Load(p, m0, n0, k0 + kFlatK);
    const int kmax = p.K - k0 < static_cast<size_t>(kFlatK) ? static_cast<int>(p.K - k0) : kFlatK;
    int k = 0;
    auto quad = [&](int k) {
      float4 a[R], b[R];
#pragma unroll
      for (int i = 0; i < R; ++i) a[i] = *reinterpret_cast<const float4*>(&As[ty + kSide * i][k]);
#pragma unroll
      for (int j = 0; j < R; ++j) b[j] = *reinterpret_cast<const float4*>(&Bs[tx + kSide * j][k]);
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) {
          if (kLane) {
            // k0 and k are multiples of 4: the four products go to lanes 0-3 or 4-7.
            float* l = c[i][j];
            if ((k & 4) == 0) {
              l[0] = l[0] + a[i].x * b[j].x; l[1] = l[1] + a[i].y * b[j].y;
              l[2] = l[2] + a[i].z * b[j].z; l[3] = l[3] + a[i].w * b[j].w;
            } else {
              l[4 % (kLane ? 8 : 1)] = l[4 % (kLane ? 8 : 1)] + a[i].x * b[j].x;
              l[5 % (kLane ? 8 : 1)] = l[5 % (kLane ? 8 : 1)] + a[i].y * b[j].y;
              l[6 % (kLane ? 8 : 1)] = l[6 % (kLane ? 8 : 1)] + a[i].z * b[j].z;
              l[7 % (kLane ? 8 : 1)] = l[7 % (kLane ? 8 : 1)] + a[i].w * b[j].w;
            }
          } else {
            float t = a[i].x * b[j].x;
            t = t + a[i].y * b[j].y;
            t = t + a[i].z * b[j].z;
            t = t + a[i].w * b[j].w;
            c[i][j][0] = c[i][j][0] + t;
          }
        }
    };
    if (kmax == kFlatK) {   // (quads' products do not wait for one another: only the sums are a chain)
#pragma unroll 8
      for (; k < kFlatK; k += 4) quad(k);
    } else {
      for (; k + 4 <= kmax; k += 4) quad(k);
    }
    for (; k < kmax; ++k)   // the K % 4 tail, one term at a time
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) {
          const float x = As[ty + kSide * i][k] * Bs[tx + kSide * j][k];
#pragma unroll
          for (int l = 0; l < (kLane ? 8 : 1); ++l)
            if (!kLane || l == (k & 7)) c[i][j][l] = c[i][j][l] + x;
        }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const size_t m = m0 + ty + kSide * i, n = n0 + tx + kSide * j;
      if (m >= p.M || n >= p.N) continue;
      float v = c[i][j][0];
      if (kLane) {
#pragma unroll
        for (int l = 1; l < (kLane ? 8 : 1); ++l) v = v + c[i][j][l];
        v = p.alpha * v;
      }
      if (p.addend) v = p.addend[m * p.N + n] + v;
      if (p.bias) v = v + p.bias[n];
      p.C[m * p.N + n] = ApplyAct(v, p.act);
    }
}

unsigned Blocks(size_t extent, size_t tile) { return static_cast<unsigned>((extent + tile - 1) / tile); }

size_t QuadTiles(size_t M, size_t N) {
  if (N <= 16) return static_cast<size_t>(Blocks(M, 256)) * Blocks(N, 16);
  if (M <= 16) return static_cast<size_t>(Blocks(N, 256)) * Blocks(M, 16);
  return static_cast<size_t>(Blocks(M, 64)) * Blocks(N, 64);
}
size_t LaneTiles(size_t M, size_t N) {
  if (N <= 16) return static_cast<size_t>(Blocks(M, 128)) * Blocks(N, 16);
  if (M <= 16) return static_cast<size_t>(Blocks(N, 128)) * Blocks(M, 16);
  return static_cast<size_t>(Blocks(M, 64)) * Blocks(N, 32);
}

// The flat kernel where the tile kernels would leave SMs idle: 32 x 32 outputs per block if that still makes a block
// per SM, else 16 x 16, and 8 x 8 where those are few: a block is bound by its own shared memory and chains of sums (57 x 128 x 784
// 10.1 / 8.4 us, 32 x 8 x 1024 12.1 / 9.5; of a transposed A, whose rows of eight are half a sector, 10.2 / 11.3: 16 x 16).
template <bool kLane, bool TA, bool TB, typename BT>
void LaunchFlat(const Params& p, cudaStream_t s) {
  auto blocks = [&](size_t t) { return static_cast<size_t>(Blocks(p.M, t)) * Blocks(p.N, t); };
  if (blocks(32) >= 148)
    Next(GemmFlatKernel<kLane, TA, TB, BT, 32>, dim3(Blocks(p.N, 32), Blocks(p.M, 32)), FlatShape<32>::kThreads, 0, s)(p);
  else if (TA || blocks(16) > 37)
    Next(GemmFlatKernel<kLane, TA, TB, BT, 16>, dim3(Blocks(p.N, 16), Blocks(p.M, 16)), FlatShape<16>::kThreads, 0, s)(p);
  else if constexpr (!TA)
    Next(GemmFlatKernel<kLane, TA, TB, BT, 8>, dim3(Blocks(p.N, 8), Blocks(p.M, 8)), FlatShape<8>::kThreads, 0, s)(p);
}

template <bool TA, typename BT>
void LaunchQuad(const Params& p, unsigned z, cudaStream_t s) {
  if (z == 1 && !p.partials && QuadTiles(p.M, p.N) < 148) {
    LaunchFlat<false, TA, false, BT>(p, s);
  } else if (p.N <= 16) {
    Next(GemmQuadKernel<TA, BT, 256, 16>, dim3(Blocks(p.N, 16), Blocks(p.M, 256), z), kThreads, 0, s)(p);
  } else if (p.M <= 16) {
    Next(GemmQuadKernel<TA, BT, 16, 256>, dim3(Blocks(p.N, 256), Blocks(p.M, 16), z), kThreads, 0, s)(p);
  } else {
    Next(GemmQuadKernel<TA, BT, 64, 64>, dim3(Blocks(p.N, 64), Blocks(p.M, 64), z), kThreads, 0, s)(p);
  }
}

template <typename BT>
void LaunchLane(const Params& p, cudaStream_t s) {
  if (LaneTiles(p.M, p.N) < 148) {
    LaunchFlat<true, false, true, BT>(p, s);
  } else if (p.N <= 16) {
    Next(GemmLaneKernel<BT, 128, 16>, dim3(Blocks(p.N, 16), Blocks(p.M, 128)), kThreads, 0, s)(p);
  } else if (p.M <= 16) {
    Next(GemmLaneKernel<BT, 16, 128>, dim3(Blocks(p.N, 128), Blocks(p.M, 16)), kThreads, 0, s)(p);
  } else {
    Next(GemmLaneKernel<BT, 64, 32>, dim3(Blocks(p.N, 32), Blocks(p.M, 64)), kThreads, 0, s)(p);
  }
}

}  // namespace

size_t SplitKChunkRows(size_t M, size_t N, size_t K) {
  const size_t tiles = QuadTiles(M, N);
  size_t rows = kSplitKChunk;
  while (rows > 32 && ((K + rows - 1) / rows) * tiles < 296) rows /= 2;
  return rows;
}

size_t SplitKChunks(size_t M, size_t N, size_t K) {
  if (K < 4 * kSplitKChunk || QuadTiles(M, N) >= 148) return 1;
  const size_t rows = SplitKChunkRows(M, N, K);
  return (K + rows - 1) / rows;
}

void MergeDeltas(const MergeTable& table, int count, uint32_t K, unsigned long long* nonfinite, cudaStream_t s) {
  size_t blocks = 1;
  for (int i = 0; i < count; ++i)
    blocks = std::max<size_t>(blocks, ((table.entry[i].M + kMergeRows - 1) / kMergeRows) * ((table.entry[i].N + 255) / 256));
  const dim3 grid(static_cast<unsigned>(blocks), static_cast<unsigned>(count));
  switch (K) {
    case 4: Next(MergeDeltasKernel<4>, grid, kThreads, 0, s)(table, nonfinite); break;
    case 8: Next(MergeDeltasKernel<8>, grid, kThreads, 0, s)(table, nonfinite); break;
    case 12: Next(MergeDeltasKernel<12>, grid, kThreads, 0, s)(table, nonfinite); break;
    default: Next(MergeDeltasKernel<16>, grid, kThreads, 0, s)(table, nonfinite); break;
  }
}

bool GemmExact(const GemmArgs& a, cudaStream_t s) {
  if (a.M == 0 || a.N == 0) return false;
  Params p{a.A, a.B, a.C, a.M, a.N, a.K, a.alpha, a.b_col_scale, a.a_k_scale,
           a.bias, a.addend, a.act, a.accumulate, 0, nullptr};
  // Only the expand kernel takes the tail add; every other path sees none.
  Params pt = p;
  if (a.tail_addend && a.tail_out && Aligned16(a.tail_addend) && Aligned16(a.tail_out)) {
    pt.tail_addend = a.tail_addend;
    pt.tail_out = a.tail_out;
  }
  const auto reduce = a.contract_fma ? fast::SkinnyReduce : exact::SkinnyReduce;
  const auto expand = a.contract_fma ? fast::SkinnyExpand : exact::SkinnyExpand;
  const auto tn_partials = a.contract_fma ? fast::SkinnyTnPartials : exact::SkinnyTnPartials;
  if (a.b_transposed) {
    if (a.b_type == BType::kF32) {
      if (reduce(p, true, s)) return false;
      if (expand(pt, true, s)) return pt.tail_out != nullptr;
    }
    switch (a.b_type) {
      case BType::kF32: LaunchLane<float>(p, s); break;
      case BType::kI8: LaunchLane<int8_t>(p, s); break;
      case BType::kBf16: LaunchLane<uint16_t>(p, s); break;
    }
    return false;
  }
  if (a.a_transposed) {
    // Adapter gradients: a [rank x width] or [width x rank] result reduced over
    // every row of the batch.  With few output tiles and a long K the chunks go
    // to separate blocks (fixed geometry: a pure function of the shape).
    const size_t chunks = SplitKChunks(a.M, a.N, a.K);
    if (chunks > 1 && a.split_scratch && !a.accumulate &&
        chunks * a.M * a.N <= a.split_scratch_floats) {
      p.k_chunk = SplitKChunkRows(a.M, a.N, a.K);
      p.partials = a.split_scratch;
      if (!tn_partials(p, chunks, s)) LaunchQuad<true, float>(p, static_cast<unsigned>(chunks), s);
      const size_t blocks = (a.M * a.N + 31) / 32;
      Next(SplitKFoldKernel, static_cast<unsigned>(blocks), 32 * kFoldGroups, 0, s)(p, chunks);
      return false;
    }
    LaunchQuad<true, float>(p, 1, s);
    return false;
  }
  if (a.b_type == BType::kF32) {
    if (reduce(p, false, s)) return false;
    if (expand(pt, false, s)) return pt.tail_out != nullptr;
  }
  switch (a.b_type) {
    case BType::kF32: LaunchQuad<false, float>(p, 1, s); break;
    case BType::kI8: LaunchQuad<false, int8_t>(p, 1, s); break;
    case BType::kBf16: LaunchQuad<false, uint16_t>(p, 1, s); break;
  }
  return false;
}

}  // namespace see::k
