// Device-side tails of evaluation and merge: the accuracy tally over the
// softmax probabilities and the finiteness scan of merged deltas.  The
// reference computes both on the host over its arena (reference:
// runtime/dispatcher/update_engine.cc:535-564 and :1051-1060); with discrete
// memory that would move the whole probability tensor over the bus, so the
// same integer results are produced here and only three counters come back.
// Integer tallies: exact whatever the order of the atomic adds.
#include "kernels.h"
#include "launch.cuh"

namespace see::k {

namespace {

// One warp per row.  argmax as the sequential scan defines it: start at column
// 0, move to column c only when row[c] > row[argmax] — the first maximum wins,
// a NaN never wins, and a NaN in column 0 is never displaced.
// kVec (C % 4 == 0, 16-byte rows): four 16-byte loads in flight per lane; with one
// scalar load at a time the rows of a 32000-wide vocabulary ran at half the memory's rate.
template <bool kVec>
__device__ void ArgmaxRows(const float* __restrict__ probs, const int32_t* __restrict__ labels, size_t N, size_t C,
                           unsigned long long* __restrict__ tally, size_t warp, size_t warps) {
  const int lane = threadIdx.x & 31;
  unsigned long long rows = 0, hits = 0;
  for (size_t r = warp; r < N; r += warps) {
    const int32_t lab = labels[r];
    if (lab < 0) continue;
    const float* row = probs + r * C;
    const float first = row[0];
    size_t arg = 0;
    if (!isnan(first)) {
      float best = first;
      size_t idx = 0;
      auto look = [&](float v, size_t c) {   // (a lane's columns ascend: its first maximum stays)
        if (v > best) { best = v; idx = c; }
      };
      if constexpr (kVec) {
        constexpr size_t kAhead = 4;
        const float4* row4 = reinterpret_cast<const float4*>(row);
        const size_t C4 = C / 4;
        for (size_t c0 = lane; c0 < C4; c0 += 32 * kAhead) {
          float4 v[kAhead];
#pragma unroll
          for (size_t u = 0; u < kAhead; ++u)
            v[u] = c0 + 32 * u < C4 ? __ldg(row4 + c0 + 32 * u) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
#pragma unroll
          for (size_t u = 0; u < kAhead; ++u) {
            const size_t c = (c0 + 32 * u) * 4;
            look(v[u].x, c);
            look(v[u].y, c + 1);
            look(v[u].z, c + 2);
            look(v[u].w, c + 3);
          }
        }
      } else {
        for (size_t c = lane; c < C; c += 32) look(row[c], c);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xFFFFFFFFu, best, o);
        const unsigned long long oi = __shfl_xor_sync(0xFFFFFFFFu, static_cast<unsigned long long>(idx), o);
        if (ov > best || (ov == best && oi < idx)) { best = ov; idx = oi; }
      }
      arg = idx;
    }
    if (lane == 0) {
      ++rows;
      if (static_cast<size_t>(lab) == arg) ++hits;
    }
  }
  if (lane == 0 && rows) {
    atomicAdd(&tally[0], rows);
    atomicAdd(&tally[1], hits);
  }
}
__device__ __forceinline__ bool ArgmaxVec(const float* probs, size_t C) {
  return (C & 3) == 0 && (reinterpret_cast<uintptr_t>(probs) & 15) == 0;
}

__global__ void ArgmaxTallyKernel(const float* __restrict__ probs, const int32_t* __restrict__ labels,
                                  size_t N, size_t C, unsigned long long* __restrict__ tally) {
  AwaitPrevious();
  const size_t warps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  const size_t warp = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5;
  if (ArgmaxVec(probs, C)) ArgmaxRows<true>(probs, labels, N, C, tally, warp, warps);
  else ArgmaxRows<false>(probs, labels, N, C, tally, warp, warps);
}

__global__ void CountNonFiniteKernel(const float* __restrict__ x, size_t n,
                                     unsigned long long* __restrict__ tally) {
  AwaitPrevious();
  unsigned long long bad = 0;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n; i += stride)
    bad += !isfinite(x[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) bad += __shfl_xor_sync(0xFFFFFFFFu, bad, o);
  if ((threadIdx.x & 31) == 0 && bad) atomicAdd(&tally[2], bad);
}

// ---- the real-row loss of an evaluated batch -------------------------------------------
// The engine scores a validation set whose last batch wraps (or any masked
// plan) over its real rows alone: the sum, in row order and in double, of each
// row's loss evaluated with the loss kernel's own expression (reference:
// runtime/dispatcher/update_engine.cc:977-1026).  The terms are made in parallel and
// added by ONE chain in row order, so the double sum has the reference's association.
// The count of rows the sum is over (the real rows, or the real TARGET rows under a
// masked loss) is an integer tally.
//
// Cross-entropy, with the accuracy tally in the same launch: block 0 is the chain, seven warps making 224 terms while
// the eighth adds the 224 before them, and the other blocks take the argmax of the rows.  The chain is a dependent
// double addition per row whatever surrounds it (about 7 ns: 29 us for 4096 rows), so it runs beside the tally's
// reading of the probabilities instead of after it.
constexpr size_t kTailThreads = 256, kTailChunk = kTailThreads - 32;
__global__ void __launch_bounds__(kTailThreads)
XentEvalTailKernel(const float* __restrict__ probs, const float* __restrict__ arg_probs, size_t arg_cols,
                   const int32_t* __restrict__ labels, size_t rows, size_t width, double* __restrict__ out,
                   unsigned long long* __restrict__ tally) {
  AwaitPrevious();
  if (blockIdx.x > 0) {
    const size_t warps = static_cast<size_t>(gridDim.x - 1) * (kTailThreads / 32);
    const size_t warp = static_cast<size_t>(blockIdx.x - 1) * (kTailThreads / 32) + (threadIdx.x >> 5);
    if (ArgmaxVec(arg_probs, arg_cols)) ArgmaxRows<true>(arg_probs, labels, rows, arg_cols, tally, warp, warps);
    else ArgmaxRows<false>(arg_probs, labels, rows, arg_cols, tally, warp, warps);
    return;
  }
  __shared__ __align__(16) double terms[2][kTailChunk];
  double sum = 0.0;
  unsigned counted = 0;
  const size_t chunks = (rows + kTailChunk - 1) / kTailChunk;
  for (size_t c = 0; c <= chunks; ++c) {
    if (threadIdx.x >= 32) {
      const size_t at = threadIdx.x - 32, r = c * kTailChunk + at;
      if (c < chunks) {
        const int32_t lab = r < rows ? labels[r] : -1;
        double t = 0.0;   // a skipped row's term: adding it leaves the sum as it is
        if (lab >= 0) {
          const float p = probs[r * width + static_cast<size_t>(lab)];
          t = -log(isnan(p) ? static_cast<double>(p) : static_cast<double>(fmaxf(p, 1e-12f)));
          ++counted;
        }
        terms[c & 1][at] = t;
      }
    } else if (c > 0) {
      const double2* t = reinterpret_cast<const double2*>(terms[(c - 1) & 1]);
#pragma unroll 16
      for (size_t j = 0; j < kTailChunk / 2; ++j) {
        const double2 v = t[j];
        sum += v.x;
        sum += v.y;
      }
    }
    __syncthreads();
  }
  counted = __reduce_add_sync(0xFFFFFFFFu, counted);
  if ((threadIdx.x & 31) == 0 && counted) atomicAdd(&tally[3], static_cast<unsigned long long>(counted));
  if (threadIdx.x == 0) out[0] = sum;
}

__global__ void SquaredDiffTermsKernel(const float* __restrict__ pred, const float* __restrict__ target,
                                       size_t n, double* __restrict__ terms) {
  AwaitPrevious();
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n; i += stride) {
    const double d = static_cast<double>(pred[i]) - target[i];
    terms[i] = d * d;
  }
}

// out[0] = the sum of the terms over the divisor (the row width of a mean squared
// error); tally[3] = n.  One warp: 32 terms per load, two
// loads ahead, and every lane makes the same chain of additions over the terms
// the shuffles bring it in row order, so a step costs one dependent double add
// (one thread that also loads: 190 us for 4096 rows; this: 35).
__global__ void OrderedFoldKernel(const double* __restrict__ terms, size_t n, double divisor, double* __restrict__ out,
                                  unsigned long long* __restrict__ tally) {
  AwaitPrevious();
  const size_t lane = threadIdx.x;
  double sum = 0.0;
  auto load = [&](size_t i0) { return i0 + lane < n ? terms[i0 + lane] : 0.0; };
  double next0 = load(0), next1 = load(32);
  for (size_t i0 = 0; i0 < n; i0 += 32) {
    const double t = next0;
    next0 = next1;
    next1 = load(i0 + 64);
#pragma unroll
    for (int j = 0; j < 32; ++j) sum += __shfl_sync(0xFFFFFFFFu, t, j);
  }
  if (lane != 0) return;
  out[0] = divisor != 0.0 ? sum / divisor : sum;
  tally[3] = n;
}

// ---- per-column int8 quantiser ----------------------------------------------------------
// scale[n] = max_k |w[k, n]| / 127, an all-zero column takes 1, and the scale
// never falls below the smallest normal float; level = round-half-away(w /
// scale) clamped to +-127, by a true division (reference:
// compiler/backend/allocation/arena_binder.cc:129-190).  A maximum does not
// depend on the order it is taken in, so atomics on the bit pattern of |w|
// (non-negative floats order like their bits) give the reference's scales exactly.
__global__ void ColumnAbsMaxKernel(const float* __restrict__ w, size_t K, size_t N,
                                   unsigned int* __restrict__ maxbits) {
  AwaitPrevious();
  const size_t n = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (n >= N) return;
  const size_t rows_per = (K + gridDim.y - 1) / gridDim.y;
  const size_t k0 = blockIdx.y * rows_per, k1 = k0 + rows_per < K ? k0 + rows_per : K;
  float m = 0.0f;
  for (size_t k = k0; k < k1; ++k) {
    const float a = fabsf(w[k * N + n]);
    if (m < a) m = a;   // std::max(m, a): a NaN never replaces m
  }
  atomicMax(&maxbits[n], __float_as_uint(m));
}

__global__ void ColumnScaleKernel(const unsigned int* __restrict__ maxbits, size_t N, float* __restrict__ scales) {
  AwaitPrevious();
  const size_t n = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (n >= N) return;
  const float m = __uint_as_float(maxbits[n]);
  const float q = __fdiv_rn(m, 127.0f);
  scales[n] = m == 0.0f ? 1.0f : (q < 1.17549435e-38f ? 1.17549435e-38f : q);
}

__global__ void QuantizeLevelsKernel(const float* __restrict__ w, const float* __restrict__ scales, size_t count,
                                     size_t N, int8_t* __restrict__ q) {
  AwaitPrevious();
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < count; i += stride) {
    float r = roundf(__fdiv_rn(w[i], scales[i % N]));   // roundf: halves away from zero, as std::round
    r = r < -127.0f ? -127.0f : (r > 127.0f ? 127.0f : r);
    q[i] = static_cast<int8_t>(r);
  }
}

}  // namespace

void XentEvalTail(const float* probs, size_t width, const float* arg_probs, size_t arg_cols, const int32_t* labels,
                  size_t real_rows, double* out, unsigned long long* tally, cudaStream_t s) {
  size_t blocks = arg_probs ? (real_rows + 7) / 8 : 0;
  if (blocks > 148 * 8) blocks = 148 * 8;
  Next(XentEvalTailKernel, static_cast<unsigned>(blocks + 1), kTailThreads, 0, s)(probs, arg_probs, arg_cols, labels,
                                                                               real_rows, width, out, tally);
}

void MseRealRowLoss(const float* pred, const float* target, size_t real_rows, size_t width, double* terms,
                    double* out, unsigned long long* tally, cudaStream_t s) {
  const size_t n = real_rows * width;
  if (n) {
    size_t blocks = (n + 255) / 256;
    if (blocks > 148 * 8) blocks = 148 * 8;
    Next(SquaredDiffTermsKernel, static_cast<unsigned>(blocks), 256, 0, s)(pred, target, n, terms);
  }
  Next(OrderedFoldKernel, 1, 32, 0, s)(terms, n, static_cast<double>(width), out, tally);
}

void QuantizeColumns(const float* w, size_t K, size_t N, int8_t* levels, float* scales,
                     unsigned int* maxbits_scratch, cudaStream_t s) {
  if (K == 0 || N == 0) return;
  cudaMemsetAsync(maxbits_scratch, 0, N * sizeof(unsigned int), s);
  unsigned slices = static_cast<unsigned>((K + 63) / 64);
  if (slices > 1024) slices = 1024;
  const dim3 grid(static_cast<unsigned>((N + 127) / 128), slices);
  Next(ColumnAbsMaxKernel, grid, 128, 0, s)(w, K, N, maxbits_scratch);
  Next(ColumnScaleKernel, static_cast<unsigned>((N + 127) / 128), 128, 0, s)(maxbits_scratch, N, scales);
  size_t blocks = (K * N + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  Next(QuantizeLevelsKernel, static_cast<unsigned>(blocks), 256, 0, s)(w, scales, K * N, N, levels);
}

void ArgmaxTally(const float* probs, const int32_t* labels, size_t N, size_t C,
                 unsigned long long* tally, cudaStream_t s) {
  if (N == 0) return;
  size_t blocks = (N + 7) / 8;
  if (blocks > 148 * 8) blocks = 148 * 8;
  Next(ArgmaxTallyKernel, static_cast<unsigned>(blocks), 256, 0, s)(probs, labels, N, C, tally);
}

void CountNonFinite(const float* x, size_t n, unsigned long long* tally, cudaStream_t s) {
  if (n == 0) return;
  size_t blocks = (n + 255) / 256;
  if (blocks > 148 * 8) blocks = 148 * 8;
  Next(CountNonFiniteKernel, static_cast<unsigned>(blocks), 256, 0, s)(x, n, tally);
}

}  // namespace see::k
