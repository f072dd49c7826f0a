// Exact causal attention on the tensor cores, where the bits are not observed: scores as accurate as dots in double that are
// rounded to f32, but for a tenth of the rounding of the row's largest score, sums of probabilities times values as accurate as
// f32 multiply-adds.
//
// Scores.  A row of Q (or K) is a fixed-point number per element: scaled by a power of two to (-256, 256) and cut into four
// signed digits of eight bits, whole numbers up to 256 (the first) and 128 and so bf16 values exactly:
//     x = 2^(e - 8) (s0 + s1 / 2^8 + s2 / 2^16 + s3 / 2^24) + r,  |r| <= 2^(e - 33),  2^e > max |x|.
// Products of digits are whole numbers, and a sum of those of up to 64 features with one i + j is below 2^23: the tensor core's
// f32 accumulator holds it exactly, in whatever order and rounding it adds.  The thirteen products of digits with i + j <= 4 meet in
// five accumulators, one for each i + j, which four multiply-adds put together.
// (Fixed-point slices: Ozaki, Ogita, Oishi, Rump, "Error-free transformations of matrix multiplication by using fast
// routines of matrix multiplication", 2012.)  The digits of K lie one under the other, so digit i of Q times all of K's
// digits that count is one product of width 64 (4 - i): the accumulators stand side by side, each i starts one further on.
//
// What is left out of a score (r, i + j > 4) is about 2^-33 of 2^(eq + ek), whatever the score is, so it matters that a row's large
// elements meet large ones.  Two things see to it.  (1) Features are balanced: each is multiplied by a power of two in Q and
// divided by it in K, so that all features are of one size in the tile's queries (by the mean exponents of 32 of them; not where
// all are alike anyway): gains that cancel between Q and K, or a feature that is large in one and small in the other, cost no bits.  (2) A row whose largest score is
// still below 2^(eq + ek - 4), that is where 2^(eq + ek - 33) exceeds 2^-29 of it (of probabilities: of the larger of it and 1,
// scaled), is made again with dots in double.  Errors against float64, by rounding to f32 alone 1: normal elements 1.000, gains of
// 2^+-2 to 2^+-12 a feature 1.001, spread of 2^+-12 within the rows 1.001, queries orthogonal to ten times as large a mean of the keys 1.005.
//
// Output sums.  P and V as three bf16 pieces each, six piece products by the same scheme, 64 keys at a time: three
// accumulators, added in f32 registers.
//
// One CTA has 128 queries of one (sequence, head) and takes 64 keys a step.  Four warps cut K and V into a ring of two
// stages; one warp issues; eight warps have two threads to a row, 32 keys each: they put the scores together, take the
// exponentials, write P's pieces where K's digits were (a stage's K is no longer needed then) and add the step's sums
// before.  The exponents follow a row's maximum lazily (they are relative to an earlier maximum until that is exceeded by 8), so
// one walk over the keys does; with probabilities to be stored (the cached form) a first walk takes the statistics.
//
// A row whose elements are not finite, or beyond 2^90 or all below 2^-90, has no such digits, and V beyond 1e28 might overflow
// in sums that are not normalised yet: the rows concerned (of an odd key, those that see it) are made again likewise, after the
// rest, up to 65 at a time by all warps of the CTA (Again); a tile of nothing but such rows is not walked at all.  NaN needs no such
// thing: it goes through a row's scale into its scores.  Measured on a B200, us, 8 x 512 positions of 12 heads of 64, statistics /
// probabilities / raw scores: 72.5 / 116 / 58.4; gains of 2^+-10 a feature 74.2 / 117 / 60.7; all NaN 73.2 / 116 / 57.3; an infinite element in
// one query 86 / 124 / 59.2; every row again 325 / 394 / 140 (the tile kernels, whatever the elements: 174 / 184 / 87.7; with neither
// balance nor test: 70.9 / 115 / 56.7).
//
// Every wait on an mbarrier is bounded; one that runs out raises DeviceStatus::wait_timeout and the CTA stores nothing.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <initializer_list>
#include <type_traits>

#include "kernels.h"
#include "launch.cuh"
#include "umma_device.cuh"

namespace see::k {

namespace {

using namespace umma_dev;

constexpr uint32_t kRows = 128, kKeys = 64, kWidth = 64;   // queries of a CTA, keys of a step, widest head
constexpr uint32_t kWorkWarps = 8, kCutWarps = 4, kWarps = kWorkWarps + kCutWarps + 1, kThreads = 32 * kWarps;
constexpr uint32_t kQSlice = kRows * 128, kKSlice = kKeys * 128, kPPiece = kRows * 128, kVPiece = kKeys * 128;
constexpr uint32_t kStageBytes = 3 * kPPiece + 3 * kVPiece;   // K's four digits, then P's three pieces; V's pieces behind
static_assert(4 * kKSlice <= 3 * kPPiece, "K's digits lie where P's pieces come");
constexpr uint32_t kParts = kWorkWarps / 4, kOwn = kKeys / kParts;   // threads to a row; keys (and features) of each
constexpr uint32_t kScoreCols = 5 * kKeys;                    // tensor memory: five accumulators of scores, three of sums
constexpr uint32_t kGroups = 4, kGroupRows = 8, kFirst = 8;   // rows that features are balanced by; rows of dP that are always dots in double
constexpr float kSlack = 8.0f;                                // how far a row's maximum may exceed its reference

enum class Form { kTiled, kCached, kScores };   // statistics; probabilities and statistics; raw scores (dP = dO V^T)

struct __align__(16) SliceCtl {
  float q_scale[kRows], k_scale[4][kKeys];   // (a step's is read after its stage may have gone on: four in turns)
  float gain[kWidth], ungain[kWidth];        // the features' powers of two: K's (V's) and Q's (dO's)
  uint2 sample[kGroups][kWidth / 2];         // of a group of queries' elements, by feature: how many, and the sum of their exponents
  double first[kFirst][kFirst];              // the first scores of a sequence
  float row_max[2][kParts][kRows];           // by parity of the step
  double denom[kParts][kRows];
  uint64_t k_full[2], v_full[2], stage_empty[2], s_full, s_empty, p_full, sum_full;
  uint32_t tmem_base;
  volatile size_t base;                      // the tile: where its (sequence, head) begins, which it is, its first query (read again
  volatile uint32_t bh, i0;                  // where they are needed: registers are short)
  volatile uint32_t failed;
  uint32_t k_top;                            // the largest scale of the keys, its bits
  uint32_t odd_rows[kRows / 32];             // a bit for each row of queries without digits ...
  uint32_t again[kRows / 32];                // ... and for each whose scores are too small for what the digits leave out:
  uint32_t nan_rows[kRows / 32];             // (rows that are NaN as they are)
  uint32_t odd_key, odd_value;               // these are made again, and all that see this key, or this row of V
  volatile uint32_t some;                    // there are any
  uint8_t list[kRows];                       // those rows, in order
};
constexpr uint32_t kSlabFloats = 32 * 8;     // a working warp's 32 x 8 f32 on their way out
constexpr size_t kSliceSmem = 1024 + 4 * kQSlice + 2 * kStageBytes + sizeof(SliceCtl);
static_assert(kSliceSmem <= 227 * 1024, "one CTA per SM");

struct SliceArgs {
  const float *q, *k, *v;
  float *o, *probs, *stats;
  uint32_t BH, S, H, d;
  float inv_sqrt_d;
  int store16;   // the score matrix takes 16-byte stores
  DeviceStatus* status;
};

// Sixteen elements of a row, zero outside the matrix.
__device__ __forceinline__ void FetchSixteen(float (&x)[16], const float* __restrict__ row, bool live, uint32_t c0, uint32_t d) {
#pragma unroll
  for (uint32_t q = 0; q < 4; ++q) {
    const uint32_t c = c0 + 4 * q;
    const float4 f = live && c < d ? __ldg(reinterpret_cast<const float4*>(row + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
    x[4 * q] = f.x; x[4 * q + 1] = f.y; x[4 * q + 2] = f.z; x[4 * q + 3] = f.w;
  }
}
// Sixteen elements times their features' factors.
__device__ __forceinline__ void ScaleSixteen(float (&x)[16], const float* gain, uint32_t c0) {
#pragma unroll
  for (int e = 0; e < 16; e += 4) {
    const float4 g = *reinterpret_cast<const float4*>(gain + c0 + e);
    x[e] *= g.x; x[e + 1] *= g.y; x[e + 2] *= g.z; x[e + 3] *= g.w;
  }
}
// The digits of a row that four neighbouring lanes hold; the factor that undoes its scale, which is NaN where an element is: its
// scores are NaN then.  *odd: it has none.
__device__ __forceinline__ float CutDigits(float (&x)[16], uint8_t* dst, uint32_t slice_bytes, uint32_t row, uint32_t c0, bool* odd) {
  uint32_t top = 0;   // the largest magnitude's bits (a NaN's are larger than any number's)
#pragma unroll
  for (int e = 0; e < 16; ++e) top = max(top, __float_as_uint(x[e]) & 0x7FFFFFFFu);
  top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, 1));
  top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, 2));
  const bool none = top >= 0x6C800000u || (top != 0 && top < 0x12800000u), nan = top > 0x7F800000u;   // 2^90, 2^-90
  *odd = none && !nan;
  const uint32_t ex = top >> 23;
  const float to = none ? 0.0f : (top == 0 ? 1.0f : __uint_as_float((261u - ex) << 23));                      // 2^(8 - e)
  const float back = nan ? NAN : none || top == 0 ? 0.0f : __uint_as_float((ex - 7u) << 23);             // 2^(e - 8)
#pragma unroll
  for (int e = 0; e < 16; ++e) x[e] = none ? 0.0f : x[e] * to;
  constexpr float kMagic = 12582912.0f;   // 1.5 * 2^23: adding and taking it away rounds to a whole number
#pragma unroll
  for (uint32_t i = 0; i < 4; ++i) {
    uint32_t w[8];
#pragma unroll
    for (int e = 0; e < 16; e += 2) {
      const float a = __fsub_rn(__fadd_rn(x[e], kMagic), kMagic), b = __fsub_rn(__fadd_rn(x[e + 1], kMagic), kMagic);
      w[e / 2] = PackBf16x2(a, b);
      x[e] = (x[e] - a) * 256.0f;
      x[e + 1] = (x[e + 1] - b) * 256.0f;
    }
    uint8_t* at = dst + i * slice_bytes;
    *reinterpret_cast<uint4*>(at + Sw128Offset(row, c0 / 8)) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4*>(at + Sw128Offset(row, c0 / 8 + 1)) = make_uint4(w[4], w[5], w[6], w[7]);
  }
  return back;
}
// An element of the sample: one, and its exponent; nothing of zeros and of what is not finite.
__device__ __forceinline__ uint32_t CountExponent(float f) {
  const uint32_t e = __float_as_uint(f) >> 23 & 0xFFu;
  return e - 1u < 254u ? (1u << 16) + e : 0u;
}
// The features' powers of two, from the means of their exponents, by every warp for itself (all write the same).  False: none is
// worth it, they are all within a factor of six of the middle, or of sixteen of one another.  (The kernel's code is cold at most of
// its launches: as little as can be comes before the first products.)
__device__ __forceinline__ bool BalanceFeatures(SliceCtl* ctl) {
  const uint32_t lane = threadIdx.x & 31;
  uint2 v = make_uint2(0, 0);
#pragma unroll
  for (uint32_t g = 0; g < kGroups; ++g) {
    const uint2 f = ctl->sample[g][lane];
    v = make_uint2(v.x + f.x, v.y + f.y);
  }
  // Mostly as many of each, and no two sums more than four powers of two an element apart: nothing to divide.
  const uint32_t most = __reduce_max_sync(0xFFFFFFFFu, max(v.x, v.y));
  const uint32_t least = __reduce_min_sync(0xFFFFFFFFu, min(v.x != 0 ? v.x : ~0u, v.y != 0 ? v.y : ~0u));
  if (most - least <= 4 * kGroups * kGroupRows) return false;
  auto mean = [](uint32_t w) {   // in eighths
    return __float2int_rn(__fdividef(static_cast<float>((w & 0xFFFFu) * 8), fmaxf(static_cast<float>(w >> 16), 1.0f)));
  };
  const int m0 = mean(v.x), m1 = mean(v.y);
  const int all = __reduce_add_sync(0xFFFFFFFFu, m0 + m1 + (v.x != 0 ? 1 << 20 : 0) + (v.y != 0 ? 1 << 20 : 0));
  const int middle = __float2int_rn(__fdividef(static_cast<float>(all & 0xFFFFF), fmaxf(static_cast<float>(all >> 20), 1.0f)));
  const int off0 = v.x != 0 ? m0 - middle : 0, off1 = v.y != 0 ? m1 - middle : 0;
  if (!__any_sync(0xFFFFFFFFu, max(abs(off0), abs(off1)) > 20)) return false;
  const int by0 = max(-64, min(64, (off0 + 4) >> 3)), by1 = max(-64, min(64, (off1 + 4) >> 3));
  *reinterpret_cast<float2*>(ctl->gain + 2 * lane) = make_float2(__uint_as_float((127 + by0) << 23), __uint_as_float((127 + by1) << 23));
  *reinterpret_cast<float2*>(ctl->ungain + 2 * lane) = make_float2(__uint_as_float((127 - by0) << 23), __uint_as_float((127 - by1) << 23));
  __syncwarp();
  return true;
}
// Two elements' bf16 pieces, packed.
__device__ __forceinline__ void CutPieces(float lo, float hi, uint32_t (&p)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    p[i] = PackBf16x2(lo, hi);
    if (i < 2) {
      lo = lo - __uint_as_float(p[i] << 16);
      hi = hi - __uint_as_float(p[i] & 0xFFFF0000u);
    }
  }
}

// A positive f32 as a double (a conversion is a sixteenth of an add's rate; 0 becomes 2^-127).
__device__ __forceinline__ double Widen(float x) {
  const uint32_t bits = __float_as_uint(x);
  return __hiloint2double(static_cast<int>((bits >> 3) + 0x38000000u), static_cast<int>(bits << 29));
}

__device__ __forceinline__ bool SliceWait(SliceCtl* ctl, uint64_t* bar, uint32_t parity) {   // a whole warp
  bool there = ctl->failed == 0 && MbarWait(bar, parity);
  there = __all_sync(0xFFFFFFFFu, there);
  if (!there) ctl->failed = 1;
  return there;
}

// Rows `first` to first + count of the list as the tile kernels' expressions have them, up to kSlots of each warp together: keys
// 64 at a time as doubles in shared memory (a conversion costs four multiply-adds), the next 64 on their way in registers, each
// dot one chain over ascending features.  Softmax forms walk the keys twice: each lane's maximum and sum, then the probabilities
// and their products with V.
constexpr uint32_t kAgainSlots = 5, kAgainLd = kKeys + 1;
struct AgainSmem {
  double k[kKeys * kAgainLd];                      // [key][feature]
  double q[kWarps * kAgainSlots * kWidth];
  float v[kKeys * kWidth];
  float w[kWarps * kAgainSlots * kKeys];           // probabilities
};
static_assert(sizeof(AgainSmem) <= 4 * kQSlice + 2 * kStageBytes, "in the place of the digits");

__device__ __noinline__ double AgainExp(double x) { return exp(x); }
template <Form kForm>
__device__ __noinline__ void Again(const SliceArgs a, AgainSmem* sm, const SliceCtl* ctl, uint32_t bh, uint32_t i0, uint32_t first,
                                   uint32_t count) {
  constexpr uint32_t kSlots = kAgainSlots;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const size_t D = static_cast<size_t>(a.H) * a.d;
  const size_t base = ctl->base;
  uint32_t row[kSlots];
  bool mine[kSlots];
  uint32_t nearest = a.S;
  double* q = sm->q + warp * kSlots * kWidth;
  float* w = sm->w + warp * kSlots * kKeys;
#pragma unroll
  for (uint32_t s = 0; s < kSlots; ++s) {
    mine[s] = warp + kWarps * s < count;
    row[s] = i0 + ctl->list[first + (mine[s] ? warp + kWarps * s : 0)];
    nearest = min(nearest, row[s]);
#pragma unroll
    for (uint32_t h = 0; h < 2; ++h) {
      const uint32_t c = lane + 32 * h;
      q[s * kWidth + c] = c < a.d ? static_cast<double>(a.q[base + static_cast<size_t>(row[s]) * D + c]) : 0.0;
    }
  }
  const uint32_t chunks = (i0 + ctl->list[first + count - 1]) / kKeys + 1;
  constexpr uint32_t kQuads = kKeys * kWidth / 4, kEach = (kQuads + kThreads - 1) / kThreads;
  float4 kf[kEach], vf[kEach];
  auto fetch = [&](float4 (&f)[kEach], const float* src, uint32_t chunk) {
#pragma unroll
    for (uint32_t e = 0; e < kEach; ++e) {
      const uint32_t idx = threadIdx.x + e * kThreads, key = chunk * kKeys + idx / (kWidth / 4), c = idx % (kWidth / 4) * 4;
      f[e] = idx < kQuads && key < a.S && c < a.d ? __ldg(reinterpret_cast<const float4*>(src + base + static_cast<size_t>(key) * D + c))
                                                   : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  // The dots of a slot's row with keys lane and lane + 32 of the chunk in shared memory, in f32.
  float dot[kSlots][2] = {};
  auto dots = [&] {
    double acc[kSlots][2] = {};
    const double *k0 = sm->k + lane * kAgainLd, *k1 = k0 + 32 * kAgainLd;
    if (!mine[0]) return;
#pragma unroll 2
    for (uint32_t c = 0; c < a.d; c += 2) {   // (d is a multiple of four)
      const double x0 = k0[c], x1 = k0[c + 1], y0 = k1[c], y1 = k1[c + 1];
#pragma unroll
      for (uint32_t s = 0; s < kSlots; ++s) {
        if (!mine[s]) continue;
        const double2 f = *reinterpret_cast<const double2*>(q + s * kWidth + c);
        acc[s][0] = fma(f.x, x0, acc[s][0]);
        acc[s][0] = fma(f.y, x1, acc[s][0]);
        acc[s][1] = fma(f.x, y0, acc[s][1]);
        acc[s][1] = fma(f.y, y1, acc[s][1]);
      }
    }
#pragma unroll
    for (uint32_t s = 0; s < kSlots; ++s) {
      dot[s][0] = static_cast<float>(acc[s][0]);
      dot[s][1] = static_cast<float>(acc[s][1]);
    }
  };
  // f(chunk) with each chunk of keys (and, where wanted, of V) in shared memory.
  auto walk = [&](bool values, auto f) {
    fetch(kf, a.k, 0);
    if (values) fetch(vf, a.v, 0);
    for (uint32_t chunk = 0; chunk < chunks; ++chunk) {
      __syncthreads();
#pragma unroll
      for (uint32_t e = 0; e < kEach; ++e) {
        const uint32_t idx = threadIdx.x + e * kThreads;
        if (idx >= kQuads) continue;
        double* k = sm->k + idx / (kWidth / 4) * kAgainLd + idx % (kWidth / 4) * 4;
        k[0] = kf[e].x; k[1] = kf[e].y; k[2] = kf[e].z; k[3] = kf[e].w;
        if (values) *reinterpret_cast<float4*>(sm->v + idx * 4) = vf[e];
      }
      __syncthreads();
      if (chunk + 1 < chunks) {
        fetch(kf, a.k, chunk + 1);
        if (values) fetch(vf, a.v, chunk + 1);
      }
      f(chunk);
    }
  };
  auto to_probs = [&](uint32_t s, uint32_t j, float x) {
    if (mine[s] && j < a.S) a.probs[(static_cast<size_t>(bh) * a.S + row[s]) * a.S + j] = x;
  };
  if constexpr (kForm == Form::kScores) {
    walk(false, [&](uint32_t chunk) {
      dots();
#pragma unroll
      for (uint32_t s = 0; s < kSlots; ++s)
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
          const uint32_t j = chunk * kKeys + lane + 32 * h;
          to_probs(s, j, j <= row[s] ? dot[s][h] : 0.0f);
        }
    });
  } else {
    float top[kSlots], inv[kSlots];
    {
      double sum[kSlots];   // of this lane's keys, relative to its maximum
#pragma unroll
      for (uint32_t s = 0; s < kSlots; ++s) { top[s] = -INFINITY; sum[s] = 0.0; }
      walk(false, [&](uint32_t chunk) {
        dots();
#pragma unroll
        for (uint32_t s = 0; s < kSlots; ++s)
#pragma unroll
          for (uint32_t h = 0; h < 2; ++h) {
            const float x = __fmul_rn(dot[s][h], a.inv_sqrt_d);   // (and no fused difference: a maximum's is 0)
            if (chunk * kKeys + lane + 32 * h > row[s] || x == -INFINITY) continue;
            if (x > top[s]) {
              sum[s] *= AgainExp(static_cast<double>(top[s]) - static_cast<double>(x));   // (0 before the first)
              top[s] = x;
            }
            sum[s] += static_cast<double>(expf(x - top[s]));
          }
      });
#pragma unroll
      for (uint32_t s = 0; s < kSlots; ++s) {
        float all = top[s];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) all = fmaxf(all, __shfl_xor_sync(0xFFFFFFFFu, all, o));
        // (A lane of NaN alone has no maximum of its own; a row of -inf alone has no sum: NaN, as an exponential of inf - inf.)
        double part = top[s] == all ? sum[s] : top[s] == -INFINITY ? (sum[s] == 0.0 ? 0.0 : NAN)
                                             : sum[s] * AgainExp(static_cast<double>(top[s]) - static_cast<double>(all));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xFFFFFFFFu, part, o);
        top[s] = all;
        inv[s] = all == -INFINITY ? NAN : 1.0f / static_cast<float>(part);
      }
    }
    float acc[kSlots][2] = {};
    walk(true, [&](uint32_t chunk) {
      dots();
#pragma unroll
      for (uint32_t s = 0; s < kSlots; ++s)
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
          const uint32_t j = chunk * kKeys + lane + 32 * h;
          const float p = j <= row[s] ? expf(__fmul_rn(dot[s][h], a.inv_sqrt_d) - top[s]) * inv[s] : 0.0f;
          if constexpr (kForm == Form::kCached) to_probs(s, j, p);
          w[s * kKeys + lane + 32 * h] = p;
        }
      __syncwarp();
      const bool all_seen = chunk * kKeys + kKeys - 1 <= nearest;   // (an unseen key's V may be NaN: it is passed by)
#pragma unroll 1
      for (uint32_t l = 0; l < kKeys; l += 4) {
        float x[4][2];
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
          x[e][0] = sm->v[(l + e) * kWidth + lane];
          x[e][1] = sm->v[(l + e) * kWidth + lane + 32];
        }
#pragma unroll
        for (uint32_t s = 0; s < kSlots; ++s) {
          if (!mine[s]) continue;
          const float4 p4 = *reinterpret_cast<const float4*>(w + s * kKeys + l);
          const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
          for (uint32_t e = 0; e < 4; ++e) {
            if (!all_seen && chunk * kKeys + l + e > row[s]) continue;
            acc[s][0] = fmaf(p[e], x[e][0], acc[s][0]);
            acc[s][1] = fmaf(p[e], x[e][1], acc[s][1]);
          }
        }
      }
      __syncwarp();
    });
#pragma unroll
    for (uint32_t s = 0; s < kSlots; ++s) {
      if (!mine[s]) continue;
      float* o = a.o + base + static_cast<size_t>(row[s]) * D;
      if (lane < a.d) o[lane] = acc[s][0];
      if (lane + 32 < a.d) o[lane + 32] = acc[s][1];
      if (a.stats && lane == 0)
        *reinterpret_cast<float4*>(a.stats + (static_cast<size_t>(bh) * a.S + row[s]) * kAttnStatsWidth) = make_float4(top[s], inv[s], 0.0f, 0.0f);
    }
  }
  if constexpr (kForm != Form::kTiled) {   // the keys no row of these sees
#pragma unroll
    for (uint32_t s = 0; s < kSlots; ++s)
      for (uint32_t j = chunks * kKeys + lane; j < a.S; j += 32) to_probs(s, j, 0.0f);
  }
  __syncthreads();
}

// A CTA's tile.
struct Place {
  uint32_t bh, i0, live, n;   // (sequence, head); its queries; steps of a walk over the keys
  size_t D, base;
  __device__ __forceinline__ Place(const SliceArgs& a, const SliceCtl* ctl) {
    bh = ctl->bh;
    i0 = ctl->i0;
    live = min(kRows, a.S - i0);
    n = (min(i0 + kRows, a.S) + kKeys - 1) / kKeys;
    D = static_cast<size_t>(a.H) * a.d;
    base = ctl->base;
  }
  __device__ __forceinline__ uint32_t RowsOf(uint32_t w) const {   // the 32 rows of a word, those there are
    return live >= 32 * w + 32 ? 0xFFFFFFFFu : live > 32 * w ? (1u << (live - 32 * w)) - 1 : 0u;
  }
  __device__ __forceinline__ bool Without(const SliceCtl* ctl) const {   // not one row has digits
    bool none = true;
#pragma unroll
    for (uint32_t w = 0; w < kRows / 32; ++w) none = none && ctl->odd_rows[w] == RowsOf(w);
    return none;
  }
};
// Behind the tile: the first scores, and rows that are made again.
template <Form kForm>
__device__ __forceinline__ void Finish(const SliceArgs& a, AgainSmem* sm, SliceCtl* ctl) {
  const Place at(a, ctl);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (kForm == Form::kScores && at.i0 == 0 && !at.Without(ctl) && threadIdx.x < kFirst * kFirst) {
    const uint32_t i = threadIdx.x / kFirst, j = threadIdx.x % kFirst;
    if (i < a.S && j <= i) a.probs[(static_cast<size_t>(at.bh) * a.S + i) * a.S + j] = static_cast<float>(ctl->first[i][j]);
  }
  if (ctl->some == 0) return;
  uint32_t words[kRows / 32], count = 0;
#pragma unroll
  for (uint32_t w = 0; w < kRows / 32; ++w) {
    auto see = [&](uint32_t key) {
      const uint32_t r0 = at.i0 + 32 * w;
      return key <= r0 ? 0xFFFFFFFFu : key - r0 >= 32 ? 0u : 0xFFFFFFFFu << (key - r0);
    };
    words[w] = (ctl->odd_rows[w] | ctl->again[w] | see(ctl->odd_key) | (see(ctl->odd_value) & ~ctl->nan_rows[w])) & at.RowsOf(w);
    count += __popc(words[w]);
  }
  if (count == 0) return;
  for (uint32_t w = 0, before = 0; w < kRows / 32; before += __popc(words[w]), ++w)
    if (warp == w && (words[w] >> lane & 1)) ctl->list[before + __popc(words[w] & ((1u << lane) - 1))] = static_cast<uint8_t>(32 * w + lane);
  __syncthreads();
  for (uint32_t first = 0; first < count; first += kWarps * kAgainSlots)
    Again<kForm>(a, sm, ctl, at.bh, at.i0, first, min(kWarps * kAgainSlots, count - first));
}

template <Form kForm>
__global__ void __launch_bounds__(kThreads, 1) AttnSliceKernel(const SliceArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* q_s = smem_raw + ((1024u - (SmemAddr(smem_raw) & 1023u)) & 1023u);
  uint8_t* ring = q_s + 4 * kQSlice;
  SliceCtl* ctl = reinterpret_cast<SliceCtl*>(ring + 2 * kStageBytes);

  const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      MbarInit(&ctl->k_full[s], kCutWarps);
      MbarInit(&ctl->v_full[s], kCutWarps);
      MbarInit(&ctl->stage_empty[s], 1);
    }
    MbarInit(&ctl->s_full, 1);
    MbarInit(&ctl->s_empty, kWorkWarps);
    MbarInit(&ctl->p_full, kWorkWarps);
    MbarInit(&ctl->sum_full, 1);
    ctl->failed = 0;
    ctl->odd_key = ctl->odd_value = 0xFFFFFFFFu;
    ctl->k_top = ctl->some = 0;
    for (uint32_t w = 0; w < kRows / 32; ++w) ctl->odd_rows[w] = ctl->again[w] = ctl->nan_rows[w] = 0;
    MbarInitFence();
    // Longest tiles first over the whole grid, so that the last wave is short ones.
    ctl->i0 = ((a.S + kRows - 1) / kRows - 1 - blockIdx.x / a.BH) * kRows;
    const uint32_t bh = blockIdx.x % a.BH;
    ctl->bh = bh;
    ctl->base = (static_cast<size_t>(bh / a.H) * a.S * a.H + bh % a.H) * a.d;
  }
  if (warp == kWorkWarps + kCutWarps) TmemAlloc(&ctl->tmem_base, 512);
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  AwaitPrevious();
  constexpr uint32_t tmem = 0;   // all 512 columns are this CTA's

  const Place at(a, ctl);
  const uint32_t i0 = at.i0, n = at.n;
  const uint32_t ahead = kForm == Form::kTiled ? 0 : n;                           // steps that only take scores
  const uint32_t total = kForm == Form::kCached ? 2 * n : n;
  const size_t D = at.D, base = at.base;
  constexpr uint32_t kEach = kKeys / (8 * kCutWarps);   // keys of a cutting thread in a step, 8 kCutWarps apart
  const uint32_t c0 = (threadIdx.x & 3) * 16;           // sixteen features of a thread that cuts
  auto fetch_keys = [&](float (&f)[kEach][16], const float* src, uint32_t u) {
#pragma unroll
    for (uint32_t h = 0; h < kEach; ++h) {
      const uint32_t key = (u < n ? u : u - n) * kKeys + ((threadIdx.x - 32 * kWorkWarps) >> 2) + h * 8 * kCutWarps;
      FetchSixteen(f[h], src + base + static_cast<size_t>(key) * D, u < total && key < a.S, c0, a.d);
    }
  };
  float k_next[kEach][16];   // a step's keys, on their way since the step before
  bool balanced;
  {   // the queries' digits, by whole warps; all that the first step needs of memory is asked for at once
    constexpr uint32_t kLoaders = kWorkWarps + kCutWarps, kTwice = kRows / 8 - kLoaders;   // warps that have rows twice
    static_assert(kTwice <= kWorkWarps, "not those that have keys");
    float x[16], second[16];
    auto fetch = [&](float (&f)[16], uint32_t r) { FetchSixteen(f, a.q + base + static_cast<size_t>(i0 + r) * D, i0 + r < a.S, c0, a.d); };
    const bool samples = warp >= kTwice && warp < kTwice + kGroups;   // a group of the sample, two features to a lane
    static_assert(kTwice + kGroups <= kWorkWarps, "warps that have no second rows");
    float2 f[kGroupRows];
    if (samples && 2 * lane < a.d) {   // (first of all: everything waits for it)
      const bool many = at.live >= kGroups * kGroupRows;   // (of few, every group has the first)
      uint32_t row = many ? (warp - kTwice) * at.live / kGroups : 0;
      const uint32_t step = many ? at.live / (kGroups * kGroupRows) : 1;
#pragma unroll
      for (uint32_t r = 0; r < kGroupRows; ++r) {
        f[r] = __ldg(reinterpret_cast<const float2*>(a.q + base + static_cast<size_t>(i0 + row) * D + 2 * lane));
        row = row + step < at.live ? row + step : 0;
      }
    }
    if (warp < kLoaders) fetch(x, threadIdx.x >> 2);
    if (warp < kTwice) fetch(second, 8 * kLoaders + (threadIdx.x >> 2));
    if (warp >= kWorkWarps && warp < kLoaders) fetch_keys(k_next, a.k, 0);
    if (samples) {
      uint2 v = make_uint2(0, 0);
#pragma unroll
      for (uint32_t r = 0; r < kGroupRows; ++r) v = make_uint2(v.x + CountExponent(f[r].x), v.y + CountExponent(f[r].y));
      ctl->sample[warp - kTwice][lane] = 2 * lane < a.d ? v : make_uint2(0, 0);
    }
    __syncthreads();
    balanced = BalanceFeatures(ctl);
    if (warp < kLoaders) {
#pragma unroll 1
      for (uint32_t r = threadIdx.x >> 2;;) {
        bool odd;
        if (balanced) ScaleSixteen(x, ctl->ungain, c0);
        const float back = CutDigits(x, q_s, kQSlice, r, c0, &odd);
        if (c0 == 0) {
          ctl->q_scale[r] = back * (kForm == Form::kScores ? 1.0f : a.inv_sqrt_d);
          if (odd) {
            atomicOr(&ctl->odd_rows[r / 32], 1u << (r & 31));
            ctl->some = 1;
          }
        }
        __syncwarp();
        r += 8 * kLoaders;
        if (r >= kRows) break;   // (whole warps)
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = second[e];
      }
      FenceProxyAsync();
    }
  }
  __syncthreads();

  bool ok = true;
  if (at.Without(ctl)) {
  } else if (warp == kWorkWarps + kCutWarps) {
    // ---- products (the whole warp walks and waits; one elected lane issues) ----
    const uint32_t k_steps = (a.d + 15) / 16;
    auto scores = [&](uint32_t u) {
      uint8_t* stage = ring + (u & 1) * kStageBytes;
      ok = ok && SliceWait(ctl, &ctl->k_full[u & 1], (u >> 1) & 1);
      if (u > 0) ok = ok && SliceWait(ctl, &ctl->s_empty, (u - 1) & 1);
      if (!ok) return;
      TcFenceAfter();
      if (ElectOne()) {
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
          const uint64_t da = MakeSmemDesc(SmemAddr(q_s + i * kQSlice)), db = MakeSmemDesc(SmemAddr(stage));
          const uint32_t idesc = MakeInstrDesc(128, kKeys * (i == 0 ? 4 : 5 - i));
          for (uint32_t k = 0; k < k_steps; ++k) {
            if (i == 1) {   // the fifth accumulator begins with the last digit
              UmmaBf16(tmem + kKeys * 1, da + 2 * k, db + 2 * k, MakeInstrDesc(128, kKeys * 3), 1u);
              UmmaBf16(tmem + kKeys * 4, da + 2 * k, db + 2 * k + (3 * kKSlice >> 4), MakeInstrDesc(128, kKeys), k != 0 ? 1u : 0u);
            } else {
              UmmaBf16(tmem + kKeys * i, da + 2 * k, db + 2 * k, idesc, (i | k) != 0 ? 1u : 0u);
            }
          }
        }
        UmmaCommit(&ctl->s_full);
        if (kForm != Form::kTiled && u < ahead) UmmaCommit(&ctl->stage_empty[u & 1]);
      }
      __syncwarp();
    };
    scores(0);
    for (uint32_t u = 0; u < total; ++u) {
      if (u + 1 < total) scores(u + 1);
      if constexpr (kForm != Form::kTiled)
        if (u < ahead) continue;
      ok = ok && SliceWait(ctl, &ctl->v_full[u & 1], (u >> 1) & 1);
      ok = ok && SliceWait(ctl, &ctl->p_full, (u - ahead) & 1);
      if (!ok) break;
      TcFenceAfter();
      if (ElectOne()) {
        const uint32_t p = SmemAddr(ring + (u & 1) * kStageBytes), v = p + 3 * kPPiece;
#pragma unroll
        for (uint32_t i = 0; i < 3; ++i) {
          const uint64_t da = MakeSmemDesc(p + i * kPPiece);
          const uint32_t idesc = MakeInstrDesc(128, kWidth * (3 - i)) | kInstrDescBMnMajor;
#pragma unroll
          for (uint32_t k = 0; k < 4; ++k)
            UmmaBf16(tmem + kScoreCols + kWidth * i, da + 2 * k, MakeSmemDescMn(v + k * 2048, kVPiece), idesc, (i | k) != 0 ? 1u : 0u);
        }
        UmmaCommit(&ctl->sum_full);
        UmmaCommit(&ctl->stage_empty[u & 1]);
      }
      __syncwarp();
    }
  } else if (warp >= kWorkWarps) {
    // ---- K's digits, V's pieces ----
    const uint32_t t = threadIdx.x - 32 * kWorkWarps, r0 = t >> 2;
    float y[kEach][16];
    auto row_of = [&](uint32_t h) { return r0 + h * 8 * kCutWarps; };
    auto sums_at = [&](uint32_t u) { return kForm == Form::kTiled || (kForm == Form::kCached && u >= ahead && u < total); };
    float top = 0.0f;   // the largest scale of this thread's keys
    if (sums_at(0)) fetch_keys(y, a.v, 0);
    for (uint32_t u = 0; u < total && ok; ++u) {
      const uint32_t s = u & 1;
      uint8_t* stage = ring + s * kStageBytes;
      if (u >= 2) ok = SliceWait(ctl, &ctl->stage_empty[s], ((u >> 1) - 1) & 1);
      if (!ok) break;
      const uint32_t key0 = (u < n ? u : u - n) * kKeys;
      if (balanced) {
#pragma unroll
        for (uint32_t h = 0; h < kEach; ++h) ScaleSixteen(k_next[h], ctl->gain, c0);
      }
      bool odd[kEach];   // (looked at behind the loop: the rows' cutting is one stream of instructions)
#pragma unroll
      for (uint32_t h = 0; h < kEach; ++h) {
        const float back = CutDigits(k_next[h], stage, kKSlice, row_of(h), c0, &odd[h]);
        if (c0 == 0) ctl->k_scale[u & 3][row_of(h)] = back;
        top = fmaxf(top, back);
      }
      if (u + 1 == n) atomicMax(&ctl->k_top, __float_as_uint(top));   // (all keys': the workers read it behind this step's scores)
      auto least = [&] {
        uint32_t at = 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t h = 0; h < kEach; ++h) at = min(at, odd[h] ? key0 + row_of(h) : 0xFFFFFFFFu);
        return at;
      };
      if (least() != 0xFFFFFFFFu) {
        atomicMin(&ctl->odd_key, least());
        ctl->some = 1;
      }
      FenceProxyAsync();
      __syncwarp();
      if (lane == 0) MbarArrive(&ctl->k_full[s]);
      fetch_keys(k_next, a.k, u + 1);
      if (sums_at(u)) {   // V's pieces while the scores are formed
        // (Sums of up to 2^23 weights of up to e^kSlack stay finite; rows that do not see the key see zeros.)
#pragma unroll
        for (uint32_t h = 0; h < kEach; ++h) {
          odd[h] = false;
#pragma unroll
          for (int e = 0; e < 16; ++e) odd[h] = odd[h] || !(fabsf(y[h][e]) < 1e28f);
        }
        if (least() != 0xFFFFFFFFu) {
          atomicMin(&ctl->odd_value, least());
          ctl->some = 1;
#pragma unroll
          for (uint32_t h = 0; h < kEach; ++h)
#pragma unroll
            for (int e = 0; e < 16; ++e) y[h][e] = odd[h] ? 0.0f : y[h][e];
        }
#pragma unroll
        for (uint32_t h = 0; h < kEach; ++h) {
          uint32_t w[3][8];
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            uint32_t p[3];
            CutPieces(y[h][e], y[h][e + 1], p);
#pragma unroll
            for (int i = 0; i < 3; ++i) w[i][e / 2] = p[i];
          }
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            uint8_t* at = stage + 3 * kPPiece + i * kVPiece;
            *reinterpret_cast<uint4*>(at + Sw128Offset(row_of(h), c0 / 8)) = make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]);
            *reinterpret_cast<uint4*>(at + Sw128Offset(row_of(h), c0 / 8 + 1)) = make_uint4(w[i][4], w[i][5], w[i][6], w[i][7]);
          }
        }
        FenceProxyAsync();
        __syncwarp();
      }
      if (lane == 0) MbarArrive(&ctl->v_full[s]);   // (every step: its phases are the stage's)
      if (sums_at(u + 1)) fetch_keys(y, a.v, u + 1);
    }
    if (kForm == Form::kScores && i0 == 0) {   // two threads to a pair of the first rows
      const uint32_t i = t >> 4, j = t >> 1 & 7, half = t & 1;
      static_assert(kForm != Form::kScores || kFirst * kFirst * 2 == 32 * kCutWarps, "all of them");
      double sum = 0.0;
      if (j <= i && i < a.S)
        for (uint32_t c = 4 * half; c < a.d; c += 8) {
          const float4 f = __ldg(reinterpret_cast<const float4*>(a.q + base + static_cast<size_t>(i) * D + c));
          const float4 g = __ldg(reinterpret_cast<const float4*>(a.k + base + static_cast<size_t>(j) * D + c));
          sum += static_cast<double>(f.x) * static_cast<double>(g.x) + static_cast<double>(f.y) * static_cast<double>(g.y) +
                 static_cast<double>(f.z) * static_cast<double>(g.z) + static_cast<double>(f.w) * static_cast<double>(g.w);
        }
      ctl->first[i][j] = sum + __shfl_xor_sync(0xFFFFFFFFu, sum, 1);
    }
  } else {
    // ---- scores, probabilities, sums: thread (row, part of the keys) ----
    const uint32_t quarter = warp & 3, part = warp >> 2, r = quarter * 32 + lane, i = i0 + r;
    const uint32_t t_s = tmem + ((quarter * 32) << 16) + part * kOwn, t_o = t_s + kScoreCols;
    const float q_scale = ctl->q_scale[r];
    float s[kOwn];
    [[maybe_unused]] float sum[kOwn];
    [[maybe_unused]] float top = -INFINITY, ref = -INFINITY, inv = 0.0f;   // the row's maximum; what its exponents are relative to
    [[maybe_unused]] double denom = 0.0;                                   // of this thread's keys, relative to ref
#pragma unroll
    for (int e = 0; e < kOwn; ++e) sum[e] = 0.0f;
    auto row_sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(1 + quarter), "n"(32 * kParts) : "memory"); };   // a quarter's rows

    auto take_scores = [&](uint32_t u) {
      ok = ok && SliceWait(ctl, &ctl->s_full, u & 1);
      const uint32_t key0 = (u < n ? u : u - n) * kKeys + part * kOwn;
      if (ok) {
        TcFenceAfter();
        const float* scale = ctl->k_scale[u & 3] + part * kOwn;
#pragma unroll
        for (uint32_t c = 0; c < kOwn; c += 16) {
          uint32_t x[16], y[16];
          TmemLoad16(t_s + 4 * kKeys + c, x);
          TmemLoad16(t_s + 3 * kKeys + c, y);
          TmemWaitLd();
#pragma unroll
          for (int e = 0; e < 16; ++e) s[c + e] = fmaf(__uint_as_float(x[e]), 0.00390625f, __uint_as_float(y[e]));
          TmemLoad16(t_s + 2 * kKeys + c, x);
          TmemLoad16(t_s + kKeys + c, y);
          TmemWaitLd();
#pragma unroll
          for (int e = 0; e < 16; ++e)
            s[c + e] = fmaf(fmaf(s[c + e], 0.00390625f, __uint_as_float(x[e])), 0.00390625f, __uint_as_float(y[e]));
          TmemLoad16(t_s + c, x);
          TmemWaitLd();
#pragma unroll
          for (int e = 0; e < 16; e += 4) {
            const float4 f = *reinterpret_cast<const float4*>(scale + c + e);
            s[c + e] = fmaf(s[c + e], 0.00390625f, __uint_as_float(x[e])) * q_scale * f.x;
            s[c + e + 1] = fmaf(s[c + e + 1], 0.00390625f, __uint_as_float(x[e + 1])) * q_scale * f.y;
            s[c + e + 2] = fmaf(s[c + e + 2], 0.00390625f, __uint_as_float(x[e + 2])) * q_scale * f.z;
            s[c + e + 3] = fmaf(s[c + e + 3], 0.00390625f, __uint_as_float(x[e + 3])) * q_scale * f.w;
          }
        }
        TcFenceBefore();
        __syncwarp();
        if (lane == 0) MbarArrive(&ctl->s_empty);
      }
      if (key0 + kOwn - 1 > i0 + quarter * 32) {   // some of these keys lie beyond some of these queries
        constexpr float kNone = kForm == Form::kScores ? 0.0f : -INFINITY;
#pragma unroll
        for (int e = 0; e < kOwn; ++e) s[e] = key0 + e <= i ? s[e] : kNone;
      }
      return key0;
    };
    // The row's maximum of this step, of all parts.
    auto step_top = [&](uint32_t u) {
      float m = s[0];
#pragma unroll
      for (int e = 1; e < kOwn; ++e) m = fmaxf(m, s[e]);
      ctl->row_max[u & 1][part][r] = m;
      row_sync();
#pragma unroll
      for (uint32_t p = 0; p < kParts; ++p) m = fmaxf(m, ctl->row_max[u & 1][p][r]);
      return m;
    };
    // s[e] becomes exp(s[e] - ref), and denom takes them in; returns the factor that older exponentials want.
    auto exponentials = [&](uint32_t u) {
      const float m = step_top(u);
      top = fmaxf(top, m);
      float factor = 1.0f;
      if (m > ref + kSlack) {   // always at a row's first key (ref = -inf)
        factor = expf(ref - m);
        ref = m;
        denom *= static_cast<double>(factor);
      }
      double d0 = 0.0, d1 = 0.0;
#pragma unroll
      for (int e = 0; e < kOwn; e += 2) {
        s[e] = expf(s[e] - ref);
        s[e + 1] = expf(s[e + 1] - ref);
        d0 += Widen(s[e]);
        d1 += Widen(s[e + 1]);
      }
      const double d = d0 + d1;
      denom += d < 0x1p100 ? d : NAN;   // (a NaN, widened, is 2^128)
      return factor;
    };
    // Eight columns of 32 rows of the score matrix at a time, through memory of the stage that holds neither K's digits nor,
    // yet, P's pieces: whole 32-byte sectors.
    auto store_scores = [&](uint32_t u, uint32_t key0) {
      static_assert(4 * kKSlice == 2 * kPPiece && kParts * kSlabFloats * 4 <= 32 * 128, "a quarter's slabs lie in its rows of P's third piece");
      float* slab = reinterpret_cast<float*>(ring + (u & 1) * kStageBytes + 2 * kPPiece + quarter * 32 * 128) + part * kSlabFloats;
#pragma unroll
      for (uint32_t c = 0; c < kOwn; c += 8) {
        __syncwarp();
#pragma unroll
        for (uint32_t q = 0; q < 2; ++q)
          *reinterpret_cast<float4*>(slab + lane * 8 + ((q ^ ((lane >> 2) & 1)) * 4)) =
              make_float4(s[c + 4 * q], s[c + 4 * q + 1], s[c + 4 * q + 2], s[c + 4 * q + 3]);
        __syncwarp();
#pragma unroll
        for (uint32_t x = 0; x < 2; ++x) {
          const uint32_t lr = x * 16 + (lane >> 1), q = lane & 1, row = i0 + quarter * 32 + lr, j = key0 + c + 4 * q;
          const float4 f = *reinterpret_cast<const float4*>(slab + lr * 8 + ((q ^ ((lr >> 2) & 1)) * 4));
          if (row >= a.S || j >= a.S) continue;
          float* to = a.probs + (static_cast<size_t>(ctl->bh) * a.S + row) * a.S + j;
          if (a.store16) {
            *reinterpret_cast<float4*>(to) = f;
          } else {
            to[0] = f.x;
            if (j + 1 < a.S) to[1] = f.y;
            if (j + 2 < a.S) to[2] = f.z;
            if (j + 3 < a.S) to[3] = f.w;
          }
        }
      }
    };
    auto add_sums = [&](uint32_t v) {   // of main step v
      ok = ok && SliceWait(ctl, &ctl->sum_full, v & 1);
      if (!ok) return;
      TcFenceAfter();
#pragma unroll
      for (uint32_t c = 0; c < kOwn; c += 16) {
        uint32_t x[16], y[16];
        TmemLoad16(t_o + 2 * kWidth + c, x);
        TmemLoad16(t_o + kWidth + c, y);
        TmemWaitLd();
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = __float_as_uint(__uint_as_float(x[e]) + __uint_as_float(y[e]));
        TmemLoad16(t_o + c, y);
        TmemWaitLd();
#pragma unroll
        for (int e = 0; e < 16; ++e) sum[c + e] += __uint_as_float(x[e]) + __uint_as_float(y[e]);
      }
      TcFenceBefore();
    };
    auto all_parts = [&] {   // the row's denominator
      ctl->denom[part][r] = denom;
      row_sync();
      double whole = 0.0;
#pragma unroll
      for (uint32_t p = 0; p < kParts; ++p) whole += ctl->denom[p][r];
      return whole;
    };
    // What the digits leave out, 2^-17 of both scales, against 2^-29 of the size that matters: beyond it the row is made again,
    // unless it is NaN.
    auto check = [&](float size, bool nan, bool exact = false) {
      const float k_top = __uint_as_float(ctl->k_top);
      const uint32_t none = __ballot_sync(0xFFFFFFFFu, nan);
      const uint32_t rows = __ballot_sync(0xFFFFFFFFu, !(q_scale * k_top <= 0x1p-12f * size && size < INFINITY) && i < a.S && !exact);
      if (part == 0 && lane == 0) {
        ctl->nan_rows[quarter] = none;
        ctl->again[quarter] = rows & ~none;
        if ((rows & ~none) != 0) ctl->some = 1;
      }
    };
    auto put_stats = [&](double whole) {   // relative to the maximum: the rows' statistics, and their factor
      inv = 1.0f / static_cast<float>(whole * exp(static_cast<double>(ref) - static_cast<double>(top)));
      check(fmaxf(1.0f, fabsf(top)), isnan(inv));
      if (a.stats && part == 0 && i < a.S && ok)
        *reinterpret_cast<float4*>(a.stats + (static_cast<size_t>(ctl->bh) * a.S + i) * kAttnStatsWidth) = make_float4(top, inv, 0.0f, 0.0f);
    };

    if constexpr (kForm == Form::kScores) {
      float size = 0.0f;
      for (uint32_t u = 0; u < n; ++u) {
        const uint32_t key0 = take_scores(u);
#pragma unroll
        for (int e = 0; e < kOwn; ++e) size = fmaxf(size, fabsf(s[e]));
        if (ok) store_scores(u, key0);
      }
      ctl->row_max[0][part][r] = size;
      row_sync();
#pragma unroll
      for (uint32_t p = 0; p < kParts; ++p) size = fmaxf(size, ctl->row_max[0][p][r]);
      check(size, isnan(q_scale), i < kFirst);
    } else {
      if constexpr (kForm == Form::kCached) {
        for (uint32_t u = 0; u < n; ++u) {
          take_scores(u);
          exponentials(u);
        }
        put_stats(all_parts());
      }
      for (uint32_t u = ahead; u < total; ++u) {
        const uint32_t v = u - ahead;
        const uint32_t key0 = take_scores(u);
        float factor = 1.0f;
        if constexpr (kForm == Form::kCached) {
#pragma unroll
          for (int e = 0; e < kOwn; ++e) s[e] = expf(s[e] - top) * inv;
          if (key0 + kOwn - 1 > i0 + quarter * 32) {   // (of a row that is NaN, too, the keys it does not see are 0)
#pragma unroll
            for (int e = 0; e < kOwn; ++e) s[e] = key0 + e <= i ? s[e] : 0.0f;
          }
          if (ok) store_scores(u, key0);
          row_sync();   // (a quarter's pieces and slabs share memory)
        } else {
          factor = exponentials(u);
        }
        if (v > 0) add_sums(v - 1);
        if (factor != 1.0f) {
#pragma unroll
          for (int e = 0; e < kOwn; ++e) sum[e] *= factor;
        }
        uint8_t* pieces = ring + (u & 1) * kStageBytes;
#pragma unroll
        for (uint32_t c = 0; c < kOwn; c += 8) {
          uint32_t w[3][4];
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            uint32_t p[3];
            CutPieces(s[c + e], s[c + e + 1], p);
#pragma unroll
            for (int x = 0; x < 3; ++x) w[x][e / 2] = p[x];
          }
          const uint32_t at = Sw128Offset(r, part * (kOwn / 8) + c / 8);
#pragma unroll
          for (int x = 0; x < 3; ++x)
            *reinterpret_cast<uint4*>(pieces + x * kPPiece + at) = make_uint4(w[x][0], w[x][1], w[x][2], w[x][3]);
        }
        FenceProxyAsync();
        __syncwarp();
        if (ok && lane == 0) MbarArrive(&ctl->p_full);
      }
      add_sums(total - ahead - 1);
      float scale = 1.0f;   // (the cached form's probabilities are what was summed)
      if constexpr (kForm == Form::kTiled) {
        const double whole = all_parts();
        put_stats(whole);
        scale = static_cast<float>(1.0 / whole);
      }
      // All products are complete: the rows leave through the ring's memory, 16-byte chunks XOR-ed with the row.
      float* tile_o = reinterpret_cast<float*>(ring);
      asm volatile("bar.sync 5, %0;" ::"n"(32 * kWorkWarps) : "memory");   // (the last products have read P)
#pragma unroll
      for (uint32_t q = 0; q < kOwn / 4; ++q)
        *reinterpret_cast<float4*>(tile_o + r * kWidth + (((part * (kOwn / 4) + q) ^ (r & 15)) * 4)) =
            make_float4(sum[4 * q] * scale, sum[4 * q + 1] * scale, sum[4 * q + 2] * scale, sum[4 * q + 3] * scale);
      asm volatile("bar.sync 5, %0;" ::"n"(32 * kWorkWarps) : "memory");
      const uint32_t chunk = threadIdx.x & 15;
      if (ok && 4 * chunk < a.d)
        for (uint32_t row = threadIdx.x >> 4; row < kRows && i0 + row < a.S; row += 2 * kWorkWarps)
          if (((ctl->odd_rows[row / 32] | ctl->again[row / 32]) >> (row & 31) & 1) == 0 && i0 + row < ctl->odd_key &&
              (i0 + row < ctl->odd_value || (ctl->nan_rows[row / 32] >> (row & 31) & 1) != 0)) *reinterpret_cast<float4*>(a.o + ctl->base + static_cast<size_t>(i0 + row) * a.H * a.d + 4 * chunk) =
              *reinterpret_cast<const float4*>(tile_o + row * kWidth + ((chunk ^ (row & 15)) * 4));
    }
    if constexpr (kForm != Form::kTiled) {   // the keys no walk reaches
      for (uint32_t row = warp; ok && row < kRows && i0 + row < a.S; row += kWorkWarps) {
        float* to = a.probs + (static_cast<size_t>(ctl->bh) * a.S + i0 + row) * a.S;
        for (uint32_t j = n * kKeys + lane; j < a.S; j += 32) to[j] = 0.0f;
      }
    }
  }
  __syncwarp();
  TcFenceBefore();
  __syncthreads();
  if (ctl->failed) {
    if (threadIdx.x == 0) a.status->wait_timeout = 1;
    DrainDelay();
    __syncthreads();
  }
  if (warp == kWorkWarps + kCutWarps) {
    TcFenceAfter();
    TmemFree(ctl->tmem_base, 512);
  }
  if (ctl->failed == 0) Finish<kForm>(a, reinterpret_cast<AgainSmem*>(q_s), ctl);
}

int SmCount() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  return cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && sms > 0 ? sms : 148;
}

// Whether the kernel is the shorter one, by estimates of both in us.  This: a CTA takes a + b a step of 64 keys (of rows that are no
// multiple of 16 bytes, single stores: b + 2), and the grid its longest CTA or the SMs' share of all with most of a shortest one
// left over, a whole number of rounds where all are equally long.  The tile kernels of k_attention.cu: the pairs of their blocks, 64
// keys at a time (by features, of which statistics and sums are half), the blocks past one to two SMs, and no less than the
// longest block's walk.  Measured on a B200, tile kernels / this, us: statistics 8 x 512 positions of 12 heads of 64 174 /
// 72.7, 32 x 128 of 4 29.0 / 15.4, 2 x 1030 of 3 71.6 / 63.3, 8 x 100 of 4 10.9 / 14.1, 64 x 32 of 4 15.7 / 19.6, 12 x 129 of 8 28.8 / 29.4;
// probabilities 184 / 117, 29.9 / 21.8, 72.3 / 126, 11.1 / 19.0, 16.0 / 24.7, 29.6 / 47.5; raw scores 87.7 / 59.0, 16.2 / 12.2, 34.5 / 63.9, 5.9 /
// 10.2, 10.7 / 15.8, 18.4 / 26.9.  Of 84 launches measured (1 x 300 to 128 x 64 positions, heads of 4 to 64) the rule takes the longer way in
// two: probabilities of 24 x 127 of 4 heads 26.3 / 25.0, raw scores of 10 x 321 of 10 heads of 60 55.0 / 53.0.
bool Shorter(Form form, size_t B, size_t S, size_t H, size_t d) {
  const int rows = 8 * AttnTileRows(B * H, S, d, form != Form::kScores);
  if (rows == 0) return true;   // (not even that: a warp a row)
  const double sms = SmCount(), units = static_cast<double>(B * H);
  const double tiles = static_cast<double>((S + kRows - 1) / kRows), chunks = static_cast<double>((S + kKeys - 1) / kKeys);
  const double a = form == Form::kScores ? 6.4 : 7.3;
  const double b = (form == Form::kTiled ? 3.4 : form == Form::kCached ? 5.9 : 2.2) + (form != Form::kTiled && S % 4 != 0 ? 2.0 : 0.0);
  double mine = a + b * chunks;
  if (tiles == 1.0) {
    mine *= std::ceil(units / sms);
  } else {
    const double steps = tiles * (tiles + 1) - (2 * tiles - chunks);   // of a unit
    mine = std::max(mine, units * (a * tiles + b * steps) / sms + (units * tiles > sms ? 0.6 * (a + 2 * b) : 0.0));
  }
  const double theirs_tiles = static_cast<double>((S + rows - 1) / rows), blocks = units * theirs_tiles, per = static_cast<double>(kKeys) / rows;
  const double keys = kKeys * (per * chunks * (chunks + 1) / 2 - (per * chunks - theirs_tiles) * chunks);   // of a unit's blocks
  const double wide = static_cast<double>(d) / 64.0, half = 0.5 + 0.5 * wide, few = rows == 8 ? 1.7 : 1.0;
  const double pairs = units * keys * rows * 1e-6 * 148.0 / sms, more = std::max(0.0, blocks - sms / 2) * 148.0 / sms;
  const double theirs = form == Form::kScores ? 5.0 + std::max(1.4 * chunks, 4.7 * wide * pairs + 0.011 * more)
                                              : 4.0 + std::max(4.1 * half * few * chunks, 9.3 * half * few * pairs + 0.022 * more);
  return mine < 0.96 * theirs;
}

template <Form kForm>
bool Launch(const SliceArgs& a, size_t blocks, cudaStream_t s) {
  static std::atomic<bool> configured[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(AttnSliceKernel<kForm>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSliceSmem)) != cudaSuccess)
      return false;
    if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
  }
  return Next(AttnSliceKernel<kForm>, static_cast<unsigned>(blocks), kThreads, kSliceSmem, s)(a) == cudaSuccess;
}

bool Fits(std::initializer_list<const void*> ps, size_t B, size_t S, size_t H, size_t d) {
  if (d % 4 != 0 || d == 0 || d > kWidth || S == 0 || B * H == 0) return false;
  if (B * H > 0x7FFFFFFF / ((S + kRows - 1) / kRows) || S > 0x7FFFFF) return false;
  for (const void* p : ps)
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;
  return true;
}

}  // namespace

bool AttnFwdSlices(const float* q, const float* k, const float* v, float* o, float* probs, float* stats, size_t B, size_t S,
                   size_t H, size_t d, SliceUse use, DeviceStatus* status, cudaStream_t s) {
  if (use == SliceUse::kNever || !Fits({q, k, v, o, stats}, B, S, H, d)) return false;
  if (use == SliceUse::kShorter && !Shorter(probs ? Form::kCached : Form::kTiled, B, S, H, d)) return false;
  const SliceArgs a{q, k, v, o, probs, stats, static_cast<uint32_t>(B * H), static_cast<uint32_t>(S), static_cast<uint32_t>(H),
                    static_cast<uint32_t>(d), 1.0f / sqrtf(static_cast<float>(d)),
                    S % 4 == 0 && (reinterpret_cast<uintptr_t>(probs) & 15) == 0, status};
  const size_t blocks = B * H * ((S + kRows - 1) / kRows);
  return probs ? Launch<Form::kCached>(a, blocks, s) : Launch<Form::kTiled>(a, blocks, s);
}

bool AttnDPSlices(const float* dout, const float* v, float* dp, size_t B, size_t S, size_t H, size_t d, SliceUse use,
                  DeviceStatus* status, cudaStream_t s) {
  if (use == SliceUse::kNever || !Fits({dout, v}, B, S, H, d)) return false;
  if (use == SliceUse::kShorter && !Shorter(Form::kScores, B, S, H, d)) return false;
  const SliceArgs a{dout, v, nullptr, nullptr, dp, nullptr, static_cast<uint32_t>(B * H), static_cast<uint32_t>(S),
                    static_cast<uint32_t>(H), static_cast<uint32_t>(d), 1.0f,
                    S % 4 == 0 && (reinterpret_cast<uintptr_t>(dp) & 15) == 0, status};
  return Launch<Form::kScores>(a, B * H * ((S + kRows - 1) / kRows), s);
}

}  // namespace see::k
