// Exact causal attention on the tensor cores, where the bits are not observed: scores as accurate as dots in double, sums
// of probabilities times values as accurate as f32 multiply-adds.
//
// Scores.  A row of Q (or K) is a fixed-point number per element: scaled by a power of two to (-128, 128) and cut into four
// signed digits of eight bits, each a whole number up to 128 and so a bf16 value exactly:
//     x = 2^(e - 7) (s0 + s1 / 2^8 + s2 / 2^16 + s3 / 2^24) + r,  |r| <= 2^(e - 32),  2^e > max |x|.
// Products of digits are whole numbers up to 2^14, and a sum of up to 4 x 64 of them is one below 2^24: the tensor core's
// f32 accumulator holds it exactly, in whatever order and rounding it adds.  The thirteen products of digits with i + j <= 4 meet in
// five accumulators, one for each i + j, which four multiply-adds put together.  What is left out (i + j > 4, r) is
// 2^-32 of 2^(eq + ek) in the middle, a fiftieth of the rounding to f32 that a dot in double ends with too.
// (Fixed-point slices: Ozaki, Ogita, Oishi, Rump, "Error-free transformations of matrix multiplication by using fast
// routines of matrix multiplication", 2012.)  The digits of K lie one under the other, so digit i of Q times all of K's
// digits that count is one product of width 64 (4 - i): the accumulators stand side by side, each i starts one further on.
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
// A row whose elements are not finite, or beyond 2^60 or all below 2^-60, has no such digits: its CTA then makes its rows
// again with dots in double, one warp a row.
//
// Every wait on an mbarrier is bounded; one that runs out raises DeviceStatus::wait_timeout and the CTA stores nothing.
#include <algorithm>
#include <cmath>
#include <initializer_list>

#include "kernels.h"
#include "launch.cuh"
#include "umma_device.cuh"

namespace see::k {

namespace {

using namespace umma_dev;

constexpr uint32_t kRows = 128, kKeys = 64, kWidth = 64;   // queries of a CTA, keys of a step, widest head
constexpr uint32_t kWorkWarps = 8, kCutWarps = 4, kThreads = 32 * (kWorkWarps + kCutWarps + 1);
constexpr uint32_t kQSlice = kRows * 128, kKSlice = kKeys * 128, kPPiece = kRows * 128, kVPiece = kKeys * 128;
constexpr uint32_t kStageBytes = 3 * kPPiece + 3 * kVPiece;   // K's four digits, then P's three pieces; V's pieces behind
static_assert(4 * kKSlice <= 3 * kPPiece, "K's digits lie where P's pieces come");
constexpr uint32_t kParts = kWorkWarps / 4, kOwn = kKeys / kParts;   // threads to a row; keys (and features) of each
constexpr uint32_t kScoreCols = 5 * kKeys;                    // tensor memory: five accumulators of scores, three of sums
constexpr float kSlack = 8.0f;                                // how far a row's maximum may exceed its reference

enum class Form { kTiled, kCached, kScores };   // statistics; probabilities and statistics; raw scores (dP = dO V^T)

struct __align__(16) SliceCtl {
  float q_scale[kRows], k_scale[4][kKeys];   // (a step's is read after its stage may have gone on: four in turns)
  float row_max[2][kParts][kRows];           // by parity of the step
  double denom[kParts][kRows];
  uint64_t k_full[2], v_full[2], stage_empty[2], s_full, s_empty, p_full, sum_full;
  uint32_t tmem_base;
  volatile uint32_t failed;
  volatile uint32_t odd;                     // some row has no digits
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
// The digits of a row that four neighbouring lanes hold; the factor that undoes their scale.  *odd: it has none.
__device__ __forceinline__ float CutDigits(float (&x)[16], uint8_t* dst, uint32_t slice_bytes, uint32_t row, uint32_t c0, bool* odd) {
  uint32_t top = 0;   // the largest magnitude's bits (a NaN's are larger than any number's)
#pragma unroll
  for (int e = 0; e < 16; ++e) top = max(top, __float_as_uint(x[e]) & 0x7FFFFFFFu);
  top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, 1));
  top = max(top, __shfl_xor_sync(0xFFFFFFFFu, top, 2));
  const bool none = top >= 0x5D800000u || (top != 0 && top < 0x21800000u);   // 2^60, 2^-60
  *odd = *odd || none;
  const uint32_t ex = top >> 23;
  const float to = none ? 0.0f : (top == 0 ? 1.0f : __uint_as_float((260u - ex) << 23));      // 2^(7 - e)
  const float back = none || top == 0 ? 1.0f : __uint_as_float((ex - 6u) << 23);             // 2^(e - 7)
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

// One row as the tile kernels' expressions have it, by a warp, three times over the keys and without memory for scores.
template <Form kForm>
__device__ __noinline__ void RowAgain(const SliceArgs& a, uint32_t bh, uint32_t i) {
  const uint32_t lane = threadIdx.x & 31, b = bh / a.H, h = bh % a.H;
  const size_t D = static_cast<size_t>(a.H) * a.d, base = static_cast<size_t>(b) * a.S * D + static_cast<size_t>(h) * a.d;
  const float* q = a.q + base + i * D;
  auto dot = [&](uint32_t j) {
    const float* k = a.k + base + j * D;
    double sum = 0.0;
    for (uint32_t c = 0; c < a.d; ++c) sum += static_cast<double>(q[c]) * static_cast<double>(k[c]);
    return static_cast<float>(sum);
  };
  auto score = [&](uint32_t j) { return __fmul_rn(dot(j), a.inv_sqrt_d); };   // (no fused difference behind it: a maximum's is 0)
  const size_t unit = static_cast<size_t>(bh) * a.S + i;
  if constexpr (kForm == Form::kScores) {
    for (uint32_t j = lane; j < a.S; j += 32) a.probs[unit * a.S + j] = j <= i ? dot(j) : 0.0f;
  } else {
    float top = -INFINITY;
    for (uint32_t j = lane; j <= i; j += 32) top = fmaxf(top, score(j));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
    double denom = 0.0;
    for (uint32_t j = lane; j <= i; j += 32) denom += static_cast<double>(expf(score(j) - top));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) denom += __shfl_xor_sync(0xFFFFFFFFu, denom, o);
    const float inv = 1.0f / static_cast<float>(denom);
    float acc[2] = {0.0f, 0.0f};
    for (uint32_t j0 = 0; j0 < a.S; j0 += 32) {
      const uint32_t j = j0 + lane;
      const float p = j <= i ? expf(score(j) - top) * inv : 0.0f;
      if (kForm == Form::kCached && j < a.S) a.probs[unit * a.S + j] = p;
      for (uint32_t l = 0; l < 32 && j0 + l <= i; ++l) {
        const float w = __shfl_sync(0xFFFFFFFFu, p, l);
        const float* v = a.v + base + static_cast<size_t>(j0 + l) * D;
        if (lane < a.d) acc[0] = fmaf(w, v[lane], acc[0]);
        if (lane + 32 < a.d) acc[1] = fmaf(w, v[lane + 32], acc[1]);
      }
    }
    float* o = a.o + base + i * D;
    if (lane < a.d) o[lane] = acc[0];
    if (lane + 32 < a.d) o[lane + 32] = acc[1];
    if (a.stats && lane == 0)
      *reinterpret_cast<float4*>(a.stats + unit * kAttnStatsWidth) = make_float4(top, inv, 0.0f, 0.0f);
  }
}

template <Form kForm>
__global__ void __launch_bounds__(kThreads, 1) AttnSliceKernel(const SliceArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* q_s = smem_raw + ((1024u - (SmemAddr(smem_raw) & 1023u)) & 1023u);
  uint8_t* ring = q_s + 4 * kQSlice;
  SliceCtl* ctl = reinterpret_cast<SliceCtl*>(ring + 2 * kStageBytes);

  const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // Longest tiles first over the whole grid, so that the last wave is short ones.
  const uint32_t tiles = (a.S + kRows - 1) / kRows, tile = tiles - 1 - blockIdx.x / a.BH, bh = blockIdx.x % a.BH;
  const uint32_t i0 = tile * kRows, keys = min(i0 + kRows, a.S);
  const uint32_t n = (keys + kKeys - 1) / kKeys;                                  // steps of a walk
  const uint32_t ahead = kForm == Form::kTiled ? 0 : n;                           // steps that only take scores
  const uint32_t total = kForm == Form::kCached ? 2 * n : n;
  const size_t D = static_cast<size_t>(a.H) * a.d;
  const size_t base = static_cast<size_t>(bh / a.H) * a.S * D + static_cast<size_t>(bh % a.H) * a.d;

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
    ctl->odd = 0;
    MbarInitFence();
  }
  if (warp == kWorkWarps + kCutWarps) TmemAlloc(&ctl->tmem_base, 512);
  TcFenceBefore();
  __syncthreads();
  TcFenceAfter();
  AwaitPrevious();
  constexpr uint32_t tmem = 0;   // all 512 columns are this CTA's

  if (warp < kWorkWarps + kCutWarps) {   // the queries' digits
    bool odd = false;
    for (uint32_t t = threadIdx.x; t < 4 * kRows; t += 32 * (kWorkWarps + kCutWarps)) {   // (whole warps)
      const uint32_t r = t >> 2, c0 = (t & 3) * 16;
      float x[16];
      FetchSixteen(x, a.q + base + static_cast<size_t>(i0 + r) * D, i0 + r < a.S, c0, a.d);
      const float back = CutDigits(x, q_s, kQSlice, r, c0, &odd);
      if (c0 == 0) ctl->q_scale[r] = back * (kForm == Form::kScores ? 1.0f : a.inv_sqrt_d);
    }
    if (odd) ctl->odd = 1;
    FenceProxyAsync();
  }
  __syncthreads();

  bool ok = true;
  if (warp == kWorkWarps + kCutWarps) {
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
    const uint32_t t = threadIdx.x - 32 * kWorkWarps, r0 = t >> 2, c0 = (t & 3) * 16;
    constexpr uint32_t kEach = kKeys / (8 * kCutWarps);   // keys of a thread, 8 kCutWarps apart
    bool odd = false;
    float x[kEach][16], y[kEach][16];   // a step's elements, on their way since the step before
    auto row_of = [&](uint32_t h) { return r0 + h * 8 * kCutWarps; };
    auto sums_at = [&](uint32_t u) { return kForm == Form::kTiled || (kForm == Form::kCached && u >= ahead && u < total); };
    auto fetch = [&](float (&f)[kEach][16], const float* src, uint32_t u) {
#pragma unroll
      for (uint32_t h = 0; h < kEach; ++h) {
        const uint32_t key = (u < n ? u : u - n) * kKeys + row_of(h);
        FetchSixteen(f[h], src + base + static_cast<size_t>(key) * D, u < total && key < a.S, c0, a.d);
      }
    };
    fetch(x, a.k, 0);
    if (sums_at(0)) fetch(y, a.v, 0);
    for (uint32_t u = 0; u < total && ok; ++u) {
      const uint32_t s = u & 1;
      uint8_t* stage = ring + s * kStageBytes;
      if (u >= 2) ok = SliceWait(ctl, &ctl->stage_empty[s], ((u >> 1) - 1) & 1);
      if (!ok) break;
#pragma unroll
      for (uint32_t h = 0; h < kEach; ++h) {
        const float back = CutDigits(x[h], stage, kKSlice, row_of(h), c0, &odd);
        if (c0 == 0) ctl->k_scale[u & 3][row_of(h)] = back;
      }
      if (odd) ctl->odd = 1;
      FenceProxyAsync();
      __syncwarp();
      if (lane == 0) MbarArrive(&ctl->k_full[s]);
      fetch(x, a.k, u + 1);
      if (sums_at(u)) {   // V's pieces while the scores are formed
#pragma unroll
        for (uint32_t h = 0; h < kEach; ++h) {
          uint32_t w[3][8];
#pragma unroll
          for (int e = 0; e < 16; e += 2) {
            odd = odd || !(fabsf(y[h][e]) < 1e36f) || !(fabsf(y[h][e + 1]) < 1e36f);
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
        if (odd) ctl->odd = 1;
        FenceProxyAsync();
        __syncwarp();
      }
      if (lane == 0) MbarArrive(&ctl->v_full[s]);   // (every step: its phases are the stage's)
      if (sums_at(u + 1)) fetch(y, a.v, u + 1);
    }
  } else {
    // ---- scores, probabilities, sums: thread (row, part of the keys) ----
    const uint32_t quarter = warp & 3, part = warp >> 2, r = quarter * 32 + lane, i = i0 + r;
    const uint32_t t_s = tmem + ((quarter * 32) << 16) + part * kOwn, t_o = t_s + kScoreCols;
    const float q_scale = ctl->q_scale[r];
    const size_t unit = static_cast<size_t>(bh) * a.S + i;
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
      denom += d0 + d1;
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
          float* to = a.probs + (static_cast<size_t>(bh) * a.S + row) * a.S + j;
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
    auto put_stats = [&](double whole) {   // relative to the maximum: the rows' statistics, and their factor
      inv = 1.0f / static_cast<float>(whole * exp(static_cast<double>(ref) - static_cast<double>(top)));
      if (a.stats && part == 0 && i < a.S && ok && ctl->odd == 0)
        *reinterpret_cast<float4*>(a.stats + unit * kAttnStatsWidth) = make_float4(top, inv, 0.0f, 0.0f);
    };

    if constexpr (kForm == Form::kScores) {
      for (uint32_t u = 0; u < n; ++u) {
        const uint32_t key0 = take_scores(u);
        if (ok) store_scores(u, key0);
      }
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
      if (ok && ctl->odd == 0 && 4 * chunk < a.d)
        for (uint32_t row = threadIdx.x >> 4; row < kRows && i0 + row < a.S; row += 2 * kWorkWarps)
          *reinterpret_cast<float4*>(a.o + base + static_cast<size_t>(i0 + row) * D + 4 * chunk) =
              *reinterpret_cast<const float4*>(tile_o + row * kWidth + ((chunk ^ (row & 15)) * 4));
    }
    if constexpr (kForm != Form::kTiled) {   // the keys no walk reaches
      for (uint32_t row = warp; ok && row < kRows && i0 + row < a.S; row += kWorkWarps) {
        float* to = a.probs + (static_cast<size_t>(bh) * a.S + i0 + row) * a.S;
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
  if (ctl->odd != 0 && ctl->failed == 0)
    for (uint32_t row = warp; row < kRows && i0 + row < a.S; row += kThreads / 32) RowAgain<kForm>(a, bh, i0 + row);
}

// Whether the kernel is the shorter one, by estimates of both in us: 64 keys a step, the longest tile's steps or an SM's share
// of them all; and the tile kernels of k_attention.cu by the pairs they take, whatever their rows (of the raw scores, by their
// features too).  Measured on a B200, tile kernels / this, us: statistics 8 x 512 positions of 12 heads of 64 176 / 69.7, 32 x 128 of 4 30.9 /
// 15.1, 2 x 1030 of 3 72.9 / 61.6, 8 x 100 of 4 12.4 / 13.3, 64 x 32 of 4 17.5 / 20.2; probabilities 186 / 114, 31.0 / 19.8, 73.9 / 133, 12.5 / 17.6;
// raw scores 90.3 / 56.0, 18.6 / 11.2, 36.0 / 64.8, 8.4 / 9.3.
bool Shorter(Form form, size_t B, size_t S, size_t H, size_t d) {
  const double tiles = static_cast<double>((S + kRows - 1) / kRows), units = static_cast<double>(B * H);
  const double longest = static_cast<double>((S + kKeys - 1) / kKeys), steps = units * (tiles * (tiles + 1) - (2 * tiles - longest));
  const double rounds = std::max(1.0, units * tiles / 148.0);
  const double step = form == Form::kCached ? 7.0 : 3.3, mine = 6.0 + step * std::max(longest, steps / 148.0) + 5.0 * (rounds - 1.0);
  double pairs = units * static_cast<double>(S) * static_cast<double>(S + 1) * 0.5e-6;
  if (form == Form::kScores) pairs *= static_cast<double>(d) / 64.0;
  const double first = std::min(pairs, 1.0), more = pairs - first;
  const double theirs = form == Form::kScores ? 6.0 + 11.0 * first + 6.0 * more : 7.0 + 21.0 * first + 13.5 * more;
  return mine < theirs;
}

template <Form kForm>
bool Launch(const SliceArgs& a, size_t blocks, cudaStream_t s) {
  if (cudaFuncSetAttribute(AttnSliceKernel<kForm>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSliceSmem)) != cudaSuccess)
    return false;
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
