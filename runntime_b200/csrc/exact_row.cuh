// One row of prefill attention key by key, by one warp.  The prefill kernels that work on tiles
// multiply a masked key's value by a probability of zero, and the f32 tensor-core kernel adds up parts
// of its operands: with an infinity or a NaN among them either gives NaN where the op's definition
// does not.  A tile whose output is not finite is computed again with this.
#pragma once

#include "common.cuh"

namespace rt {
namespace {

// Keys [lo, end] of query row `row`, head h; head sizes up to 512.
template <typename T>
__device__ __noinline__ void exact_row(const AttnParams& p, int64_t row, int h, int64_t lo, int64_t end) {
  constexpr int kCols = 16;   // per lane
  const int lane = threadIdx.x & 31, hd = p.hd;
  const int kvh = h / (p.qHeads / p.kvHeads);
  const T* q = static_cast<const T*>(p.q) + row * p.qStride + (int64_t)h * hd;
  const T* k = static_cast<const T*>(p.k) + (int64_t)kvh * hd;
  const T* v = static_cast<const T*>(p.v) + (int64_t)kvh * hd;
  float m = p.sinks ? p.sinks[h] * 0.6931471805599453f : kNegSeed, l = p.sinks ? 1.f : 0.f;
  float acc[kCols];
#pragma unroll
  for (int c = 0; c < kCols; c++) acc[c] = 0.f;
  for (int64_t j = lo; j <= end; j++) {
    float s = 0.f;
    for (int x = lane; x < hd; x += 32) s = fmaf(to_f32<T>(q[x]), to_f32<T>(k[j * p.kvStride + x]), s);
    s = warp_sum(s);
    if (p.hasKeyBias && j >= p.biasStart && j < p.biasEnd) s += p.biasValue;
    const float mNew = fmaxf(m, s), corr = __expf(m - mNew), pe = __expf(s - mNew);
    l = l * corr + pe;
    m = mNew;
#pragma unroll
    for (int c = 0; c < kCols; c++)
      if (lane + 32 * c < hd) acc[c] = fmaf(pe, to_f32<T>(v[j * p.kvStride + lane + 32 * c]), acc[c] * corr);
  }
  const float invL = l > 0.f ? 1.f / l : 0.f;
  T* out = static_cast<T*>(p.out) + (row * p.qHeads + h) * hd;
#pragma unroll
  for (int c = 0; c < kCols; c++)
    if (lane + 32 * c < hd) out[lane + 32 * c] = from_f32<T>(acc[c] * invL);
}

}  // namespace
}  // namespace rt
