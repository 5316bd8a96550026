// Row-wise softmax over the last dim, optionally masked by a [start, end) key
// range per row and a window around the diagonal: the probabilities of the
// matmul-attention path that callers keep beside the fused 'attn' op
// (packages/runntime/src/core/graph/ops/reduce.ts:12-39; kernel
// packages/runntime/src/core/kernels/reduce/softmax.ts:111-186).
//
// HBM-bound: one read of the kept scores and one write of the row.  A row is handled by one
// warp (eight rows per CTA) or by one CTA.  Memory is touched in
// 16-byte chunks at 16-byte addresses wherever the row starts: a row of an odd width begins in
// the middle of a chunk, and only its first and last chunk go element by element.  The zeros
// outside the kept range need no statistics, so they are stored while the first chunk of scores
// is on its way; then a running (max, sum) per thread, and a second look at the kept scores
// (L1/L2 by then) writes exp(x - max) / sum.
//
// Measured, f16 [6007, 6007] with 24 segments (75 MB, 11 us at the copy rate): 55.3 us with
// odd rows element by element, 20.5 us in chunks.
#include "common.cuh"

namespace rt {
namespace {

constexpr int kThreads = 256;
constexpr int kAhead = 4;
// One warp per row for narrow rows, and wherever there are rows enough to fill the chip with
// warps: no block-wide reduction, and the idle lanes of a narrow kept range cost one warp
// instead of eight (f16 [6007, 6007], 24 segments: 28.7 us with a CTA per row,
// 20.5 with a warp).
constexpr int kWarpRowCols = 2048, kWarpRows = 2048;
constexpr float kNegMax = -3.402823466e38f;

// N elements that are read and written together.
template <typename T, int N>
struct alignas(N * sizeof(T)) Chunk {
  T e[N];
};

__device__ __forceinline__ void combine(float& m, float& s, float m2, float s2) {
  const float mNew = fmaxf(m, m2);
  s = s * __expf(m - mNew) + s2 * __expf(m2 - mNew);
  m = mNew;
}

// WARP: one warp per row, else one CTA per row.  V: elements per chunk.
template <typename T, bool WARP, int V>
__global__ void __launch_bounds__(kThreads)
softmax_kernel(const T* __restrict__ x, T* __restrict__ out, const float* __restrict__ segs,
               int64_t rows, int64_t cols, int64_t wl, int64_t wr) {
  using C = Chunk<T, V>;
  // chunk and column numbers: the launcher takes V > 1 only for rows shorter than 2^31
  using I = std::conditional_t<V == 1, int64_t, int>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row = WARP ? (int64_t)blockIdx.x * (kThreads / 32) + warp : (int64_t)blockIdx.x;
  if (row >= rows) return;  // uniform per warp (WARP) or per CTA
  const int t = WARP ? lane : threadIdx.x;
  const int span = WARP ? 32 : kThreads;

  // Kept columns [lo, hi).
  int64_t lo64 = 0, hi64 = cols;
  if (segs) {
    const int64_t s0 = (int64_t)segs[2 * row], s1 = (int64_t)segs[2 * row + 1];
    lo64 = max(s0, row - min(row, wl));
    hi64 = min(s1, row + min(cols - row, wr + 1));
  }

  // The row begins `mis` elements into its first chunk (the same for x and out: see the
  // launcher), so column j is element (j + mis) % V of chunk (j + mis) / V.
  const T* xr = x + row * cols;
  T* orow = out + row * cols;
  const int mis = V == 1 ? 0 : (int)((reinterpret_cast<uintptr_t>(xr) % (V * sizeof(T))) / sizeof(T));
  const C* xc = reinterpret_cast<const C*>(xr - mis);
  C* oc = reinterpret_cast<C*>(orow - mis);
  const bool any = hi64 > lo64;
  const I lo = any ? (I)lo64 + mis : 0, hi = any ? (I)hi64 + mis : 0, end = (I)cols + mis;
  const I nc = (end + V - 1) / V;
  const I q0 = lo / V, q1 = (hi + V - 1) / V;  // chunks that touch the kept range
  // Chunks [w0, w1) lie wholly in the row; at most one on either side does not.
  const I w0 = mis ? 1 : 0, w1 = end / V;
  auto load = [&](I c) {
    C v;
    if (V == 1 || (c >= w0 && c < w1)) {
      v = xc[c];
    } else {
#pragma unroll
      for (int e = 0; e < V; e++) v.e[e] = (c * V + e >= mis && c * V + e < end) ? xc[c].e[e] : from_f32<T>(0.f);
    }
    return v;
  };
  auto store = [&](I c, const C& v) {
    if (V == 1 || (c >= w0 && c < w1)) {
      oc[c] = v;
    } else {
#pragma unroll
      for (int e = 0; e < V; e++)
        if (c * V + e >= mis && c * V + e < end) oc[c].e[e] = v.e[e];
    }
  };

  // Kept chunks are taken kAhead at a time, so that as many loads are in flight per thread.
  C ahead[kAhead];
  auto loadAhead = [&](I c) {
#pragma unroll
    for (int u = 0; u < kAhead; u++)
      if (c + u * span < q1) ahead[u] = load(c + u * span);
  };
  loadAhead(q0 + t);
  {
    C zero;
#pragma unroll
    for (int e = 0; e < V; e++) zero.e[e] = from_f32<T>(0.f);
    const I left = min(q0, w1), right = max(q1, w0);
#pragma unroll 4
    for (I c = w0 + t; c < left; c += span) oc[c] = zero;
#pragma unroll 4
    for (I c = right + t; c < w1; c += span) oc[c] = zero;
    if (V > 1 && t < 2) {   // the row's ragged chunks, where no kept column is in them
      const I c = t == 0 ? 0 : nc - 1;
      if ((c < w0 || c >= w1) && (c < q0 || c >= q1)) store(c, zero);
    }
  }

  float m = kNegMax, s = 0.f;
  for (I c = q0 + t; c < q1; c += kAhead * span) {
    if (c != q0 + t) loadAhead(c);
#pragma unroll
    for (int u = 0; u < kAhead; u++) {
      const I at = (c + u * span) * V;
      if (c + u * span >= q1) break;
      float f[V];
      float mNew = m;
      const bool inner = at >= lo && at + V <= hi;
#pragma unroll
      for (int e = 0; e < V; e++) {
        f[e] = to_f32<T>(ahead[u].e[e]);
        if (inner || (at + e >= lo && at + e < hi)) mNew = fmaxf(mNew, f[e]);
      }
      // one rescale of the running sum per chunk
      float add = 0.f;
#pragma unroll
      for (int e = 0; e < V; e++) {
        const float pe = __expf(f[e] - mNew);
        add += (inner || (at + e >= lo && at + e < hi)) ? pe : 0.f;
      }
      s = s * __expf(m - mNew) + add;
      m = mNew;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    combine(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
  if (!WARP) {
    __shared__ float sM[kThreads / 32], sS[kThreads / 32];
    if (lane == 0) sM[warp] = m, sS[warp] = s;
    __syncthreads();
    m = sM[0], s = sS[0];
#pragma unroll
    for (int w = 1; w < kThreads / 32; w++) combine(m, s, sM[w], sS[w]);
  }
  const float inv = s > 0.f ? 1.f / s : 0.f;

  for (I c = q0 + t; c < q1; c += kAhead * span) {
    if (q1 - q0 > kAhead * span) loadAhead(c);   // else the chunks are still in their registers
#pragma unroll
    for (int u = 0; u < kAhead; u++) {
      const I at = (c + u * span) * V;
      if (c + u * span >= q1) break;
      C v = ahead[u];
      const bool inner = at >= lo && at + V <= hi;
#pragma unroll
      for (int e = 0; e < V; e++) {
        const bool kept = inner || (at + e >= lo && at + e < hi);
        v.e[e] = from_f32<T>(kept ? __expf(to_f32<T>(v.e[e]) - m) * inv : 0.f);
      }
      store(c + u * span, v);
    }
  }
}

template <typename T, int V>
cudaError_t softmax_chunked(const T* x, T* out, const float* segs, int64_t rows, int64_t cols,
                            int64_t wl, int64_t wr, cudaStream_t s) {
  const bool warpRows = cols <= kWarpRowCols || rows >= kWarpRows;
  const int64_t blocks = warpRows ? (rows + kThreads / 32 - 1) / (kThreads / 32) : rows;
  if (blocks > 0x7fffffffll) return cudaErrorInvalidValue;
  const unsigned g = (unsigned)blocks;
  if (warpRows) softmax_kernel<T, true, V><<<g, kThreads, 0, s>>>(x, out, segs, rows, cols, wl, wr);
  else softmax_kernel<T, false, V><<<g, kThreads, 0, s>>>(x, out, segs, rows, cols, wl, wr);
  return cudaGetLastError();
}

// The widest chunk at whose boundaries x and out agree: 16 bytes unless a caller's own memory
// puts them at different offsets from one.
template <typename T>
cudaError_t softmax_typed(const void* x, void* out, const float* segs, int64_t rows, int64_t cols,
                          int64_t wl, int64_t wr, cudaStream_t s) {
  auto* xi = static_cast<const T*>(x);
  auto* oi = static_cast<T*>(out);
  const uintptr_t apart = reinterpret_cast<uintptr_t>(x) ^ reinterpret_cast<uintptr_t>(out);
  const bool shortRows = cols < (1ll << 31) - 4096;
  if (shortRows && apart % 16 == 0) return softmax_chunked<T, 16 / sizeof(T)>(xi, oi, segs, rows, cols, wl, wr, s);
  if (shortRows && apart % 8 == 0) return softmax_chunked<T, 8 / sizeof(T)>(xi, oi, segs, rows, cols, wl, wr, s);
  return softmax_chunked<T, 1>(xi, oi, segs, rows, cols, wl, wr, s);
}

}  // namespace

cudaError_t launch_softmax(const void* x, void* out, const float* segs, int64_t rows, int64_t cols,
                           int64_t wl, int64_t wr, int dtype, cudaStream_t s) {
  return dtype == RT_F16 ? softmax_typed<__half>(x, out, segs, rows, cols, wl, wr, s)
                         : softmax_typed<float>(x, out, segs, rows, cols, wl, wr, s);
}

}  // namespace rt
