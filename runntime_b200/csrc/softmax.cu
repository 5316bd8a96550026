// Row-wise softmax over the last dim, optionally masked by a [start, end) key
// range per row and a window around the diagonal: the probabilities of the
// matmul-attention path that callers keep beside the fused 'attn' op
// (packages/runntime/src/core/graph/ops/reduce.ts:12-39; kernel
// packages/runntime/src/core/kernels/reduce/softmax.ts:111-186).
//
// HBM-bound: one read of the kept scores and one write of the row.  A row is handled by one
// warp (narrow rows, eight per CTA), by one CTA, or with three others (softmax_group_kernel); the first pass keeps a running (max, sum) per
// thread, the second re-reads the row (it is in L1/L2 by then) and writes exp(x - max) / sum.
//
// Rows that start on four elements are taken four at a time.  Any other row begins in the middle of
// a 16-byte chunk: memory is still touched in 16-byte chunks at 16-byte addresses, only the row's
// first and last chunk go element by element, and the zeros outside the kept range, which need no
// statistics, are stored while the first scores are on their way.  Element by element, chunks, us: f16
// [6007, 6007] with 24 segments (75 MB, 11 us at the copy rate) 55.5, 20.8 (55.3, 24.6 through the
// operator; 17.2 with four rows to a CTA and as a dependent launch), with one 74.6, 71.9; f32
// 51.4, 31.0 with 24.  On aligned rows the quads are the faster ones: f16 [12288, 12288] with 2
// segments 119 against 141, [2500, 2500] with 3 12.4 against 18.7.
#include "common.cuh"

namespace rt {
namespace {

constexpr int kThreads = 256;
constexpr int kAhead = 2, kCtas = 5;
// One warp per row up to kWarpRowCols columns, one CTA beyond.  Of that CTA one warp alone takes a
// kept range of up to kWarpKept columns, without a block barrier, while all of them store the
// zeros (f16 [6007, 6007], 24 segments: 28.7 us with all warps on the kept range, 20.8).
constexpr int kWarpRowCols = 2048, kWarpKept = 1024;
// A warp's rows that start anywhere go element by element where they have no mask or are narrow: between
// the ragged ends there are too few chunks to pay for them, and an exponential per element costs
// less than the registers of eight.  f16, chunks and elements, us: [70000, 3] 39.2, 19.4, [20000, 515] 31.3, 17.3,
// [2047, 2047] without segments 13.4, 8.9; [515, 515] in 5 segments 3.9, 3.5, [1001, 1001] in 5 4.2, 4.4,
// [2047, 2047] in 5 6.2, 8.5.
constexpr int kElementCols = 768;
constexpr float kNegMax = -3.402823466e38f;

template <typename T>
struct Quad;
template <>
struct Quad<float> {
  using type = float4;
  static __device__ __forceinline__ void unpack(const float4& v, float (&f)[4]) {
    f[0] = v.x, f[1] = v.y, f[2] = v.z, f[3] = v.w;
  }
  static __device__ __forceinline__ float4 pack(const float (&f)[4]) {
    return make_float4(f[0], f[1], f[2], f[3]);
  }
};
template <>
struct Quad<__half> {
  using type = uint2;
  static __device__ __forceinline__ void unpack(const uint2& v, float (&f)[4]) {
    const __half2* h = reinterpret_cast<const __half2*>(&v);
    const float2 a = __half22float2(h[0]), b = __half22float2(h[1]);
    f[0] = a.x, f[1] = a.y, f[2] = b.x, f[3] = b.y;
  }
  static __device__ __forceinline__ uint2 pack(const float (&f)[4]) {
    uint2 v;
    __half2* h = reinterpret_cast<__half2*>(&v);
    h[0] = __floats2half2_rn(f[0], f[1]);
    h[1] = __floats2half2_rn(f[2], f[3]);
    return v;
  }
};

__device__ __forceinline__ void combine(float& m, float& s, float m2, float s2) {
  const float mNew = fmaxf(m, m2);
  s = s * __expf(m - mNew) + s2 * __expf(m2 - mNew);
  m = mNew;
}

// Rows that start on four elements: quads.  WARP: one warp per row, else one CTA per row.
template <typename T, bool WARP>
__global__ void __launch_bounds__(kThreads)
softmax_quad_kernel(const T* x, T* out, const float* segs, int64_t rows, int64_t cols, int64_t wl, int64_t wr) {
  grid_dependency_wait();
  using Q = Quad<T>;
  using QV = typename Q::type;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row = WARP ? (int64_t)blockIdx.x * (kThreads / 32) + warp : (int64_t)blockIdx.x;
  if (row >= rows) return;  // uniform per warp (WARP) or per CTA
  const int t = WARP ? lane : threadIdx.x;
  const int span = WARP ? 32 : kThreads;

  // Kept columns [lo, hi).
  int64_t lo = 0, hi = cols;
  if (segs) {
    const int64_t s0 = (int64_t)segs[2 * row], s1 = (int64_t)segs[2 * row + 1];
    lo = max(s0, row - min(row, wl));
    hi = min(s1, row + min(cols - row, wr + 1));
  }

  const T* xr = x + row * cols;
  T* orow = out + row * cols;
  float m = kNegMax, s = 0.f;
  // Quads of columns [q0, q1) touch the kept range; only the first and the last of them
  // can hold masked columns (32-bit column arithmetic: the launcher takes this path only for
  // rows shorter than 2^31).
  const int lo32 = (int)lo, hi32 = (int)hi;
  const int q0 = lo32 >> 2, q1 = hi32 > lo32 ? (hi32 + 3) >> 2 : q0;
  const QV* xq = reinterpret_cast<const QV*>(xr);
  {
    for (int i = q0 + t; i < q1; i += span) {
      float f[4];
      Q::unpack(xq[i], f);
      const int j = i * 4;
      const bool inner = j >= lo32 && j + 4 <= hi32;
      if (!inner) {
#pragma unroll
        for (int e = 0; e < 4; e++)
          if (j + e < lo32 || j + e >= hi32) f[e] = kNegMax;
      }
      // one running-sum rescale per quad instead of per element: five exponentials for four columns
      const float mNew = fmaxf(m, fmaxf(fmaxf(f[0], f[1]), fmaxf(f[2], f[3])));
      float add = 0.f;
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const float pe = __expf(f[e] - mNew);
        add += (inner || (j + e >= lo32 && j + e < hi32)) ? pe : 0.f;
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

  {
    QV* oq = reinterpret_cast<QV*>(orow);
    const int nq = (int)(cols >> 2);
    // zeros either side of the kept range: stores only
    const float z4[4] = {0.f, 0.f, 0.f, 0.f};
    const QV zero = Q::pack(z4);
#pragma unroll 4
    for (int i = t; i < q0; i += span) oq[i] = zero;
#pragma unroll 4
    for (int i = q1 + t; i < nq; i += span) oq[i] = zero;
    for (int i = q0 + t; i < q1; i += span) {
      float f[4];
      Q::unpack(xq[i], f);
      const int j = i * 4;
      if (j >= lo32 && j + 4 <= hi32) {
#pragma unroll
        for (int e = 0; e < 4; e++) f[e] = __expf(f[e] - m) * inv;
      } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
          f[e] = (j + e >= lo32 && j + e < hi32) ? __expf(f[e] - m) * inv : 0.f;
      }
      oq[i] = Q::pack(f);
    }
  }
}

// N elements that are read and written together.
template <typename T, int N>
struct alignas(N * sizeof(T)) Chunk {
  T e[N];
};

// Who works on a row: a warp; all warps of a CTA; or one warp on the kept columns while all warps
// store the zeros.
enum class By { Warp, Cta, WarpInCta };

// Kept columns [lo, hi) of a row.
__device__ __forceinline__ void kept_range(const float* segs, int64_t row, int64_t cols, int64_t wl, int64_t wr,
                                           int64_t& lo, int64_t& hi) {
  lo = 0, hi = cols;
  if (segs) {
    const int64_t s0 = (int64_t)segs[2 * row], s1 = (int64_t)segs[2 * row + 1];
    lo = max(s0, row - min(row, wl));
    hi = min(s1, row + min(cols - row, wr + 1));
  }
}

// One row.  V: elements per chunk.
template <typename T, By BY, int V, int TH = kThreads>   // TH: threads of the CTA
__device__ __forceinline__ void softmax_row(const T* __restrict__ x, T* __restrict__ out, int64_t row, int64_t cols,
                                            int64_t lo64, int64_t hi64, float* sM, float* sS) {
  using C = Chunk<T, V>;
  // chunk and column numbers: the launcher takes V > 1 only for rows shorter than 2^31
  using I = std::conditional_t<V == 1, int64_t, int>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = BY == By::Cta ? threadIdx.x : lane;      // for the kept columns
  const int span = BY == By::Cta ? TH : 32;
  const int zt = BY == By::Warp ? lane : threadIdx.x;    // for the zeros
  const int zspan = BY == By::Warp ? 32 : TH;
  const bool keeps = BY != By::WarpInCta || warp == 0;

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
  if (keeps) loadAhead(q0 + t);
  {
    C zero;
#pragma unroll
    for (int e = 0; e < V; e++) zero.e[e] = from_f32<T>(0.f);
    const I left = min(q0, w1), right = max(q1, w0);
#pragma unroll 4
    for (I c = w0 + zt; c < left; c += zspan) oc[c] = zero;
#pragma unroll 4
    for (I c = right + zt; c < w1; c += zspan) oc[c] = zero;
    if (V > 1 && zt < 2) {   // the row's ragged chunks, where no kept column is in them
      const I c = zt == 0 ? 0 : nc - 1;
      if ((c < w0 || c >= w1) && (c < q0 || c >= q1)) store(c, zero);
    }
  }

  if (!keeps) return;

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
  // one exponential per thread and one per warp: the maxima first, then the sums brought to them
  const float top = warp_max(m);
  s = warp_sum(s * __expf(m - top));
  m = top;
  if (BY == By::Cta) {
    constexpr int kWarps = TH / 32;
    if (lane == 0) sM[warp] = m, sS[warp] = s;
    __syncthreads();
    const float mw = sM[lane % kWarps];
    m = mw;
#pragma unroll
    for (int o = kWarps / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    s = sS[lane % kWarps] * __expf(mw - m);
#pragma unroll
    for (int o = kWarps / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
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
__global__ void __launch_bounds__(kThreads, kCtas)
softmax_cta_kernel(const T* x, T* out, const float* segs, int64_t cols,
                   int64_t wl, int64_t wr) {
  grid_dependency_wait();
  __shared__ float sM[kThreads / 32], sS[kThreads / 32];
  int64_t lo, hi;
  kept_range(segs, blockIdx.x, cols, wl, wr, lo, hi);
  if (hi - lo <= kWarpKept) softmax_row<T, By::WarpInCta, V>(x, out, blockIdx.x, cols, lo, hi, nullptr, nullptr);
  else softmax_row<T, By::Cta, V>(x, out, blockIdx.x, cols, lo, hi, sM, sS);
}

// Long half-precision rows that start anywhere, four to a CTA: where all four keep few columns each
// warp takes a row of its own, else the CTA takes them in turn.  A CTA per row spends a narrow row's time
// waiting for one warp's scores, statistics and stores in turn (20.6 us for 11.5 at the copy
// rate); four at once overlap them.  The last quarter of the rows go one to a CTA, so that a launch whose
// rows are wide does not end on a few CTAs with four of them (n columns, segments, us, a CTA per
// row and this: 6007, 24 22.4, 18.5; 6007, 6 42.4, 28.7; 7001, 60 27.0, 22.6; 10239, 9 61.9, 53.8; 6007, 1 71.9, 70.1;
// 9001, 1 149.9, 149.7).  With fewer rows than the chip takes four at a time wide ones lose (4097, 1
// 41.7, 45.7; 2101, 1 15.7, 25.0), narrow ones would gain (2101, 24 9.1, 5.0; 4097, 24 14.4, 9.7), and the host, which
// has the ranges on the device only, cannot tell them apart; so the line lies where no rows lose (4999, 1
// 53.9, 54.0).  Rows of more than 20 KB lose, whose zeros are better written by eight warps (f32 6007, 24
// 30.1, 32.7), and f32 ones (4097, 1 41.2, 49.4).
constexpr int kGroupRows = 4, kGroup = 32 * kGroupRows, kGroupMinRows = 5000, kGroupRowBytes = 20480;
template <int V>
__global__ void __launch_bounds__(kGroup, 10)
softmax_group_kernel(const __half* x, __half* out, const float* segs,
                     int64_t cols, int64_t wl, int64_t wr, int groups) {
  using T = __half;
  grid_dependency_wait();
  __shared__ float sM[2][kGroupRows], sS[2][kGroupRows];
  const bool group = (int)blockIdx.x < groups;
  int64_t row = group ? (int64_t)blockIdx.x * kGroupRows : (int64_t)groups * (kGroupRows - 1) + blockIdx.x;
  int64_t lo, hi;
  if (group) {
    const int64_t mine = row + (threadIdx.x >> 5);
    kept_range(segs, mine, cols, wl, wr, lo, hi);
    if (__syncthreads_and(hi - lo <= kWarpKept)) {
      softmax_row<T, By::Warp, V>(x, out, mine, cols, lo, hi, nullptr, nullptr);
      return;
    }
  } else {
    kept_range(segs, row, cols, wl, wr, lo, hi);
    if (hi - lo <= kWarpKept) {
      softmax_row<T, By::WarpInCta, V, kGroup>(x, out, row, cols, lo, hi, nullptr, nullptr);
      return;
    }
  }
#pragma unroll 1
  for (int r = 0; r < (group ? kGroupRows : 1); r++, row++) {
    // (two sets of sums: a row's are read while the next one's are written)
    kept_range(segs, row, cols, wl, wr, lo, hi);
    softmax_row<T, By::Cta, V, kGroup>(x, out, row, cols, lo, hi, sM[r & 1], sS[r & 1]);
  }
}

// A row by a warp, element by element.
template <typename T, bool MASKED>
__global__ void __launch_bounds__(kThreads)
softmax_element_kernel(const T* x, T* out, const float* segs, int64_t rows,
                       int64_t cols, int64_t wl, int64_t wr) {
  grid_dependency_wait();
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (row >= rows) return;
  int64_t lo = 0, hi = cols;
  if (MASKED) kept_range(segs, row, cols, wl, wr, lo, hi);
  const T* xr = x + row * cols;
  T* orow = out + row * cols;
  float m = kNegMax, s = 0.f;
  for (int64_t j = lo + lane; j < hi; j += 32) combine(m, s, to_f32<T>(xr[j]), 1.f);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    combine(m, s, __shfl_xor_sync(0xffffffffu, m, o), __shfl_xor_sync(0xffffffffu, s, o));
  const float inv = s > 0.f ? 1.f / s : 0.f;
  for (int64_t j = lane; j < cols; j += 32) {
    const bool kept = !MASKED || (j >= lo && j < hi);
    orow[j] = from_f32<T>(kept ? __expf(to_f32<T>(xr[j]) - m) * inv : 0.f);
  }
}

template <typename T, int V>
__global__ void __launch_bounds__(kThreads, kCtas)
softmax_warp_kernel(const T* x, T* out, const float* segs, int64_t rows,
                    int64_t cols, int64_t wl, int64_t wr) {
  grid_dependency_wait();
  const int64_t row = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
  if (row >= rows) return;
  int64_t lo, hi;
  kept_range(segs, row, cols, wl, wr, lo, hi);
  softmax_row<T, By::Warp, V>(x, out, row, cols, lo, hi, nullptr, nullptr);
}

template <typename T, int V>
cudaError_t softmax_chunked(const T* x, T* out, const float* segs, int64_t rows, int64_t cols,
                            int64_t wl, int64_t wr, cudaStream_t s) {
  const bool warpRows = cols <= kWarpRowCols;
  const int64_t blocks = warpRows ? (rows + kThreads / 32 - 1) / (kThreads / 32) : rows;
  if (blocks > 0x7fffffffll) return cudaErrorInvalidValue;
  const unsigned g = (unsigned)blocks;
  if constexpr (sizeof(T) == 2 && V > 1) {
    if (segs && rows >= kGroupMinRows && cols > kWarpRowCols && cols * 2 <= kGroupRowBytes) {
      const int groups = (int)(rows / 4 * 3 / kGroupRows);
      return launch_dependent(softmax_group_kernel<V>, dim3((unsigned)(rows - (int64_t)groups * (kGroupRows - 1))),
                              dim3(kGroup), 0, s, x, out, segs, cols, wl, wr, groups);
    }
  }
  if (warpRows)
    return launch_dependent(softmax_warp_kernel<T, V>, dim3(g), dim3(kThreads), 0, s, x, out, segs, rows, cols, wl, wr);
  return launch_dependent(softmax_cta_kernel<T, V>, dim3(g), dim3(kThreads), 0, s, x, out, segs, cols, wl, wr);
}

// The widest chunk at whose boundaries x and out agree: 16 bytes unless a caller's own memory
// puts them at different offsets from one.
template <typename T>
cudaError_t softmax_typed(const void* x, void* out, const float* segs, int64_t rows, int64_t cols,
                          int64_t wl, int64_t wr, cudaStream_t s) {
  auto* xi = static_cast<const T*>(x);
  auto* oi = static_cast<T*>(out);
  const uintptr_t both = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out);
  if (cols % 4 == 0 && cols < (1ll << 31) - 8 && both % (4 * sizeof(T)) == 0) {
    const bool warpRows = cols <= kWarpRowCols;
    const int64_t blocks = warpRows ? (rows + kThreads / 32 - 1) / (kThreads / 32) : rows;
    if (blocks > 0x7fffffffll) return cudaErrorInvalidValue;
    if (warpRows) return launch_dependent(softmax_quad_kernel<T, true>, dim3((unsigned)blocks), dim3(kThreads), 0, s, xi, oi, segs, rows, cols, wl, wr);
    return launch_dependent(softmax_quad_kernel<T, false>, dim3((unsigned)blocks), dim3(kThreads), 0, s, xi, oi, segs, rows, cols, wl, wr);
  }
  if (cols <= (segs ? kElementCols : kWarpRowCols)) {
    const int64_t blocks = (rows + kThreads / 32 - 1) / (kThreads / 32);
    if (blocks > 0x7fffffffll) return cudaErrorInvalidValue;
    const unsigned g = (unsigned)blocks;
    if (segs) return launch_dependent(softmax_element_kernel<T, true>, dim3(g), dim3(kThreads), 0, s, xi, oi, segs, rows, cols, wl, wr);
    return launch_dependent(softmax_element_kernel<T, false>, dim3(g), dim3(kThreads), 0, s, xi, oi, segs, rows, cols, wl, wr);
  }
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
