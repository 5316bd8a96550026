// localAttention (local_attn.cu has the op's definition) on the tensor cores: f16, heads of
// 64 or 128, windows up to 32.
//
// A CTA takes 64 consecutive rows of one head: TMA brings their q rows and the K and V rows
// they see (64 + WP, WP = 16 or 32 rows of halo before them; rows before the first are
// zero-filled) into shared memory, 128-byte swizzled.  Each of four warps owns 16 rows and
// 16 + WP keys and stays in registers from the scores to the output:
//     S = q' K^T,  R = q' rel^T,  s_ij = cap tanh((kScale S_ij + R_i,i-j) / cap),  O = P V,
// with mma.sync m16n8k16, the scores' fragments becoming the A operand of P V.  R is one row
// of distances per query; it goes through shared memory to be read along the diagonals.
//
// (mma.sync and not tcgen05: the contraction is a band.  A 128-row tcgen05 tile would compute
// 128 x 160 scores for the 12 or 32 each row uses and take them through tensor memory, while
// at 16 rows a warp computes 32 or 48 per row and nothing leaves its registers; the tensor
// time is a third of the HBM time either way.)
//
// Precision is that of f32 products: q' = q qScale and rel are f32, P is f32.  Each is scaled
// by a power of two per row and split into two halves hi + lo, 22 bits, and multiplied in two
// (three for R) MMAs with f32 accumulation; K and V are halves already.  No operand can
// overflow: the scale puts the row's largest element at 2^13.
//
// What bounds it: latency and instructions, about 2 800 per warp and 16 rows, of which 250 tensor
// or ldmatrix (ncu: issue slots 40 % busy at 12 warps per SM, DRAM 30 %).  [32769, 3 x 8 x 128],
// window 12: 528 us for one warp per row on the FP32 pipes (local_attn.cu) -> 98 us; the slab and
// the output at the copy rate are 42 us.
#include "common.cuh"
#include "sm100.cuh"
#include "tc_common.cuh"

namespace rt {
namespace {

using namespace sm100;
using namespace tc;

constexpr int kRows = 64, kLocalThreads = 128;

__device__ __forceinline__ void ldmatrix4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack2(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
// Two f32 values as halves hi and what is left of them as halves lo.
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  hi = pack2(h);
  lo = pack2(__floats2half2_rn(x - f.x, y - f.y));
}
// 2^(13 - e) for a row whose largest magnitude is in [2^e, 2^(e+1)), and its inverse; 1 for an
// all-zero row.  Both stay normal f32 numbers: e is clamped, which only rows of numbers below
// 2^-100 or above 2^100 meet.
__device__ __forceinline__ float row_scale(float mx, float& inverse) {
  int e = ((__float_as_int(mx) >> 23) & 255) - 127;
  if (mx == 0.f) e = 13;
  e = min(max(e, -100), 100);
  inverse = __int_as_float((e - 13 + 127) << 23);
  return __int_as_float((13 - e + 127) << 23);
}

// Byte offset of the 16-byte piece `chunk` (eight halves) of row `row` in a tile kept as
// boxes of 64 columns x `rows` rows, 128-byte swizzled (as TMA lays them down).
__device__ __forceinline__ uint32_t piece(int row, int chunk, int rows) {
  return (uint32_t)((chunk >> 3) * rows * 128 + row * 128 + (((chunk & 7) ^ (row & 7)) << 4));
}

template <int HD, int WP>
struct Local {
  static constexpr int kKeys = kRows + WP;              // staged K and V rows
  static constexpr int kQBytes = kRows * HD * 2, kKBytes = kKeys * HD * 2;
  static constexpr int kRelBytes = WP * HD * 2;         // one half of the split bias rows
  static constexpr int kSkew = WP + 7;                  // row pitch of R: eight banks from row to row on a diagonal
  static constexpr int kSkewBytes = 4 * 16 * kSkew * 4;
  static constexpr int kQ = 0, kK = kQBytes, kV = kK + kKBytes, kRelHi = kV + kKBytes,
                       kRelLo = kRelHi + kRelBytes, kSkewAt = kRelLo + kRelBytes,
                       kSmem = kSkewAt + kSkewBytes + 1024;
};

template <int HD, int WP>
__global__ void __launch_bounds__(kLocalThreads, 3)
local_attn_tc_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapKV,
                     const float* __restrict__ rel, const float* __restrict__ qScale,
                     __half* __restrict__ out, int64_t rows, int heads, int window, float kScale,
                     float softcap, int* status) {
  using L = Local<HD, WP>;
  constexpr int NT = (16 + WP) / 8, KS = HD / 16;       // key tiles of a warp, steps of the head
  extern __shared__ unsigned char smemRaw[];
  __shared__ __align__(8) uint64_t sFull;
  __shared__ float sRelInv[WP], sScale[HD];
  __shared__ int sAbort;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;               // fragment row and column pair
  const uint32_t base = (smem_u32(smemRaw) + 1023u) & ~1023u;
  unsigned char* const generic = smemRaw + (base - smem_u32(smemRaw));
  const int h = (int)(blockIdx.x % (unsigned)heads);
  const int64_t t0 = (int64_t)(blockIdx.x / (unsigned)heads) * kRows;
  const int width = heads * HD;

  if (tid == 0) {
    sAbort = 0;
    mbar_init(smem_u32(&sFull), 1);
    fence_barrier_init();
    const uint32_t bar = smem_u32(&sFull);
    mbar_expect_tx(bar, L::kQBytes + 2 * L::kKBytes);
#pragma unroll
    for (int c = 0; c < HD; c += 64) {
      tma_load_2d(base + L::kQ + c * 2 * kRows, &mapQ, h * HD + c, (int)t0, bar);
      tma_load_2d(base + L::kK + c * 2 * L::kKeys, &mapKV, width + h * HD + c, (int)t0 - WP, bar);
      tma_load_2d(base + L::kV + c * 2 * L::kKeys, &mapKV, 2 * width + h * HD + c, (int)t0 - WP, bar);
    }
  }
  // Bias rows, split into halves: a warp per distance.
  for (int j = warp; j < WP; j += 4) {
    float v[HD / 32];
    float mx = 0.f;
#pragma unroll
    for (int i = 0; i < HD / 64; i++) {
      const float2 f = j < window ? *reinterpret_cast<const float2*>(
                                        rel + (int64_t)j * width + (int64_t)h * HD + i * 64 + lane * 2)
                                  : make_float2(0.f, 0.f);
      v[2 * i] = f.x;
      v[2 * i + 1] = f.y;
      mx = fmaxf(mx, fmaxf(fabsf(f.x), fabsf(f.y)));
    }
    mx = warp_max(mx);
    float inv;
    const float sc = row_scale(mx, inv);
#pragma unroll
    for (int i = 0; i < HD / 64; i++) {
      uint32_t hi, lo;
      split2(v[2 * i] * sc, v[2 * i + 1] * sc, hi, lo);
      const uint32_t at = piece(j, i * 8 + (lane >> 2), WP) + (lane & 3) * 4;
      *reinterpret_cast<uint32_t*>(generic + L::kRelHi + at) = hi;
      *reinterpret_cast<uint32_t*>(generic + L::kRelLo + at) = lo;
    }
    if (lane == 0) sRelInv[j] = inv;
  }
  for (int x = tid; x < HD; x += kLocalThreads) sScale[x] = qScale[x];
  __syncthreads();
  const bool ok = mbar_wait(smem_u32(&sFull), 0, &sAbort);
  if (!__syncthreads_and(ok)) {
    if (tid == 0) atomicOr(status, kStatusWaitTimeout);
    return;
  }

  // q' = q qScale of rows g and g + 8 of the warp's 16, as A fragments: largest magnitude of a
  // row first, then scaled and split.
  const int r0 = warp * 16;
  uint32_t qh[KS][4], ql[KS][4];
  float mx[2] = {0.f, 0.f};
  auto scaled = [&](uint32_t w, int x) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    return make_float2(f.x * sScale[x], f.y * sScale[x + 1]);
  };
#pragma unroll
  for (int k = 0; k < KS; k++) {
    ldmatrix4(base + L::kQ + piece(r0 + (lane & 15), 2 * k + (lane >> 4), kRows), qh[k]);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float2 f = scaled(qh[k][i], k * 16 + (i >> 1) * 8 + t4 * 2);
      mx[i & 1] = fmaxf(mx[i & 1], fmaxf(fabsf(f.x), fabsf(f.y)));
    }
  }
  float qsc[2], qinv[2];
#pragma unroll
  for (int i = 0; i < 2; i++) {
    mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 1));
    mx[i] = fmaxf(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 2));
    qsc[i] = row_scale(mx[i], qinv[i]);
  }
#pragma unroll
  for (int k = 0; k < KS; k++)
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float2 f = scaled(qh[k][i], k * 16 + (i >> 1) * 8 + t4 * 2);
      split2(f.x * qsc[i & 1], f.y * qsc[i & 1], qh[k][i], ql[k][i]);
    }

  // R [16, WP], to shared memory in its natural order (row, distance).
  float* const skew = reinterpret_cast<float*>(generic + L::kSkewAt) + warp * 16 * L::kSkew;
#pragma unroll
  for (int n = 0; n < WP / 8; n += 2) {
    float r[2][4] = {};
#pragma unroll
    for (int k = 0; k < KS; k++) {
      const uint32_t at = piece(n * 8 + (lane & 7) + ((lane >> 4) << 3), 2 * k + ((lane >> 3) & 1), WP);
      uint32_t bh[4], bl[4];
      ldmatrix4(base + L::kRelHi + at, bh);
      ldmatrix4(base + L::kRelLo + at, bl);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        mma16816(r[e], qh[k], bh[2 * e], bh[2 * e + 1]);
        mma16816(r[e], qh[k], bl[2 * e], bl[2 * e + 1]);
        mma16816(r[e], ql[k], bh[2 * e], bh[2 * e + 1]);
      }
    }
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int j = (n + e) * 8 + t4 * 2 + (i & 1);
        skew[(g + (i >> 1) * 8) * L::kSkew + j] = r[e][i] * (qinv[i >> 1] * sRelInv[j]);
      }
  }
  __syncwarp();

  // Scores of the warp's keys (staged rows r0 .. r0 + 16 + WP), soft cap, mask.
  float s[NT][4];
  float m[2] = {-3.402823466e38f, -3.402823466e38f};
  const float kq[2] = {qinv[0] * kScale, qinv[1] * kScale};
  const int64_t firstKey = t0 - WP + r0;
#pragma unroll
  for (int n = 0; n < NT; n += 2) {
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
      for (int i = 0; i < 4; i++) s[n + e][i] = 0.f;
    if (WP - (8 * n + 15) >= window) {   // both tiles lie before every row's window
#pragma unroll
      for (int e = 0; e < 2; e++)
#pragma unroll
        for (int i = 0; i < 4; i++) s[n + e][i] = -3.402823466e38f;
      continue;
    }
#pragma unroll
    for (int k = 0; k < KS; k++) {
      uint32_t b[4];
      ldmatrix4(base + L::kK + piece(r0 + n * 8 + (lane & 7) + ((lane >> 4) << 3),
                                     2 * k + ((lane >> 3) & 1), L::kKeys), b);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        mma16816(s[n + e], qh[k], b[2 * e], b[2 * e + 1]);
        mma16816(s[n + e], ql[k], b[2 * e], b[2 * e + 1]);
      }
    }
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int row = g + (i >> 1) * 8, c = (n + e) * 8 + t4 * 2 + (i & 1), dist = row + WP - c;
        const bool seen = dist >= 0 && dist < window && firstKey + c >= 0;
        float x = -3.402823466e38f;
        if (seen) {
          x = fmaf(s[n + e][i], kq[i >> 1], skew[row * L::kSkew + dist]);
          x = softcap * tanhf(x / softcap);
          m[i >> 1] = fmaxf(m[i >> 1], x);
        }
        s[n + e][i] = x;
      }
  }
  float sum[2] = {0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 2; i++) {
    m[i] = fmaxf(m[i], __shfl_xor_sync(0xffffffffu, m[i], 1));
    m[i] = fmaxf(m[i], __shfl_xor_sync(0xffffffffu, m[i], 2));
  }
#pragma unroll
  for (int n = 0; n < NT; n++)
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float x = s[n][i];
      s[n][i] = x > -3e38f ? expf(x - m[i >> 1]) : 0.f;
      sum[i >> 1] += s[n][i];
    }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 1);
    sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 2);
  }

  // O = P V: tiles n and n + 1 of the scores are one k-step's A fragment.
  float o[HD / 8][4];
#pragma unroll
  for (int x = 0; x < HD / 8; x++)
#pragma unroll
    for (int i = 0; i < 4; i++) o[x][i] = 0.f;
#pragma unroll
  for (int n = 0; n < NT; n += 2) {
    if (WP - (8 * n + 15) >= window) continue;
    uint32_t ph[4], pl[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
      split2(s[n + (i >> 1)][(i & 1) * 2], s[n + (i >> 1)][(i & 1) * 2 + 1], ph[i], pl[i]);
#pragma unroll
    for (int x = 0; x < HD / 8; x += 2) {
      uint32_t b[4];
      ldmatrix4_trans(base + L::kV + piece(r0 + n * 8 + (lane & 15), x + (lane >> 4), L::kKeys), b);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        mma16816(o[x + e], ph, b[2 * e], b[2 * e + 1]);
        mma16816(o[x + e], pl, b[2 * e], b[2 * e + 1]);
      }
    }
  }

  // Through the warp's own q rows (read long ago) to whole 16-byte pieces of output rows.
  const float inv[2] = {1.f / sum[0], 1.f / sum[1]};   // distance 0 always exists: sum >= 1
#pragma unroll
  for (int x = 0; x < HD / 8; x++)
#pragma unroll
    for (int i = 0; i < 2; i++)
      *reinterpret_cast<__half2*>(generic + L::kQ + piece(r0 + g + i * 8, x, kRows) + t4 * 4) =
          __floats2half2_rn(o[x][2 * i] * inv[i], o[x][2 * i + 1] * inv[i]);
  __syncwarp();
#pragma unroll
  for (int i = lane; i < 16 * HD / 8; i += 32) {
    const int r = i / (HD / 8), c = i % (HD / 8);
    const int64_t row = t0 + r0 + r;
    if (row < rows)
      *reinterpret_cast<uint4*>(out + row * width + (int64_t)h * HD + c * 8) =
          *reinterpret_cast<const uint4*>(generic + L::kQ + piece(r0 + r, c, kRows));
  }
}

template <int HD, int WP>
cudaError_t launch(const void* qkv, const float* rel, const float* qScale, void* out, int64_t rows,
                   int heads, int window, float kScale, float softcap, int* status, cudaStream_t s,
                   std::string* err) {
  using L = Local<HD, WP>;
  const int64_t cols = 3ll * heads * HD;
  CUtensorMap mq, mkv;
  if (!make_map(&mq, qkv, rows, cols, cols, kRows, err) ||
      !make_map(&mkv, qkv, rows, cols, cols, L::kKeys, err))
    return cudaErrorInvalidValue;
  auto kern = local_attn_tc_kernel<HD, WP>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kSmem);
  if (e != cudaSuccess) return e;
  const int64_t blocks = (rows + kRows - 1) / kRows * heads;
  kern<<<(unsigned)blocks, kLocalThreads, L::kSmem, s>>>(mq, mkv, rel, qScale, static_cast<__half*>(out),
                                                         rows, heads, window, kScale, softcap, status);
  return cudaGetLastError();
}

}  // namespace

// f16, heads of 64 or 128, tensors on 16-byte boundaries, coordinates within 31 bits.
bool local_attn_tc_supported(const void* qkv, const float* rel, const void* out, int64_t rows,
                             int heads, int hd, int dtype) {
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  return dtype == RT_F16 && (hd == 64 || hd == 128) && al(qkv) && al(rel) && al(out) &&
         3ll * heads * hd < (1ll << 31) && (rows + kRows) * heads < (1ll << 31) && encode_fn() != nullptr;
}

cudaError_t launch_local_attn_tc(const void* qkv, const float* rel, const float* qScale, void* out,
                                 int64_t rows, int heads, int hd, int window, float kScale,
                                 float softcap, int* status, cudaStream_t s, std::string* err) {
  if (hd == 64)
    return window <= 16 ? launch<64, 16>(qkv, rel, qScale, out, rows, heads, window, kScale, softcap, status, s, err)
                        : launch<64, 32>(qkv, rel, qScale, out, rows, heads, window, kScale, softcap, status, s, err);
  return window <= 16 ? launch<128, 16>(qkv, rel, qScale, out, rows, heads, window, kScale, softcap, status, s, err)
                      : launch<128, 32>(qkv, rel, qScale, out, rows, heads, window, kScale, softcap, status, s, err);
}

}  // namespace rt
