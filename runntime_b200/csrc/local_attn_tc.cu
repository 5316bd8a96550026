// localAttention (local_attn.cu has the op's definition) on the tensor cores: f16, heads of
// 64 or 128, windows up to 32.
//
// A CTA takes 64 consecutive rows of one head: TMA brings their q rows and the K and V rows
// they see (64 + WP, WP = 16 or 32 rows of halo before them; rows before the first are
// zero-filled) into shared memory, 128-byte swizzled.  Each of four warps owns 16 rows and
// 16 + WP keys:
//     S = q' K^T,  R = q' rel^T,  s_ij = cap tanh((kScale S_ij + R_i,i-j) / cap),  O = P V,
// with mma.sync m16n8k16.  R is one row of distances per query; the scores go through shared
// memory to where a lane finds them by (row, distance), as R's fragments lie, so that the soft cap
// and the exponential run on 16 or 32 elements of a row and not on its 32 or 48 keys, and
// the probabilities come back as the A operand of P V.  A CTA stays with its head and walks its row
// tiles, so that the bias rows are split once.
//
// (mma.sync and not tcgen05: the contraction is a band.  A 128-row tcgen05 tile would compute
// 128 x 160 scores for the 12 or 32 each row uses and take them through tensor memory, while
// at 16 rows a warp computes 32 or 48 per row; the tensor time is a third of the HBM time
// either way.)
//
// Precision is that of f32 products: q' = q qScale and rel are f32, P is f32.  Each is scaled
// by a power of two (per row; P, whose largest is one, by 2^13) and split into two halves hi + lo,
// 22 bits, and multiplied in two (three for R) MMAs with f32 accumulation; K and V are halves
// already.  No operand can overflow: the scale puts the row's largest element at 2^13.  (Without a scale
// P had an absolute 2^-25 in place of 22 bits: a key that weighs e^-12 was off by 2^-9 of itself.)  The
// tensor core adds into its accumulator less carefully than an FMA does, so the products of halves hi are
// added 32 columns at a time (64 in the widest form), the 2^-11 smaller ones apart.
//
// What bounds it: instructions, about 2 000 per warp and 16 rows, at 12 warps per SM (issue slots 46 %
// busy, DRAM 40 %).
// [32769, 3 x 8 x 128], window 12: 528 us for one warp per row on the FP32 pipes (local_attn.cu), 98 us
// with the soft cap on the scores' own fragments and the bias rows split for every tile, 74 us (73
// as a dependent launch); the slab and the output at the copy rate are 40 us.
#include "common.cuh"
#include "sm100.cuh"
#include "tc_common.cuh"

namespace rt {
namespace {

using namespace sm100;
using namespace tc;

constexpr int kRows = 64, kLocalThreads = 128;
constexpr float kProbScale = 8192.f;   // 2^13

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
// ... into zeros.
__device__ __forceinline__ void mma16816_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%10, %10, %10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
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
  // A warp's scores [16][16 + WP] f32, then its probabilities as halves hi and lo, eight rows at
  // two places each: in the warp's own q rows (of each 64-column box) where these are long enough.
  static constexpr int kScorePitch = (WP == 16 ? 40 : 56) * 4;  // float2 stores of four rows: distinct banks
  static constexpr int kProbPitch = WP == 16 ? 80 : 112;        // 16-byte pieces of eight rows: distinct banks
  static constexpr bool kOwn = HD < 128;
  static constexpr int kEight = kOwn ? 8 * kScorePitch : kRows * 128;   // from rows 0..7 to rows 8..15
  static constexpr int kQ = 0, kK = kQBytes, kV = kK + kKBytes, kRelHi = kV + kKBytes,
                       kRelLo = kRelHi + kRelBytes, kScratch = kRelLo + kRelBytes,
                       kSmem = kScratch + (kOwn ? 4 * 2 * 8 * kScorePitch : 0) + 1024;
  static_assert(16 * kProbPitch <= 8 * kScorePitch && (kOwn || 8 * kScorePitch <= 16 * 128), "fits its place");
};

// One row of one head from global memory, by one warp: rows whose tile holds numbers that are not
// finite, which a probability of zero or a low half would turn into NaN.
template <int HD>
__device__ __noinline__ void exact_row(const __half* qkv, const float* rel, const float* qScale, __half* out,
                                       int64_t t, int h, int heads, int window, float kScale, float softcap) {
  const int lane = threadIdx.x & 31;
  const int64_t width = (int64_t)heads * HD, col = (int64_t)h * HD;
  const int n = (int)min((int64_t)window, t + 1);
  float mine = -3.402823466e38f;     // lane j: the score j rows back
  for (int j = 0; j < n; j++) {
    float s = 0.f;
    for (int x = lane; x < HD; x += 32)
      s = fmaf(__half2float(qkv[t * 3 * width + col + x]) * qScale[x],
               fmaf(__half2float(qkv[(t - j) * 3 * width + width + col + x]), kScale, rel[j * width + col + x]), s);
    s = softcap * tanhf(warp_sum(s) / softcap);
    if (lane == j) mine = s;
  }
  const float m = warp_max(mine), e = lane < n ? expf(mine - m) : 0.f, inv = 1.f / warp_sum(e);
  for (int x = lane; x < HD; x += 32) {
    float acc = 0.f;
    for (int j = 0; j < n; j++)
      acc = fmaf(__shfl_sync(0xffffffffu, e, j), __half2float(qkv[(t - j) * 3 * width + 2 * width + col + x]), acc);
    out[t * width + col + x] = __float2half_rn(acc * inv);
  }
}

template <int HD, int WP>
__global__ void __launch_bounds__(kLocalThreads, 3)
local_attn_tc_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapKV,
                     const __half* qkv, const float* rel, const float* qScale, __half* out, int64_t rows, int heads,
                     int window, float kScale, float softcap, int* status) {
  using L = Local<HD, WP>;
  grid_dependency_wait();
  constexpr int NT = (16 + WP) / 8, KS = HD / 16;       // key tiles of a warp, steps of the head
  // Steps that an accumulator adds up before it joins the f32 sum.  (The widest form has no registers for
  // the sums of two: 4 bytes spilled, [9000, 3 x 8 x 128] with a window of 32 4 % slower.)
  constexpr int kSteps = HD == 128 && WP == 32 ? 4 : 2;
  extern __shared__ unsigned char smemRaw[];
  __shared__ __align__(8) uint64_t sFull;
  __shared__ float sRelInv[WP];
  __shared__ __align__(8) float sScale[HD];             // read in pairs
  __shared__ int sAbort;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;               // fragment row and column pair
  const uint32_t base = (smem_u32(smemRaw) + 1023u) & ~1023u;
  unsigned char* const generic = smemRaw + (base - smem_u32(smemRaw));
  const int h = (int)(blockIdx.x % (unsigned)heads);    // the launcher makes the grid a multiple of heads
  const int width = heads * HD;
  const int64_t tiles = (rows + kRows - 1) / kRows, step = gridDim.x / (unsigned)heads;
  const uint32_t bar = smem_u32(&sFull);

  auto load = [&](int64_t tile) {
    mbar_expect_tx(bar, L::kQBytes + 2 * L::kKBytes);
#pragma unroll
    for (int c = 0; c < HD; c += 64) {
      const int t0 = (int)(tile * kRows);
      tma_load_2d(base + L::kQ + c * 2 * kRows, &mapQ, h * HD + c, t0, bar);
      tma_load_2d(base + L::kK + c * 2 * L::kKeys, &mapKV, width + h * HD + c, t0 - WP, bar);
      tma_load_2d(base + L::kV + c * 2 * L::kKeys, &mapKV, 2 * width + h * HD + c, t0 - WP, bar);
    }
  };
  if (tid == 0) {
    sAbort = 0;
    mbar_init(bar, 1);
    fence_barrier_init();
    load(blockIdx.x / (unsigned)heads);
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

  const int r0 = warp * 16;
  unsigned char* const scratch =
      generic + (L::kOwn ? L::kScratch + warp * 2 * 8 * L::kScorePitch : L::kQ + r0 * 128);
  float* const score0 = reinterpret_cast<float*>(scratch + g * L::kScorePitch);   // row g; row g + 8 is kEight on
  uint32_t parity = 0;
  for (int64_t tile = blockIdx.x / (unsigned)heads; tile < tiles; tile += step, parity ^= 1) {
    const int64_t t0 = tile * kRows;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(bar, parity, &sAbort));
    if (ok) {
      // q' = q qScale of rows g and g + 8 of the warp's 16, as A fragments: largest magnitude of a
      // row first, then scaled and split.
      uint32_t qh[KS][4], ql[KS][4];
      float2 qf[KS][4];
      float mx[2] = {0.f, 0.f};
#pragma unroll
      for (int k = 0; k < KS; k++) {
        ldmatrix4(base + L::kQ + piece(r0 + (lane & 15), 2 * k + (lane >> 4), kRows), qh[k]);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&qh[k][i]));
          const float2 sc = *reinterpret_cast<const float2*>(&sScale[k * 16 + (i >> 1) * 8 + t4 * 2]);
          qf[k][i] = make_float2(f.x * sc.x, f.y * sc.y);
          mx[i & 1] = fmaxf(mx[i & 1], fmaxf(fabsf(qf[k][i].x), fabsf(qf[k][i].y)));
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
        for (int i = 0; i < 4; i++)
          split2(qf[k][i].x * qsc[i & 1], qf[k][i].y * qsc[i & 1], qh[k][i], ql[k][i]);

      // R [16, WP]: this lane has rows g (0, 1) and g + 8 (2, 3), distances 8 n + 2 t4 and the next.
      float r[WP / 8][4];
#pragma unroll
      for (int n = 0; n < WP / 8; n += 2) {
        float d[2][4], small[2][4];
#pragma unroll
        for (int k = 0; k < KS; k++) {
          const uint32_t at = piece(n * 8 + (lane & 7) + ((lane >> 4) << 3), 2 * k + ((lane >> 3) & 1), WP);
          uint32_t bh[4], bl[4];
          ldmatrix4(base + L::kRelHi + at, bh);
          ldmatrix4(base + L::kRelLo + at, bl);
#pragma unroll
          for (int e = 0; e < 2; e++) {
            if (k % kSteps == 0) mma16816_first(d[e], qh[k], bh[2 * e], bh[2 * e + 1]);
            else mma16816(d[e], qh[k], bh[2 * e], bh[2 * e + 1]);
            if (k == 0) mma16816_first(small[e], qh[k], bl[2 * e], bl[2 * e + 1]);
            else mma16816(small[e], qh[k], bl[2 * e], bl[2 * e + 1]);
            mma16816(small[e], ql[k], bh[2 * e], bh[2 * e + 1]);
            if (k % kSteps == kSteps - 1) {
#pragma unroll
              for (int i = 0; i < 4; i++) r[n + e][i] = k < kSteps ? d[e][i] : r[n + e][i] + d[e][i];
            }
          }
        }
#pragma unroll
        for (int e = 0; e < 2; e++)
#pragma unroll
          for (int i = 0; i < 4; i++) r[n + e][i] += small[e][i];
      }
      __syncwarp();      // the warp's q rows are in registers: their place is free

      // Scores of the warp's keys (staged rows r0 .. r0 + 16 + WP), to where a lane finds the keys
      // at its own distances.
#pragma unroll
      for (int n = 0; n < NT; n += 2) {
        if (WP - (8 * n + 15) >= window) continue;   // both tiles lie before every row's window
        float s[2][4], d[2][4], small[2][4];
#pragma unroll
        for (int k = 0; k < KS; k++) {
          uint32_t b[4];
          ldmatrix4(base + L::kK + piece(r0 + n * 8 + (lane & 7) + ((lane >> 4) << 3),
                                         2 * k + ((lane >> 3) & 1), L::kKeys), b);
#pragma unroll
          for (int e = 0; e < 2; e++) {
            if (k % kSteps == 0) mma16816_first(d[e], qh[k], b[2 * e], b[2 * e + 1]);
            else mma16816(d[e], qh[k], b[2 * e], b[2 * e + 1]);
            if (k == 0) mma16816_first(small[e], ql[k], b[2 * e], b[2 * e + 1]);
            else mma16816(small[e], ql[k], b[2 * e], b[2 * e + 1]);
            if (k % kSteps == kSteps - 1) {
#pragma unroll
              for (int i = 0; i < 4; i++) s[e][i] = k < kSteps ? d[e][i] : s[e][i] + d[e][i];
            }
          }
        }
#pragma unroll
        for (int e = 0; e < 2; e++)
#pragma unroll
          for (int i = 0; i < 2; i++)
            *reinterpret_cast<float2*>(score0 + i * (L::kEight / 4) + (n + e) * 8 + t4 * 2) =
                make_float2(s[e][2 * i] + small[e][2 * i], s[e][2 * i + 1] + small[e][2 * i + 1]);
      }
      __syncwarp();

      // Soft cap, mask and softmax by (row, distance).
      float m[2] = {-3.402823466e38f, -3.402823466e38f}, sum[2] = {0.f, 0.f};
#pragma unroll
      for (int n = 0; n < WP / 8; n++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int row = g + (i >> 1) * 8, dist = n * 8 + t4 * 2 + (i & 1);
          float x = -3.402823466e38f;
          if (dist < window && dist <= t0 + r0 + row) {
            const float dot = score0[(i >> 1) * (L::kEight / 4) + row + WP - dist];
            x = fmaf(dot, qinv[i >> 1] * kScale, r[n][i] * (qinv[i >> 1] * sRelInv[dist]));
            x = softcap * tanhf(x / softcap);
            m[i >> 1] = fmaxf(m[i >> 1], x);
          }
          r[n][i] = x;
        }
#pragma unroll
      for (int i = 0; i < 2; i++) {
        m[i] = fmaxf(m[i], __shfl_xor_sync(0xffffffffu, m[i], 1));
        m[i] = fmaxf(m[i], __shfl_xor_sync(0xffffffffu, m[i], 2));
      }
      __syncwarp();      // every score is read: its place takes the probabilities
#pragma unroll
      for (int i = lane; i < 2 * 16 * L::kProbPitch / 16; i += 32) {
        constexpr int kPieces = 16 * L::kProbPitch / 16;
        *reinterpret_cast<uint4*>(scratch + (i / kPieces) * L::kEight + i % kPieces * 16) = make_uint4(0, 0, 0, 0);
      }
      __syncwarp();
#pragma unroll
      for (int n = 0; n < WP / 8; n++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int row = g + (i >> 1) * 8, dist = n * 8 + t4 * 2 + (i & 1);
          if (dist < window && dist <= t0 + r0 + row) {
            const float pe = expf(r[n][i] - m[i >> 1]);
            sum[i >> 1] += pe;
            __half* at = reinterpret_cast<__half*>(scratch + (i >> 1) * L::kEight + g * L::kProbPitch) + row + WP - dist;
            const __half hi = __float2half_rn(pe * kProbScale);
            *at = hi;
            at[8 * L::kProbPitch / 2] = __float2half_rn(fmaf(pe, kProbScale, -__half2float(hi)));
          }
        }
#pragma unroll
      for (int i = 0; i < 2; i++) {
        sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 1);
        sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 2);
      }
      __syncwarp();

      // O = P V, sixteen keys at a time, the small products first.
      float o[HD / 8][4];
#pragma unroll
      for (int x = 0; x < HD / 8; x++)
#pragma unroll
        for (int i = 0; i < 4; i++) o[x][i] = 0.f;
#pragma unroll
      for (int n = 0; n < NT; n += 2) {
        if (WP - (8 * n + 15) >= window) continue;
        uint32_t ph[4], pl[4];
        const uint32_t at = smem_u32(scratch) + ((lane >> 3) & 1) * L::kEight + (lane & 7) * L::kProbPitch +
                            (n + (lane >> 4)) * 16;
        ldmatrix4(at, ph);
        ldmatrix4(at + 8 * L::kProbPitch, pl);
#pragma unroll
        for (int x = 0; x < HD / 8; x += 2) {
          uint32_t b[4];
          ldmatrix4_trans(base + L::kV + piece(r0 + n * 8 + (lane & 15), x + (lane >> 4), L::kKeys), b);
#pragma unroll
          for (int e = 0; e < 2; e++) {
            mma16816(o[x + e], pl, b[2 * e], b[2 * e + 1]);
            mma16816(o[x + e], ph, b[2 * e], b[2 * e + 1]);
          }
        }
      }
      __syncwarp();      // the probabilities are read: q's place takes the output

      // Through the warp's own q rows to whole 16-byte pieces of output rows.
      // distance 0 always exists: sum >= 1
      const float inv[2] = {1.f / (sum[0] * kProbScale), 1.f / (sum[1] * kProbScale)};
      bool odd = false;
#pragma unroll
      for (int x = 0; x < HD / 8; x++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const float a = o[x][2 * i] * inv[i], b = o[x][2 * i + 1] * inv[i];
          odd |= !(fabsf(a) + fabsf(b) < INFINITY);
          *reinterpret_cast<__half2*>(generic + L::kQ + piece(r0 + g + i * 8, x, kRows) + t4 * 4) =
              __floats2half2_rn(a, b);
        }
      odd = __any_sync(0xffffffffu, odd);
#pragma unroll
      for (int i = lane; i < 16 * HD / 8; i += 32) {
        const int rr = i / (HD / 8), c = i % (HD / 8);
        const int64_t row = t0 + r0 + rr;
        if (row < rows)
          *reinterpret_cast<uint4*>(out + row * width + (int64_t)h * HD + c * 8) =
              *reinterpret_cast<const uint4*>(generic + L::kQ + piece(r0 + rr, c, kRows));
      }
      if (odd) {
        __syncwarp();
        for (int i = 0; i < 16 && t0 + r0 + i < rows; i++)
          exact_row<HD>(qkv, rel, qScale, out, t0 + r0 + i, h, heads, window, kScale, softcap);
      }
    }
    // Everyone is done with the tile; what the threads wrote into it comes before the next copy.
    fence_proxy_async();
    if (!__syncthreads_and(ok)) {
      if (tid == 0) atomicOr(status, kStatusWaitTimeout);
      return;
    }
    if (tid == 0 && tile + step < tiles) load(tile + step);
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
  // As many blocks of a head as are resident at once (three per SM): each splits its head's bias
  // rows once and walks every step-th tile.
  const int64_t tiles = (rows + kRows - 1) / kRows, most = 3 * 148 / heads;
  const int64_t perHead = tiles < most ? tiles : most < 1 ? 1 : most;
  return launch_dependent(kern, dim3((unsigned)(perHead * heads)), dim3(kLocalThreads), L::kSmem, s, mq, mkv,
                          static_cast<const __half*>(qkv), rel, qScale, static_cast<__half*>(out), rows, heads, window,
                          kScale, softcap, status);
}

}  // namespace

// f16, heads of 64 or 128, tensors on 16-byte boundaries, coordinates within 31 bits, more than a few
// rows: a block's set-up, bias rows split among it, takes 5 to 12 us by window and head, a warp per row on
// the FP32 pipes (local_attn.cu) 5 to 7 for one to eight rows and 7 to 14 for twelve.
bool local_attn_tc_supported(const void* qkv, const float* rel, const void* out, int64_t rows,
                             int heads, int hd, int dtype) {
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  return dtype == RT_F16 && (hd == 64 || hd == 128) && rows > 8 && al(qkv) && al(rel) && al(out) &&
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
