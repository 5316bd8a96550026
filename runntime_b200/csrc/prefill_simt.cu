// General prefill attention on the FP32 pipes: every option of the 'attn' op,
// f32 or f16 storage, head sizes up to 512 that are a multiple of four, rows that start on four
// elements.  It takes the shapes that the tensor-core kernels do not; prefill_rows.cu takes the rest,
// and rows that see few keys.
//
// A CTA owns 32 query rows of one query head and walks the 64-key tiles of the union of its
// rows' bands.  K (64 keys x 64 columns at a time) and V
// (whole rows, 16 KB at a time) come through a ring of shared-memory chunks that cp.async
// fills three chunks ahead.  A warp owns 8 rows: lane x scores keys x and x + 32 and
// accumulates 4 columns in 128, so that K and V are read from shared memory with every lane at
// its own 16 bytes (a 16-byte load takes four passes whether or not half of its lanes repeat
// the other half's addresses) while q and the probabilities are broadcasts, one pass each, and the
// probabilities never leave the warp.  Heads of up to 32 or 64 columns need only 8 or 16 lanes
// for V: the rest of the warp takes other keys, added up at the end.
//
// The products are packed two to an instruction (fma.rn.f32x2): along the head for the
// scores, which leaves every score in two partial sums, along the columns for the output.
//
// What bounds it: the FMA pipes.  A two-wide FMA with three different operands issues every
// three cycles (48 TFLOP/s over the chip, measured; 73 with operands repeated), and two CTAs of four
// warps per SM leave a third of that unused.  f32, 8 sequences of 92..484 rows, 3 heads of 256 on
// one K/V head (2.4 GFLOP): 583 us with one score and HDP/32 columns per lane and 16-row tiles, 155 us.
//
// Replaces the reference's prefill routes
// (packages/runntime/src/core/kernels/attention/attn.ts:105-199,327-649 and
// attnFlash.ts:93-276) with one kernel; math and masking rules are theirs.
#include "common.cuh"
#include "exact_row.cuh"
#include "sm100.cuh"

namespace rt {
namespace {

constexpr int BQ = 32;      // query rows per CTA
constexpr int BK = 64;      // keys per tile
constexpr int kThreads = 128;
constexpr int kRows = 8;    // rows per warp
constexpr int PS = BK + 4;  // row pitch of the probabilities

using f32x2 = unsigned long long;
__device__ __forceinline__ void fma2(f32x2& d, f32x2 a, f32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ f32x2 pair(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 parts(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void scale2(f32x2& d, f32x2 a) {
  asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a));
}
// 16 bytes to shared memory in the background; zeros if !read.
__device__ __forceinline__ void copy_async16(float* dst, const void* src, bool read) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sm100::smem_u32(dst)), "l"(src),
               "r"(read ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __half* p) {
  const uint2 w = *reinterpret_cast<const uint2*>(p);
  const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w.x));
  const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store4(float* p, const float (&f)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
}
__device__ __forceinline__ void store4(__half* p, const float (&f)[4]) {
  const __half2 a = __floats2half2_rn(f[0], f[1]), b = __floats2half2_rn(f[2], f[3]);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

template <int HDP>  // head size rounded up to 32, 64, 128, 256 or 512
struct Shape {
  static constexpr int kDims = HDP < 64 ? HDP : 64;        // head columns per K chunk
  static constexpr int kKeyPitch = kDims + 4;              // eight consecutive keys: 32 distinct banks
  static constexpr int kVRows = HDP <= 64 ? BK : 4096 / HDP;  // keys per V chunk
  static constexpr int kVChunks = BK / kVRows;
  static constexpr int kChunk = BK * kKeyPitch > kVRows * HDP ? BK * kKeyPitch : kVRows * HDP;
  static constexpr int kStages = HDP == 64 ? 3 : 4;        // (a third CTA per SM is worth the stage)
  static constexpr int kQPitch = HDP + 4;
  static constexpr int kQuads = HDP <= 128 ? 1 : HDP / 128;   // 4-column pieces of the output per lane
  static constexpr int kSplit = HDP == 32 ? 4 : HDP == 64 ? 2 : 1;  // lanes that share a piece, by keys
  static constexpr int kSmem = 4 * (BQ * kQPitch + BQ * PS + kStages * kChunk);
  static constexpr int kCtas = HDP <= 64 ? 3 : HDP <= 256 ? 2 : 1;  // per SM
};

template <typename T, int HDP>
__global__ void __launch_bounds__(kThreads, Shape<HDP>::kCtas)
prefill_simt_kernel(const AttnParams p, int tilesPerSeq) {
  using S = Shape<HDP>;
  constexpr int NP = 2 * S::kQuads;          // column pairs of the output per lane and row
  constexpr int NJ = BK / 32;                // keys per lane
  constexpr bool ASYNC = sizeof(T) == 4;
  extern __shared__ __align__(16) float smem[];
  float* sQ = smem;                          // [BQ][kQPitch]
  float* sP = sQ + BQ * S::kQPitch;          // [BQ][PS]
  float* ring = sP + BQ * PS;                // [kStages][kChunk]
  __shared__ int64_t sLo[BQ], sEnd[BQ];

  const int hd = p.hd;
  const int tid = threadIdx.x, lane = tid & 31, r8 = tid / 32 * kRows;
  const int colLane = lane % (32 / S::kSplit), keyLane = lane / (32 / S::kSplit);
  // Later rows first: under a causal mask they are the longest.
  const int64_t tile = (int64_t)gridDim.x - 1 - blockIdx.x;
  // In a padded batch a tile stays inside its sequence.
  int64_t row0 = tile * BQ, rowEnd = p.qLen;
  if (p.seqStride > 0) {
    const int64_t b = tile / tilesPerSeq;
    row0 = b * p.seqStride + (tile - b * tilesPerSeq) * BQ;
    rowEnd = (b + 1) * p.seqStride;
  }
  const int h = blockIdx.y;
  const int kvh = h / (p.qHeads / p.kvHeads);
  const T* __restrict__ q = static_cast<const T*>(p.q) + (int64_t)h * hd;
  const T* __restrict__ k = static_cast<const T*>(p.k) + (int64_t)kvh * hd;
  const T* __restrict__ v = static_cast<const T*>(p.v) + (int64_t)kvh * hd;

  if (tid < BQ) {
    int64_t lo = 1, end = 0;
    if (row0 + tid < rowEnd) row_band(p, row0 + tid, lo, end);
    sLo[tid] = lo;
    sEnd[tid] = end;
  }
  // q, with zeros in the columns past the head and the rows past the tensor
  constexpr int Q4 = HDP / 4;
  for (int i = tid; i < BQ * Q4; i += kThreads) {
    const int r = i / Q4, x = (i % Q4) * 4;
    if (x >= hd) continue;
    const bool in = row0 + r < rowEnd;
    *reinterpret_cast<float4*>(sQ + r * S::kQPitch + x) =
        in ? load4(q + (row0 + r) * p.qStride + x) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();

  int64_t tileLo = INT64_MAX, tileEnd = -1;
#pragma unroll 8
  for (int r = 0; r < BQ; r++) {
    if (sLo[r] <= sEnd[r]) {
      tileLo = sLo[r] < tileLo ? sLo[r] : tileLo;
      tileEnd = sEnd[r] > tileEnd ? sEnd[r] : tileEnd;
    }
  }
  const int64_t span = tileEnd >= tileLo ? tileEnd - tileLo + 1 : 0;
  const int64_t tiles = (span + BK - 1) / BK;
  const int kChunks = (hd + S::kDims - 1) / S::kDims;   // K chunks per tile
  const int perTile = kChunks + S::kVChunks;

  // ---- the ring's filling side: chunks in the order they are used ----
  int64_t fillTile = 0;
  int fillPart = 0, fillStage = 0;
  auto fill = [&]() {
    if (fillTile < tiles) {
      float* dst = ring + fillStage * S::kChunk;
      const int64_t k0 = tileLo + fillTile * BK;
      const int nk = (int)min((int64_t)BK, tileEnd + 1 - k0);
      const bool isK = fillPart < kChunks;
      // [rows][width] of k or v from row r0 and column x0
      const T* src = isK ? k + k0 * p.kvStride : v + k0 * p.kvStride;
      const int r0 = isK ? 0 : (fillPart - kChunks) * S::kVRows;
      const int x0 = isK ? fillPart * S::kDims : 0;
      constexpr int KW = S::kDims / 4, VW = HDP / 4;
      constexpr int NK = BK * KW / kThreads, NV = S::kVRows * VW / kThreads;
      auto piece = [&](int r, int x, int pitch) {
        const bool in = r0 + r < nk;
        float* d = dst + r * pitch + x;
        const T* s = in ? src + (r0 + r) * p.kvStride + x0 + x : src;
        if (ASYNC) copy_async16(d, s, in);
        else *reinterpret_cast<float4*>(d) = in ? load4(s) : make_float4(0.f, 0.f, 0.f, 0.f);
      };
      if (isK) {
#pragma unroll
        for (int i = 0; i < NK; i++) {
          const int idx = tid + i * kThreads, r = idx / KW, x = (idx % KW) * 4;
          if (x0 + x < hd) piece(r, x, S::kKeyPitch);
        }
      } else {
#pragma unroll
        for (int i = 0; i < NV; i++) {
          const int idx = tid + i * kThreads, r = idx / VW, x = (idx % VW) * 4;
          if (x < hd) piece(r, x, HDP);
        }
      }
      if (++fillPart == perTile) fillPart = 0, fillTile++;
    }
    if (ASYNC) copies_commit();   // one group per chunk, empty ones at the end
    if (++fillStage == S::kStages) fillStage = 0;
  };
  int useStage = 0;
  // The next chunk has arrived for everyone, and everyone is done with the one before it,
  // whose place is filled again.
  auto advance = [&]() -> const float* {
    if (ASYNC) copies_wait<S::kStages - 2>();
    __syncthreads();
    const float* at = ring + useStage * S::kChunk;
    fill();
    if (++useStage == S::kStages) useStage = 0;
    return at;
  };
  for (int i = 0; i < S::kStages - 1; i++) fill();

  float m[kRows], l[kRows];   // l: this lane's share of the row sum
  f32x2 acc[kRows][NP];
#pragma unroll
  for (int i = 0; i < kRows; i++) {
    m[i] = kNegSeed;
    l[i] = 0.f;
    if (p.sinks) {
      m[i] = p.sinks[h] * 0.6931471805599453f;
      l[i] = lane == 0 ? 1.f : 0.f;
    }
#pragma unroll
    for (int c = 0; c < NP; c++) acc[i][c] = 0ull;
  }
  const float* qRow = sQ + r8 * S::kQPitch;
  float* pRow = sP + r8 * PS;

  for (int64_t t = 0; t < tiles; t++) {
    const int64_t k0 = tileLo + t * BK;
    const int nk = (int)min((int64_t)BK, tileEnd + 1 - k0);

    // ---- scores: rows r8 + i, keys lane + 32 j ----
    f32x2 s2[kRows][NJ];
#pragma unroll
    for (int i = 0; i < kRows; i++)
#pragma unroll
      for (int j = 0; j < NJ; j++) s2[i][j] = 0ull;
    for (int kc = 0; kc < kChunks; kc++) {
      const float* sK = advance() + lane * S::kKeyPitch;
      const float* sq = qRow + kc * S::kDims;
      const int steps = min(S::kDims, hd - kc * S::kDims) >> 2;
      auto dots = [&](auto n) {   // the first n x 32 keys of the tile
#pragma unroll 4
        for (int x = 0; x < steps; x++) {
          ulonglong2 kk[decltype(n)::value];
#pragma unroll
          for (int j = 0; j < decltype(n)::value; j++)
            kk[j] = *reinterpret_cast<const ulonglong2*>(sK + j * 32 * S::kKeyPitch + 4 * x);
#pragma unroll
          for (int i = 0; i < kRows; i++) {
            const ulonglong2 qq = *reinterpret_cast<const ulonglong2*>(sq + i * S::kQPitch + 4 * x);
#pragma unroll
            for (int j = 0; j < decltype(n)::value; j++) {
              fma2(s2[i][j], qq.x, kk[j].x);
              fma2(s2[i][j], qq.y, kk[j].y);
            }
          }
        }
      };
      if (nk > 32) dots(std::integral_constant<int, 2>{});
      else dots(std::integral_constant<int, 1>{});
    }

    // ---- online softmax; probabilities to shared memory for this warp ----
#pragma unroll
    for (int i = 0; i < kRows; i++) {
      const int lo = (int)min(max(sLo[r8 + i] - k0, (int64_t)-1), (int64_t)BK);
      const int end = (int)max(min(sEnd[r8 + i] - k0, (int64_t)BK), (int64_t)-1);
      float sc[NJ];
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < NJ; j++) {
        const int key = lane + j * 32;
        const float2 two = parts(s2[i][j]);
        float x = two.x + two.y;
        if (p.hasKeyBias && k0 + key >= p.biasStart && k0 + key < p.biasEnd) x += p.biasValue;
        sc[j] = (key >= lo && key <= end) ? x : -INFINITY;
        mx = fmaxf(mx, sc[j]);
      }
      mx = warp_max(mx);
      const float mNew = fmaxf(m[i], mx);
      const float corr = __expf(m[i] - mNew);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < NJ; j++) {
        const int key = lane + j * 32;
        const float pe = (key >= lo && key <= end) ? __expf(sc[j] - mNew) : 0.f;
        pRow[i * PS + key] = pe;
        sum += pe;
      }
      l[i] = l[i] * corr + sum;
      m[i] = mNew;
      const f32x2 c2 = pair(corr, corr);
#pragma unroll
      for (int c = 0; c < NP; c++) scale2(acc[i][c], c2);
    }
    __syncwarp();

    // ---- output: the same rows, columns 4 colLane + 128 c ----
#pragma unroll 1
    for (int vc = 0; vc < S::kVChunks; vc++) {
      const float* sV = advance() + 4 * colLane + 4 * keyLane * HDP;
      const int key0 = vc * S::kVRows;
      const int keys = min(S::kVRows, nk - key0);   // the rows past the last key hold zeros
      const float* pk = pRow + key0 + 4 * keyLane;
#pragma unroll 1
      for (int kk = 0; kk < keys; kk += 4 * S::kSplit) {
        float4 pr[kRows];
#pragma unroll
        for (int i = 0; i < kRows; i++) pr[i] = *reinterpret_cast<const float4*>(pk + i * PS + kk);
#pragma unroll
        for (int e = 0; e < 4; e++) {
          ulonglong2 vv[S::kQuads];
#pragma unroll
          for (int c = 0; c < S::kQuads; c++)
            vv[c] = *reinterpret_cast<const ulonglong2*>(sV + (kk + e) * HDP + 128 * c);
#pragma unroll
          for (int i = 0; i < kRows; i++) {
            const float x = e == 0 ? pr[i].x : e == 1 ? pr[i].y : e == 2 ? pr[i].z : pr[i].w;
            const f32x2 pp = pair(x, x);
#pragma unroll
            for (int c = 0; c < S::kQuads; c++) {
              fma2(acc[i][2 * c], pp, vv[c].x);
              fma2(acc[i][2 * c + 1], pp, vv[c].y);
            }
          }
        }
      }
    }
  }

  T* __restrict__ out = static_cast<T*>(p.out) + (int64_t)h * hd;
  const int64_t qw = (int64_t)p.qHeads * hd;
  const bool out4 = reinterpret_cast<uintptr_t>(p.out) % (4 * sizeof(T)) == 0;
  bool odd = false;   // something that is not finite
#pragma unroll
  for (int i = 0; i < kRows; i++) {
    const float sum = warp_sum(l[i]);
    const float invL = sum > 0.f ? 1.f / sum : 0.f;  // empty band -> zeros
    const int64_t row = row0 + r8 + i;
    T* o = out + row * qw;
#pragma unroll
    for (int c = 0; c < S::kQuads; c++) {
      const int x = 4 * colLane + 128 * c;
      const float2 a = parts(acc[i][2 * c]), b = parts(acc[i][2 * c + 1]);
      float f[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
      for (int e = 0; e < 4; e++) {
#pragma unroll
        for (int d = 16; d >= 32 / S::kSplit; d >>= 1) f[e] += __shfl_xor_sync(0xffffffffu, f[e], d);
        f[e] *= invL;
      }
      if (row >= rowEnd || keyLane != 0) continue;
#pragma unroll
      for (int e = 0; e < 4; e++) odd |= x + e < hd && !(fabsf(f[e]) < INFINITY);
      if (out4 && x < hd) {
        store4(o + x, f);
      } else {
#pragma unroll
        for (int e = 0; e < 4; e++)
          if (x + e < hd) o[x + e] = from_f32<T>(f[e]);
      }
    }
  }
  if (__any_sync(0xffffffffu, odd)) {
    for (int i = 0; i < kRows; i++)
      if (row0 + r8 + i < rowEnd) exact_row<T>(p, row0 + r8 + i, h, sLo[r8 + i], sEnd[r8 + i]);
  }
}

template <typename T, int HDP>
cudaError_t launch(const AttnParams& p, cudaStream_t s) {
  auto kern = prefill_simt_kernel<T, HDP>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape<HDP>::kSmem);
  if (e != cudaSuccess) return e;
  const int64_t perSeq = p.seqStride > 0 ? (p.seqStride + BQ - 1) / BQ : 0;
  const int64_t tiles = p.seqStride > 0 ? p.qLen / p.seqStride * perSeq : (p.qLen + BQ - 1) / BQ;
  kern<<<dim3((unsigned)tiles, (unsigned)p.qHeads), kThreads, Shape<HDP>::kSmem, s>>>(p, (int)perSeq);
  return cudaGetLastError();
}

// Every row of q, k and v of every head starts on four elements.  Without that this kernel's loads, one
// element each and a division for its place, cost more than its tiles save: [300, 8 x 33] f32 64 us, 42
// in 16-row pieces (prefill_rows.cu), [1000, 8 x 129] 707 and 715.
bool by_fours(const AttnParams& p, uintptr_t bytes) {
  const uintptr_t bases = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) |
                          reinterpret_cast<uintptr_t>(p.v);
  return p.hd % 4 == 0 && p.qStride % 4 == 0 && p.kvStride % 4 == 0 && bases % bytes == 0;
}

template <typename T>
cudaError_t dispatch_hd(const AttnParams& p, cudaStream_t s) {
  if (p.hd <= 32) return launch<T, 32>(p, s);
  if (p.hd <= 64) return launch<T, 64>(p, s);
  if (p.hd <= 128) return launch<T, 128>(p, s);
  if (p.hd <= 256) return launch<T, 256>(p, s);
  return launch<T, 512>(p, s);
}

}  // namespace

cudaError_t launch_prefill_simt(const AttnParams& p, int dtype, cudaStream_t s) {
  if (!by_fours(p, dtype == RT_F16 ? 8 : 16) || prefill_rows_better(p, dtype)) return launch_prefill_rows(p, dtype, s);
  return dtype == RT_F16 ? dispatch_hd<__half>(p, s) : dispatch_hd<float>(p, s);
}

}  // namespace rt
