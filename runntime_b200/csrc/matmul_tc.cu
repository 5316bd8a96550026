// Tensor-core matmul for the projections of a prefill (f16, more than 16 rows):
// out [M, N] = act(a [M, K] * b [K, N] + bias) + addend, f32 accumulation in tensor
// memory.  Same op as matmul.cu (packages/runntime/src/core/graph/ops/matmul.ts:28-99).
//
// One CTA per SM walks the 128 x BN output tiles (columns fastest).  Warp 8 streams K in
// steps of 64 through a ring of TMA loads: a 128 x 64 piece of a (K-major, 128-byte
// swizzle) and a 64 x BN piece of b as 64-column boxes (b is [K, N] row-major, that is
// MN-major for the MMA, the layout the V tiles of the attention kernels use).  Warp 9
// issues four tcgen05.mma (M = 128, N = BN, K = 16) per stage into one of two accumulators,
// so the K loop of a tile runs under the read-out of the tile before.  Warp 10 fetches the
// addend's tile into the staging buffer by TMA.  Warps 0-7 read the accumulator (a
// row and half of the columns per thread), apply bias, activation and addend in registers, leave the halves in the
// staging buffer in the swizzled layout (16 bytes per thread, no bank conflicts) and one
// thread stores it by TMA, which also clips the matrix edge.  Rows, columns and K past the
// matrices are zero-filled.  Every wait is bounded (sm100.cuh).
//
// What bounds it: with one tile per CTA (a speech clip, a few paragraphs) latency, launch to
// store; with many, the read-out's instructions where the activation has some, else the MMAs.
// The activation is a template parameter: with the seven of them in one kernel the read-out
// was larger than the instruction cache and stalled on fetches.  Measured, that kernel (a CTA
// per tile, stores and addend by row) and this one, launches back to back: [415, 288] x
// [288, 864] 9.0 -> 4.0 us; [4352, 384] x [384, 1152] 20.2 -> 9.1, x [384, 1536] + gelu 55 ->
// 12.9; [4352, 1536] x [1536, 384] + addend 24 -> 11.2; [32768, 1024] x [1024, 3072] 323 -> 204
// (1 011 TFLOP/s); 8192 x 4096 x 4096 279 -> 245 (1 124).
#include <cfloat>
#include "common.cuh"
#include "sm100.cuh"
#include "tc_common.cuh"

namespace rt {
namespace {

using namespace sm100;
using namespace tc;

constexpr int GBM = 128, GBK = 64;
constexpr int kReadThreads = 256;                   // two warpgroups, half of a tile's columns each
constexpr int kGemmThreads = kReadThreads + 96;
constexpr int kABytes = GBM * GBK * 2;
constexpr int kBoxBytes = GBM * 64 * 2;   // 64 columns of a tile in the staging buffer

template <int BN>
struct Gemm {
  static constexpr int kBBytes = GBK * BN * 2, kStage = kABytes + kBBytes;
  static constexpr int kStagings = BN == 256 ? 1 : 2;       // output tiles in flight to memory
  static constexpr int kStages = BN == 256 ? 3 : BN == 128 ? 5 : 6;
  static constexpr int kStaging = BN / 64 * kBoxBytes;
  static constexpr int kSmem = kStages * kStage + kStagings * kStaging + 1024;
};

// Barrier over the read-out warps that also ands a predicate: a wait that gave up in one
// thread ends the loop in all of them.
__device__ __forceinline__ bool readout_all(bool ok) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.aligned.pred q, 1, 256, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(ok ? 1u : 0u)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z),
               "r"(v.w)
               : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return fma2(a, b, make_float2(0.f, 0.f)); }

// gelu of a pair, the erf polynomial of act_apply in a form without the sign: x/2 (1 + erf(z)) =
// max(x, 0) - |x|/2 * poly(t) e^(-z^2), z = x / sqrt 2.  Packed arithmetic, one reciprocal and
// one exponential instruction per element: the special-function unit (16 per clock) is what is
// left to bound it, 2 048 cycles for a 128 x 128 tile ([4352, 384] x [384, 1536] + gelu: 15.1 us
// with the scalar form, 12.9 with this one).  +inf stays +inf: |x| ends at the largest finite number
// above zero, where the second term is an exact zero, and -inf is NaN as in x * 0.
__device__ __forceinline__ float2 gelu_pair(float2 x) {
  auto both = [](float c) { return make_float2(c, c); };
  const float2 ax = make_float2(fabsf(fminf(x.x, FLT_MAX)), fabsf(fminf(x.y, FLT_MAX)));
  const float2 d = fma2(ax, both(0.3275911f * 0.70710678118654752f), both(1.f));
  float2 t;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t.x) : "f"(d.x));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t.y) : "f"(d.y));
  float2 poly = fma2(both(1.061405429f), t, both(-1.453152027f));
  poly = fma2(poly, t, both(1.421413741f));
  poly = fma2(poly, t, both(-0.284496736f));
  poly = fma2(poly, t, both(0.254829592f));
  const float2 u = mul2(mul2(x, x), both(-0.5f * kLog2e));
  const float2 e = make_float2(fast_exp2(u.x), fast_exp2(u.y));
  const float2 w = mul2(mul2(poly, t), e);
  return fma2(mul2(ax, both(-0.5f)), w, make_float2(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f)));
}

// addMode: 0 = no addend, 1 = by TMA, 2 = element by element (an addend off a 16-byte boundary).
template <int BN, int ACT>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
               const __grid_constant__ CUtensorMap mapAdd, const __grid_constant__ CUtensorMap mapOut,
               const __half* bias, const __half* addend, int addMode,
               int64_t M, int64_t K, int64_t N, int tilesN, int tiles, int* status) {
  using G = Gemm<BN>;
  extern __shared__ unsigned char smemRaw[];
  __shared__ __align__(8) uint64_t sFull[G::kStages], sEmpty[G::kStages], sAccFull[2], sAccEmpty[2];
  __shared__ __align__(8) uint64_t sAddFull[2], sStgFree[2];
  __shared__ __align__(16) float sBias[2][BN];
  __shared__ uint32_t sTmemBase;
  __shared__ int sAbort;
  const int tid = threadIdx.x, warp = tid >> 5;
  const uint32_t smemBase = (smem_u32(smemRaw) + 1023u) & ~1023u;
  const uint32_t stgBase = smemBase + G::kStages * G::kStage;
  const int nk = (int)((K + GBK - 1) / GBK);

  if (tid == 0) {
    sAbort = 0;
    for (int s = 0; s < G::kStages; s++) {
      mbar_init(smem_u32(&sFull[s]), 1);
      mbar_init(smem_u32(&sEmpty[s]), 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(smem_u32(&sAccFull[b]), 1);
      mbar_init(smem_u32(&sAccEmpty[b]), kReadThreads / 32);
      mbar_init(smem_u32(&sAddFull[b]), 1);
      mbar_init(smem_u32(&sStgFree[b]), 1);
    }
    fence_barrier_init();
  }
  if (warp == 8 && elect_one()) {
    prefetch_tensormap(&mapA);
    prefetch_tensormap(&mapB);
    prefetch_tensormap(&mapOut);
  }
  if (warp == 9) {
    tmem_alloc(smem_u32(&sTmemBase), 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sTmemBase;
  // Everything above touched no global memory; what follows reads tensors the grid before
  // this one may have written and overwrites out, which it may still read.
  grid_dependency_wait();

  if (warp == 8) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      int it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const int row0 = tile / tilesN * GBM, col0 = tile % tilesN * BN;
        for (int k = 0; k < nk; k++, it++) {
          const int s = it % G::kStages;
          if (it >= G::kStages && !mbar_poll(smem_u32(&sEmpty[s]), ((it / G::kStages) - 1) & 1, &sAbort)) {
            ok = false;
            break;
          }
          const uint32_t bar = smem_u32(&sFull[s]);
          const uint32_t dA = smemBase + s * G::kStage, dB = dA + kABytes;
          mbar_expect_tx(bar, G::kStage);
          tma_load_2d(dA, &mapA, k * GBK, row0, bar);                  // 64 k x 128 rows
#pragma unroll
          for (int c = 0; c < BN; c += 64)                             // 64 columns x 64 k each
            tma_load_2d(dB + c * GBK * 2, &mapB, col0 + c, k * GBK, bar);
        }
      }
      if (!ok) sAbort = 1;
      grid_launch_dependents();
    }
  } else if (warp == 9) {
    // ------------------------------ MMA issuer --------------------------------
    constexpr uint32_t idesc = instr_desc(BN, true);
    constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO, version, SW128
    constexpr uint32_t kLboA = (16u >> 4) << 16;                          // K-major operand
    constexpr uint32_t kLboB = ((uint32_t)(GBK * 128) >> 4) << 16;        // MN-major: next 64 columns
    bool ok = true;
    int it = 0, t = 0;
    for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, t++) {
      const int b = t & 1;
      if (t >= 2) ok = mbar_poll_warp(smem_u32(&sAccEmpty[b]), ((t >> 1) - 1) & 1, &sAbort);
      for (int k = 0; k < nk && ok; k++, it++) {
        const int s = it % G::kStages;
        ok = mbar_poll_warp(smem_u32(&sFull[s]), (it / G::kStages) & 1, &sAbort);
        if (!ok) break;
        tc_fence_after_sync();
        if (elect_one()) {
          const uint32_t aLo = (((smemBase + s * G::kStage) >> 4) & 0x3fffu) | kLboA;
          const uint32_t bLo = (((smemBase + s * G::kStage + kABytes) >> 4) & 0x3fffu) | kLboB;
#pragma unroll
          for (int kk = 0; kk < GBK / 16; kk++) {
            const uint64_t aDesc = ((uint64_t)kDescHi << 32) | (aLo + kk * 2);
            const uint64_t bDesc = ((uint64_t)kDescHi << 32) | (bLo + kk * (2048 >> 4));
            mma_f16_ss(tmem + b * BN, aDesc, bDesc, idesc, (k > 0 || kk > 0) ? 1u : 0u);
          }
          tc_commit(smem_u32(&sEmpty[s]));
          if (k == nk - 1) tc_commit(smem_u32(&sAccFull[b]));
        }
        __syncwarp();
      }
    }
    if (!ok) sAbort = 1;
  } else if (warp == 10) {
    // ------------------------------ addend loads ------------------------------
    if (addMode == 1 && elect_one()) {
      int t = 0;
      for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, t++) {
        const int row0 = tile / tilesN * GBM, col0 = tile % tilesN * BN;
        const int g = t % G::kStagings;
        if (t >= G::kStagings &&
            !mbar_poll(smem_u32(&sStgFree[g]), ((t / G::kStagings) - 1) & 1, &sAbort)) {
          sAbort = 1;
          break;
        }
        const uint32_t bar = smem_u32(&sAddFull[g]);
        mbar_expect_tx(bar, G::kStaging);
#pragma unroll
        for (int c = 0; c < BN / 64; c++)
          tma_load_2d(stgBase + g * G::kStaging + c * kBoxBytes, &mapAdd, col0 + c * 64, row0, bar);
      }
    }
  } else {
    // ------------------------------ read-out ----------------------------------
    const int row = tid & 127, half = tid >> 7;   // row of the tile, half of its columns
    int t = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, t++) {
      const int row0 = tile / tilesN * GBM, col0 = tile % tilesN * BN;
      const int b = t & 1, g = t % G::kStagings;
      if (tid < BN) {
        const int c = tid;
        sBias[b][c] = (bias && col0 + c < N) ? __half2float(bias[col0 + c]) : 0.f;
      }
      bool ok = mbar_poll(smem_u32(&sAccFull[b]), (t >> 1) & 1, &sAbort);
      if (ok && addMode == 1)
        ok = mbar_poll(smem_u32(&sAddFull[g]), (t / G::kStagings) & 1, &sAbort);
      if (!ok) sAbort = 1;
      // (also: this tile's bias is in place, and the store that last used the staging buffer
      // has read it — thread 0 waited for that before it came here)
      if (!readout_all(ok)) break;
      tc_fence_after_sync();
      const uint32_t acc0 = tmem + b * BN + ((uint32_t)((warp & 3) * 32) << 16);
      const uint32_t stg = stgBase + g * G::kStaging + row * 128;
#pragma unroll 1
      for (int c = half * (BN / 2); c < (half + 1) * (BN / 2); c += 32) {
        uint32_t acc[32];
        tmem_ld32(acc0 + c, acc);
        tmem_wait_ld();
        const uint32_t box = stg + (c >> 6) * kBoxBytes;
#pragma unroll
        for (int v = 0; v < 4; v++) {
          const uint32_t at = box + (((((c & 32) >> 3) + v) ^ (row & 7)) << 4);
          const float4 b0 = *reinterpret_cast<const float4*>(&sBias[b][c + v * 8]);
          const float4 b1 = *reinterpret_cast<const float4*>(&sBias[b][c + v * 8 + 4]);
          const float bs[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
          float y[8];
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            const float x0 = __uint_as_float(acc[v * 8 + e]) + bs[e];
            const float x1 = __uint_as_float(acc[v * 8 + e + 1]) + bs[e + 1];
            if (ACT == 2) {
              const float2 r = gelu_pair(make_float2(x0, x1));
              y[e] = r.x;
              y[e + 1] = r.y;
            } else {
              y[e] = act_apply<ACT, true>(x0);
              y[e + 1] = act_apply<ACT, true>(x1);
            }
          }
          if (addMode == 1) {
            const uint4 w = ld_shared_v4(at);
            const __half2* h = reinterpret_cast<const __half2*>(&w);
#pragma unroll
            for (int e = 0; e < 4; e++) {
              const float2 f = __half22float2(h[e]);
              y[2 * e] += f.x;
              y[2 * e + 1] += f.y;
            }
          } else if (addMode == 2 && row0 + row < M) {
            for (int e = 0; e < 8; e++) {
              const int64_t n = col0 + c + v * 8 + e;
              if (n < N) y[e] += __half2float(addend[(int64_t)(row0 + row) * N + n]);
            }
          }
          uint4 w;
          __half2* h = reinterpret_cast<__half2*>(&w);
#pragma unroll
          for (int e = 0; e < 4; e++) h[e] = __floats2half2_rn(y[2 * e], y[2 * e + 1]);
          st_shared_v4(at, w);
        }
      }
      tc_fence_before_sync();
      fence_proxy_async();
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(smem_u32(&sAccEmpty[b]));
      readout_all(true);
      if (tid == 0) {
#pragma unroll
        for (int c = 0; c < BN / 64; c++)
          if (col0 + c * 64 < N)
            tma_store_2d(&mapOut, stgBase + g * G::kStaging + c * kBoxBytes, col0 + c * 64, row0);
        bulk_commit();
        bulk_wait_read<G::kStagings - 1>();   // the store before the last kStagings - 1 has been read
        if (t >= G::kStagings - 1) mbar_arrive(smem_u32(&sStgFree[(t + 1) % G::kStagings]));
      }
    }
    if (tid == 0) bulk_wait<0>();   // shared memory stays until the stores are done with it
  }

  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && sAbort) atomicOr(status, kStatusWaitTimeout);
  if (warp == 9) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 2 * BN);
  }
}

// ---- up to 16 rows (the projections of a decode step) -------------------------------
// HBM-bound: the weights are read once, 2 K N bytes.  The product is computed
// transposed, out^T [N, M] = b^T [N, K] * a^T [K, M], so that 128 columns of the weights
// fill the 128 rows of one tcgen05.mma (A operand MN-major, exactly as TMA lays a
// [64 k, 64 columns] box of b down) and the few rows of a are its N = 16 side.  The
// tensor core is far from busy; it is here because it takes the weights straight from
// shared memory, where a SIMT kernel spends 64 FMAs per 16-byte load.
//
// One CTA owns 128 output columns and one slice of K; the slices of a column tile form
// a thread-block cluster (1, 2, 4 or 8 CTAs).  Each CTA streams its slice through a
// three-stage TMA ring into a 16-column accumulator; the CTAs of rank > 0 then write
// their accumulators into the shared memory of rank 0 (distributed shared memory),
// one hardware cluster barrier orders that, and rank 0 adds them, applies bias,
// activation and addend and stores.  One launch, no atomics, no scratch.
#ifndef RT_SK_STAGES
#define RT_SK_STAGES 3
#endif
#ifndef RT_SK_CTAS_PER_SM
#define RT_SK_CTAS_PER_SM 2
#endif
#ifndef RT_SK_MIN_CTAS
#define RT_SK_MIN_CTAS 3
#endif
constexpr int SKN = 128, SKM = 16, SKK = 64, SKSTAGES = RT_SK_STAGES;
constexpr int kSkB = SKK * SKN * 2, kSkA = SKM * SKK * 2, kSkStage = kSkB + kSkA;   // 16 KB + 2 KB
constexpr int kSkThreads = 192;
constexpr int kSkMaxCluster = 8;

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// The address, in the cluster's shared window, of `addr` in the CTA of rank `rank`.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
// The hardware barrier over all threads of the cluster, in its two halves.
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Optional per-CTA timeline for kernel development (off unless the translation unit is
// compiled with RT_SK_TRACE): thread 0 of every CTA stores the GPU-wide nanosecond timer at
// eight points of the kernel.
#ifdef RT_SK_TRACE
__device__ unsigned long long gSkTrace[4096 * 8];
#define SK_MARK(i)                                                                        \
  do {                                                                                    \
    if (threadIdx.x == (i == 2 ? 160 : 0)) {                                              \
      unsigned long long t_;                                                              \
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));                              \
      gSkTrace[((blockIdx.y * gridDim.x + blockIdx.x) & 4095) * 8 + (i)] = t_;            \
    }                                                                                     \
  } while (0)
#else
#define SK_MARK(i) \
  do {             \
  } while (0)
#endif

// rowsPad: 8 or 16, the rows of a that are exchanged and stored (M <= rowsPad).
__global__ void __launch_bounds__(kSkThreads, RT_SK_MIN_CTAS)
gemm_tc_skinny_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                      const __half* bias, const __half* addend, __half* out, int M, int64_t K, int64_t N, int stepsPerRank,
                      int rowsPad, int act, int* status) {
  extern __shared__ unsigned char smemRaw[];
  __shared__ __align__(8) uint64_t sFull[SKSTAGES], sEmpty[SKSTAGES], sAcc;
  __shared__ uint32_t sTmemBase;
  __shared__ int sAbort;
  const int tid = threadIdx.x, warp = tid >> 5;
  SK_MARK(0);
  const uint32_t smemBase = (smem_u32(smemRaw) + 1023u) & ~1023u;
  const uint32_t redBase = smemBase + SKSTAGES * kSkStage;   // [rank - 1][rowsPad][128] f32, rank 0 only
  const uint32_t rank = cluster_rank(), ranks = cluster_size();
  const int64_t col0 = (int64_t)blockIdx.x * SKN;
  const int nkAll = (int)((K + SKK - 1) / SKK);
  const int it0 = (int)rank * stepsPerRank;
  const int nk = max(0, min(stepsPerRank, nkAll - it0));     // K steps of this CTA; may be none

  if (tid == 0) {
    sAbort = 0;
    for (int s = 0; s < SKSTAGES; s++) {
      mbar_init(smem_u32(&sFull[s]), 1);
      mbar_init(smem_u32(&sEmpty[s]), 1);
    }
    mbar_init(smem_u32(&sAcc), 1);
    fence_barrier_init();
  }
  if (warp == 5) {
    tmem_alloc(smem_u32(&sTmemBase), 32);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sTmemBase;
  SK_MARK(1);
  // The first weights may be asked into the L2 meanwhile, whoever wrote them last ([8, 4096] x [4096, 4096]
  // 15.9 -> 15.6 us among launches, x [4096, 12288] 19.6 -> 19.2; twice as many steps take the bandwidth
  // from the grid that is still at work: 17.8 and 23.4).
  constexpr int kPrefetchSteps = 6;
  if (warp == 4 && elect_one()) {
    for (int it = 0; it < min(nk, kPrefetchSteps); it++) {
      tma_prefetch_2d(&mapB, (int)col0, (it0 + it) * SKK);
      tma_prefetch_2d(&mapB, (int)col0 + 64, (it0 + it) * SKK);
    }
  }
  // Everything above touched no global memory; what follows reads tensors the grid before
  // this one may have written (a, addend) and overwrites out, which it may still read.
  grid_dependency_wait();
  cluster_arrive();   // first barrier: every CTA of the cluster is running (waited on below)

  if (warp == 4) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      prefetch_tensormap(&mapA);
      prefetch_tensormap(&mapB);
      for (int it = 0; it < nk; it++) {
        const int s = it % SKSTAGES;
        if (it >= SKSTAGES && !mbar_park(smem_u32(&sEmpty[s]), ((it / SKSTAGES) - 1) & 1, &sAbort)) {
          sAbort = 1;
          break;
        }
        const uint32_t bar = smem_u32(&sFull[s]);
        const uint32_t dB = smemBase + s * kSkStage, dA = dB + kSkB;
        const int k0 = (it0 + it) * SKK;
        mbar_expect_tx(bar, kSkStage);
        tma_load_2d(dB, &mapB, (int)col0, k0, bar);                  // 64 columns x 64 k
        tma_load_2d(dB + SKK * 128, &mapB, (int)col0 + 64, k0, bar);
        tma_load_2d(dA, &mapA, k0, 0, bar);                          // 64 k x 16 rows of a
      }
    }
  } else if (warp == 5) {
    // ------------------------------ MMA issuer --------------------------------
    // D [128 columns of b, 16 rows of a]: A = b^T (MN-major), B = a (K-major), f32 D.
    constexpr uint32_t idesc = (1u << 4) | (1u << 15) | ((uint32_t)(SKM >> 3) << 17) |
                               ((uint32_t)(SKN >> 4) << 24);
    constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO, version, SW128
    constexpr uint32_t kLboMn = ((uint32_t)(SKK * 128) >> 4) << 16;       // next 64 columns of b
    constexpr uint32_t kLboK = (16u >> 4) << 16;
    bool ok = true;
    for (int it = 0; it < nk && ok; it++) {
      const int s = it % SKSTAGES;
      ok = __all_sync(0xffffffffu, mbar_park(smem_u32(&sFull[s]), (it / SKSTAGES) & 1, &sAbort));
      if (!ok) break;
      tc_fence_after_sync();
      if (it == 0) SK_MARK(2);
      if (elect_one()) {
        // In a cluster the shared-window address of a CTA carries its rank above the
        // offset; the descriptor's address field takes the 14 offset bits only (left
        // in, the rank lands in the leading-dimension field beside it).
        const uint32_t wLo = (((smemBase + s * kSkStage) >> 4) & 0x3fffu) | kLboMn;
        const uint32_t xLo = (((smemBase + s * kSkStage + kSkB) >> 4) & 0x3fffu) | kLboK;
#pragma unroll
        for (int kk = 0; kk < SKK / 16; kk++) {
          const uint64_t wDesc = ((uint64_t)kDescHi << 32) | (wLo + kk * (2048 >> 4));
          const uint64_t xDesc = ((uint64_t)kDescHi << 32) | (xLo + kk * 2);
          mma_f16_ss(tmem, wDesc, xDesc, idesc, (it > 0 || kk > 0) ? 1u : 0u);
        }
        tc_commit(smem_u32(&sEmpty[s]));
        if (it == nk - 1) tc_commit(smem_u32(&sAcc));
      }
      __syncwarp();
    }
    if (!ok) sAbort = 1;
  }

  // Accumulator of this CTA: thread = column, 16 values = rows of a.
  float acc[SKM];
#pragma unroll
  for (int m = 0; m < SKM; m++) acc[m] = 0.f;
  if (warp < 4 && nk > 0) {
    const bool ok = __all_sync(0xffffffffu, mbar_park(smem_u32(&sAcc), 0, &sAbort));
    if (!ok) sAbort = 1;
    if (ok) {
      tc_fence_after_sync();
      uint32_t raw[SKM];
      tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16), raw);
      tmem_wait_ld();
#pragma unroll
      for (int m = 0; m < SKM; m++) acc[m] = __uint_as_float(raw[m]);
    }
  }
  SK_MARK(3);
  grid_launch_dependents();   // the weights of this CTA are in: the next grid may set itself up
  __syncwarp();
  cluster_wait();
  if (warp < 4 && rank > 0) {
    const uint32_t dst = map_to_rank(redBase, 0) + (((rank - 1) * rowsPad) * SKN + tid) * 4;
#pragma unroll
    for (int m = 0; m < SKM; m++)
      if (m < rowsPad) st_cluster_f32(dst + m * SKN * 4, acc[m]);
  }
  // Second barrier: the partial sums are in rank 0's shared memory.  Every thread of every
  // CTA of the cluster reaches both barriers whatever happened above.
  __syncwarp();
  cluster_arrive();
  cluster_wait();
  SK_MARK(4);

  if (warp < 4 && rank == 0) {
    const float* red = reinterpret_cast<const float*>(smemRaw + (redBase - smem_u32(smemRaw)));
    for (uint32_t r = 1; r < ranks; r++)
#pragma unroll
      for (int m = 0; m < SKM; m++)
        if (m < rowsPad) acc[m] += red[((r - 1) * rowsPad + m) * SKN + tid];
    const int64_t n = col0 + tid;
    if (n < N) {
      const float bv = bias ? __half2float(bias[n]) : 0.f;
      act_dispatch(act, [&](auto code) {
#pragma unroll
        for (int m = 0; m < SKM; m++) {
          if (m < M) {
            float y = act_apply<decltype(code)::value>(acc[m] + bv);
            if (addend) y += __half2float(addend[(int64_t)m * N + n]);
            out[(int64_t)m * N + n] = __float2half_rn(y);
          }
        }
      });
    }
  }

  SK_MARK(5);
  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && sAbort) atomicOr(status, kStatusWaitTimeout);
  if (warp == 5) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 32);
  }
  SK_MARK(6);
}

}  // namespace

// f16, whole 16-byte row pitches, at least one box of every operand.  Up to 16 rows go
// to the cluster kernel (which wants a full tile of columns), more to the tiled one.
bool matmul_tc_supported(const void* a, const void* b, const void* out, int64_t M, int64_t K,
                         int64_t N, int dtype) {
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  return dtype == RT_F16 && M >= 1 && K >= 64 && N >= (M <= SKM ? SKN : 64) && K % 8 == 0 &&
         N % 8 == 0 && al(a) && al(b) && al(out) && M < (1ll << 31) - 256 && N < (1ll << 31) - 256 &&
         K < (1ll << 31) - 256 &&
         ((M + GBM - 1) / GBM) * ((N + 63) / 64) < (1ll << 31) && encode_fn() != nullptr;
}

namespace {
constexpr int kSms = 148;

// Columns of an output tile: the width whose slowest SM is done first.  Microseconds, measured:
// a K step is bound by the L2 delivering its operands (24 / 32 / 48 KB at about 90 GB/s per SM),
// the read-out takes 8 ns a column, 24 with an activation, and hides under the K loop of the
// next tile.  [16384, 384] x [384, 1152]: 32 / 20 / 24 us with 64 / 128 / 256 columns,
// [32768, 1024] x [1024, 3072]: 378 / 253 / 204, [415, 288] x [288, 864]: 4.0 / 4.8 / 7.0.
int tile_columns(int64_t M, int64_t K, int64_t N, int act) {
  const double nk = (double)((K + GBK - 1) / GBK);
  int best = 64;
  double bestCost = 1e30;
  for (int bn : {64, 128, 256}) {
    const int64_t tiles = ((N + bn - 1) / bn) * ((M + GBM - 1) / GBM);
    const double waves = (double)((tiles + kSms - 1) / kSms);
    const double loop = nk * (bn == 256 ? 0.545 : bn == 128 ? 0.33 : 0.285);
    const double readout = bn * (act ? 0.024 : 0.008);
    const double cost = waves * ((loop > readout ? loop : readout) + 0.2) + readout;
    if (cost < bestCost) best = bn, bestCost = cost;
  }
  return best;
}

cudaError_t launch_skinny(const void* a, const void* b, const void* bias, const void* addend,
                          void* out, int64_t M, int64_t K, int64_t N, int act, int* status,
                          cudaStream_t s, std::string* err) {
  CUtensorMap ma, mb;
  if (!make_map(&ma, a, M, K, K, SKM, err) || !make_map(&mb, b, K, N, N, SKK, err))
    return cudaErrorInvalidValue;
  // Slices of K: enough CTAs for two per SM, at least two K steps each.
  const int64_t tiles = (N + SKN - 1) / SKN;
  const int nkAll = (int)((K + SKK - 1) / SKK);
  int cluster = 1;
  while (cluster < kSkMaxCluster && tiles * cluster < RT_SK_CTAS_PER_SM * 148 && nkAll / (cluster * 2) >= 2) cluster *= 2;
  const int stepsPerRank = (nkAll + cluster - 1) / cluster;
  const int rowsPad = M <= 8 ? 8 : 16;
  const int smem = SKSTAGES * kSkStage + 1024 + (cluster - 1) * rowsPad * SKN * 4;
  cudaError_t e = cudaFuncSetAttribute(gemm_tc_skinny_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)tiles, (unsigned)cluster);
  cfg.blockDim = dim3(kSkThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = (unsigned)cluster;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, gemm_tc_skinny_kernel, ma, mb, static_cast<const __half*>(bias),
                            static_cast<const __half*>(addend), static_cast<__half*>(out), (int)M,
                            K, N, stepsPerRank, rowsPad, act, status);
}
}  // namespace

namespace {
template <int BN, int ACT>
cudaError_t launch_tiled(const void* a, const void* b, const void* bias, const void* addend,
                         void* out, int64_t M, int64_t K, int64_t N, int* status, cudaStream_t s,
                         std::string* err) {
  using G = Gemm<BN>;
  CUtensorMap ma, mb, madd, mo;
  if (!make_map(&ma, a, M, K, K, GBM, err) || !make_map(&mb, b, K, N, N, GBK, err) ||
      !make_map(&mo, out, M, N, N, GBM, err))
    return cudaErrorInvalidValue;
  madd = mo;
  int addMode = 0;
  if (addend) {
    addMode = (reinterpret_cast<uintptr_t>(addend) & 15u) == 0 ? 1 : 2;
    if (addMode == 1 && !make_map(&madd, addend, M, N, N, GBM, err)) return cudaErrorInvalidValue;
  }
  auto kern = gemm_tc_kernel<BN, ACT>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, G::kSmem);
  if (e != cudaSuccess) return e;
  const int64_t tilesN = (N + BN - 1) / BN, tiles = tilesN * ((M + GBM - 1) / GBM);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles < kSms ? tiles : kSms));
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = G::kSmem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, ma, mb, madd, mo, static_cast<const __half*>(bias),
                            static_cast<const __half*>(addend), addMode, M, K, N, (int)tilesN,
                            (int)tiles, status);
}

template <int BN>
cudaError_t launch_tiled_act(const void* a, const void* b, const void* bias, const void* addend,
                             void* out, int64_t M, int64_t K, int64_t N, int act, int* status,
                             cudaStream_t s, std::string* err) {
  switch (act) {
    case 1: return launch_tiled<BN, 1>(a, b, bias, addend, out, M, K, N, status, s, err);
    case 2: return launch_tiled<BN, 2>(a, b, bias, addend, out, M, K, N, status, s, err);
    case 3: return launch_tiled<BN, 3>(a, b, bias, addend, out, M, K, N, status, s, err);
    case 4: return launch_tiled<BN, 4>(a, b, bias, addend, out, M, K, N, status, s, err);
    case 5: return launch_tiled<BN, 5>(a, b, bias, addend, out, M, K, N, status, s, err);
    case 6: return launch_tiled<BN, 6>(a, b, bias, addend, out, M, K, N, status, s, err);
    default: return launch_tiled<BN, 0>(a, b, bias, addend, out, M, K, N, status, s, err);
  }
}
}  // namespace

cudaError_t launch_matmul_tc(const void* a, const void* b, const void* bias, const void* addend,
                             void* out, int64_t M, int64_t K, int64_t N, int act, int* status,
                             cudaStream_t s, std::string* err) {
  if (M <= SKM) return launch_skinny(a, b, bias, addend, out, M, K, N, act, status, s, err);
  const int bn = tile_columns(M, K, N, act);
  if (bn == 256) return launch_tiled_act<256>(a, b, bias, addend, out, M, K, N, act, status, s, err);
  if (bn == 128) return launch_tiled_act<128>(a, b, bias, addend, out, M, K, N, act, status, s, err);
  return launch_tiled_act<64>(a, b, bias, addend, out, M, K, N, act, status, s, err);
}

}  // namespace rt
