// f32 matmul of more than a decode step's rows on the tensor cores: tf32 MMAs in threes, as in
// prefill_f32_tc.cu (which says why the products are whole to 2^-22 and how the accumulators are
// kept short).  K and N multiples of four, tensors on 16 bytes; other shapes are matmul.cu's.
//
// A CTA of four warps computes 64 x 64 of the output, a warp 32 x 32; chunks of 32 rows of b and
// columns of a come through a ring of three that cp.async fills.  An operand pair costs a warp 64
// instructions of splitting for 24 MMAs, and three CTAs per SM cover each other's chunk barriers;
// 64-wide tiles because the row counts in use (a clip's 40..1250, a batch's few thousand) would
// leave SMs idle with wider ones.
//
// Through the operator API, us (FP32 pipes -> here): [415, 288] x [288, 864] 50 -> 28, [4352, 384] x
// [384, 1536] 251 -> 109, [4352, 1536] x [1536, 384] 313 -> 110, [8192, 4096] x [4096, 512] 2082 -> 623
// (55 of the 92 TFLOP/s); error against 64 bits 3.0e-7 .. 1.1e-6 of the norm -> 1.4e-7 .. 2.4e-7.
//
// A result that is not finite is computed again in whole f32 products (see exact_row.cuh).
#include "common.cuh"
#include "sm100.cuh"
#include "tf32.cuh"

namespace rt {
namespace {

constexpr int TM = 64, TN = 64, TK = 32, kThreads = 128, kStages = 3;
// Half a warp's 8-byte loads of a are four rows x four pieces, a quarter's 16-byte loads of b four
// rows (every second one) x two pieces: these pitches give them distinct banks.
constexpr int kAPitch = TK + 8, kBPitch = TN + 4;
constexpr int kAFloats = TM * kAPitch, kStage = kAFloats + TK * kBPitch;
constexpr int kSmem = 4 * kStages * kStage;

__global__ void __launch_bounds__(kThreads, 3)
matmul_f32_tc_kernel(const float* a, const float* b, const float* bias, const float* addend, float* out, int64_t M,
                     int64_t K, int64_t N, int act) {
  extern __shared__ __align__(16) float ring[];
  grid_dependency_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;      // fragment row and column
  const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
  const int64_t row0 = (int64_t)blockIdx.y * TM, col0 = (int64_t)blockIdx.x * TN;
  const int64_t chunks = (K + TK - 1) / TK;

  int64_t filled = 0;
  int fillStage = 0;
  auto fill = [&]() {
    if (filled < chunks) {
      float* dst = ring + fillStage * kStage;
      const int64_t k0 = filled * TK;
#pragma unroll
      for (int i = 0; i < TM * TK / 4 / kThreads; i++) {
        const int idx = tid + i * kThreads, r = idx / (TK / 4), x = idx % (TK / 4) * 4;
        const bool in = row0 + r < M && k0 + x < K;
        copy_async16(dst + r * kAPitch + x, in ? a + (row0 + r) * K + k0 + x : a, in);
      }
#pragma unroll
      for (int i = 0; i < TK * TN / 4 / kThreads; i++) {
        const int idx = tid + i * kThreads, r = idx / (TN / 4), x = idx % (TN / 4) * 4;
        const bool in = k0 + r < K && col0 + x < N;
        copy_async16(dst + kAFloats + r * kBPitch + x, in ? b + (k0 + r) * N + col0 + x : b, in);
      }
      filled++;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (++fillStage == kStages) fillStage = 0;
  };
  for (int i = 0; i < kStages - 1; i++) fill();

  // s[m][j]: rows wm + 16 m + g (0, 1) and + 8 (2, 3), columns wn + 8 t4 + j and 4 further on
  float s[2][4][4], cross[2][4][4];
#pragma unroll
  for (int m = 0; m < 2; m++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) s[m][j][e] = cross[m][j][e] = 0.f;

  int useStage = 0;
  for (int64_t c = 0; c < chunks; c++) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();
    const float* sA = ring + useStage * kStage + (wm + g) * kAPitch + 2 * t4;
    const float* sB = ring + useStage * kStage + kAFloats + 2 * t4 * kBPitch + wn + 4 * g;
    fill();
    if (++useStage == kStages) useStage = 0;
    float d[2][4][4];
#pragma unroll
    for (int k = 0; k < TK / 8; k++) {
      // operand columns t4 and t4 + 4 are 2 t4 and 2 t4 + 1 of the eight
      uint32_t ah[2][4], al[2][4];
#pragma unroll
      for (int m = 0; m < 2; m++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
          const float2 f = *reinterpret_cast<const float2*>(sA + (16 * m + 8 * i) * kAPitch + 8 * k);
          split(f.x, ah[m][i], al[m][i]);
          split(f.y, ah[m][i + 2], al[m][i + 2]);
        }
      const float4 v0 = *reinterpret_cast<const float4*>(sB + 8 * k * kBPitch);
      const float4 v1 = *reinterpret_cast<const float4*>(sB + (8 * k + 1) * kBPitch);
      const float e0[4] = {v0.x, v0.y, v0.z, v0.w}, e1[4] = {v1.x, v1.y, v1.z, v1.w};
#pragma unroll
      for (int j = 0; j < 4; j++) {
        uint32_t bh0, bl0, bh1, bl1;
        split(e0[j], bh0, bl0);
        split(e1[j], bh1, bl1);
#pragma unroll
        for (int m = 0; m < 2; m++) {
          mma_tf32(cross[m][j], ah[m], bl0, bl1);
          if (k == 0) mma_tf32_first(d[m][j], ah[m], bh0, bh1);
          else mma_tf32(d[m][j], ah[m], bh0, bh1);
          mma_tf32(cross[m][j], al[m], bh0, bh1);
        }
      }
    }
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) s[m][j][e] += d[m][j][e];
  }

  act_dispatch(act, [&](auto code) {
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int half = 0; half < 2; half++) {
          const int64_t r = row0 + wm + 16 * m + g + 8 * i, n = col0 + wn + 8 * t4 + 4 * half;
          if (r >= M || n >= N) continue;
          float y[4];
#pragma unroll
          for (int j = 0; j < 4; j++) {
            y[j] = s[m][j][2 * i + half] + cross[m][j][2 * i + half];
            if (!(fabsf(y[j]) < INFINITY)) {
              y[j] = 0.f;
              for (int64_t x = 0; x < K; x++) y[j] = fmaf(a[r * K + x], b[x * N + n + j], y[j]);
            }
          }
          if (bias) {
#pragma unroll
            for (int j = 0; j < 4; j++) y[j] += bias[n + j];
          }
#pragma unroll
          for (int j = 0; j < 4; j++) y[j] = act_apply<decltype(code)::value>(y[j]);
          if (addend) {
            const float4 f = *reinterpret_cast<const float4*>(addend + r * N + n);
            y[0] += f.x, y[1] += f.y, y[2] += f.z, y[3] += f.w;
          }
          *reinterpret_cast<float4*>(out + r * N + n) = make_float4(y[0], y[1], y[2], y[3]);
        }
  });
}

}  // namespace

bool matmul_f32_tc_supported(const void* a, const void* b, const void* addend, const void* out, int64_t M,
                             int64_t K, int64_t N, int dtype) {
  const uintptr_t bases = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) |
                          reinterpret_cast<uintptr_t>(addend) | reinterpret_cast<uintptr_t>(out);
  return dtype == RT_F32 && M > 16 && K % 4 == 0 && N % 4 == 0 && bases % 16 == 0 && (M + TM - 1) / TM <= 65535 &&
         (N + TN - 1) / TN < (1ll << 31);
}

cudaError_t launch_matmul_f32_tc(const void* a, const void* b, const void* bias, const void* addend, void* out,
                                 int64_t M, int64_t K, int64_t N, int act, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(matmul_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  if (e != cudaSuccess) return e;
  const dim3 grid((unsigned)((N + TN - 1) / TN), (unsigned)((M + TM - 1) / TM));
  return launch_dependent(matmul_f32_tc_kernel, grid, dim3(kThreads), kSmem, s, static_cast<const float*>(a),
                          static_cast<const float*>(b), static_cast<const float*>(bias),
                          static_cast<const float*>(addend), static_cast<float*>(out), M, K, N, act);
}

}  // namespace rt
