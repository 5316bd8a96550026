// f16 prefill attention of packed short segments with heads of up to 32 columns (a text encoder over
// sentences or paragraphs, whose caller says how long the longest is).  Longer or unknown rows and
// wider heads are prefill_tc3.cu's.
//
// A CTA of four warps owns 64 query rows of one head, a warp 16 of them from the scores to the output
// in registers (mma.sync m16n8k16: the scores' fragments become the A operand of P V).  K and V
// tiles of 64 keys come by cp.async, two in flight; a warp passes over the tiles that none of its
// rows sees.
//
// Why not the 128-row tcgen05 tile of prefill_tc3.cu: a row that sees some 150 keys gives a CTA two or
// three key tiles, so the kernel is the latency of one CTA's chain (loads, MMA, tensor memory, softmax,
// MMA, read-out), most of a 128 x 128 tile of packed segments is masked, and half of its 64
// columns are padding.  Here four CTAs per SM overlap their chains and a 16-row warp skips what it
// does not see.  32 paragraphs of 16..256 tokens, 12 heads of 32: 33.9 us there, 20.6 here
// when this was written; among other launches 24.7, and 19.4 as a dependent launch whose key range is one redux.
// What bounds it: the exponentials and the fragments' way through shared memory, at 16 warps per SM.
#include "common.cuh"
#include "sm100.cuh"

namespace rt {
namespace {

constexpr int BQ = 64, BK = 64, HDP = 32, kThreads = 128;   // HDP: head columns, padded
constexpr int kPitch = HDP * 2 + 16;               // bytes: eight rows' 16-byte pieces in distinct banks
constexpr int kTile = BK * kPitch;
constexpr int kSmem = BQ * kPitch + 4 * kTile;     // q, two stages of K and V

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
// CB bytes to shared memory in the background; zeros if !read.
template <int CB>
__device__ __forceinline__ void copy_async(uint32_t dst, const void* src, bool read) {
  if constexpr (CB == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(read ? 16 : 0) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(read ? 8 : 0) : "memory");
}

// CB: bytes that rows of q, k, v and out can be moved by (16, or 8 for heads like 20).
template <int CB>
__global__ void __launch_bounds__(kThreads, 4)
prefill_mma_kernel(const AttnParams p, int tilesPerSeq) {
  constexpr int NT = BK / 8, KS = HDP / 16, NC = HDP / 8;
  constexpr int E = CB / 2, W = HDP / E;      // elements per piece, pieces per row
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int64_t sLo[BQ], sEnd[BQ];
  const int hd = p.hd;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;     // fragment row and column pair
  const uint32_t base = sm100::smem_u32(smem), sQ = base, sKV = base + BQ * kPitch;
  const int h = (int)(blockIdx.x % (unsigned)p.qHeads);
  // Later rows first: under a causal mask they are the longest.
  const int64_t tile = (int64_t)(gridDim.x / (unsigned)p.qHeads) - 1 - blockIdx.x / (unsigned)p.qHeads;
  // In a padded batch a tile stays inside its sequence.
  int64_t row0 = tile * BQ, rowEnd = p.qLen;
  if (p.seqStride > 0) {
    const int64_t b = tile / tilesPerSeq;
    row0 = b * p.seqStride + (tile - b * tilesPerSeq) * BQ;
    rowEnd = (b + 1) * p.seqStride;
  }
  rowEnd = min(rowEnd, row0 + BQ);
  const int kvh = h / (p.qHeads / p.kvHeads);
  grid_dependency_wait();
  const __half* __restrict__ q = static_cast<const __half*>(p.q) + (int64_t)h * hd;
  const __half* __restrict__ k = static_cast<const __half*>(p.k) + (int64_t)kvh * hd;
  const __half* __restrict__ v = static_cast<const __half*>(p.v) + (int64_t)kvh * hd;

  for (int i = tid; i < BQ * W; i += kThreads) {
    const int r = i / W, x = (i % W) * E;
    const bool in = row0 + r < rowEnd && x < hd;
    copy_async<CB>(sQ + r * kPitch + x * 2, in ? q + (row0 + r) * p.qStride + x : q, in);
  }
  if (tid < BQ) {
    int64_t lo = 1, end = 0;
    if (row0 + tid < rowEnd) row_band(p, row0 + tid, lo, end);
    sLo[tid] = lo;
    sEnd[tid] = end;
  }
  __syncthreads();
  int64_t tileLo, tileEnd;   // keys some row of the CTA sees
  {
    const bool a = sLo[lane] <= sEnd[lane], b = sLo[lane + 32] <= sEnd[lane + 32];
    // (key numbers are below 2^30: see prefill_mma_supported)
    const int first = min(a ? (int)sLo[lane] : INT32_MAX, b ? (int)sLo[lane + 32] : INT32_MAX);
    const int last = max(a ? (int)sEnd[lane] : -1, b ? (int)sEnd[lane + 32] : -1);
    tileLo = __reduce_min_sync(0xffffffffu, first);
    tileEnd = __reduce_max_sync(0xffffffffu, last);
  }
  const int span = tileEnd >= tileLo ? (int)(tileEnd - tileLo + 1) : 0;   // keys from here on relative to tileLo
  const int tiles = (span + BK - 1) / BK;
  // ... rows g and g + 8 of this warp, and the warp's whole range
  int lo[2], end[2], wLo = INT32_MAX, wEnd = -1, aLo = -1, aEnd = INT32_MAX;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const int r = warp * 16 + g + 8 * i;
    const bool any = sLo[r] <= sEnd[r];
    lo[i] = any ? (int)(sLo[r] - tileLo) : INT32_MAX;
    end[i] = any ? (int)(sEnd[r] - tileLo) : -1;
    wLo = min(wLo, lo[i]), wEnd = max(wEnd, end[i]);
    aLo = max(aLo, lo[i]), aEnd = min(aEnd, end[i]);
  }
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    wLo = min(wLo, __shfl_xor_sync(0xffffffffu, wLo, o)), wEnd = max(wEnd, __shfl_xor_sync(0xffffffffu, wEnd, o));
    aLo = max(aLo, __shfl_xor_sync(0xffffffffu, aLo, o)), aEnd = min(aEnd, __shfl_xor_sync(0xffffffffu, aEnd, o));
  }

  auto fill = [&](int t) {
    if (t < tiles) {
      const uint32_t dst = sKV + (t & 1) * 2 * kTile;
#pragma unroll
      for (int i = 0; i < BK * W / kThreads; i++) {
        const int idx = tid + i * kThreads, r = idx / W, x = (idx % W) * E;
        const bool in = t * BK + r < span && x < hd;   // zeros past the last key and column
        const int64_t at = in ? (tileLo + t * BK + r) * p.kvStride + x : 0;
        copy_async<CB>(dst + r * kPitch + x * 2, k + at, in);
        copy_async<CB>(dst + kTile + r * kPitch + x * 2, v + at, in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fill(0);      // (with q's copies in its group)
  fill(1);

  float m[2], l[2];     // l: this lane's share of the row sum
#pragma unroll
  for (int i = 0; i < 2; i++) {
    m[i] = p.sinks ? p.sinks[h] * 0.6931471805599453f : kNegSeed;
    l[i] = p.sinks && t4 == 0 ? 1.f : 0.f;
  }
  float o[NC][4];
#pragma unroll
  for (int c = 0; c < NC; c++)
#pragma unroll
    for (int e = 0; e < 4; e++) o[c][e] = 0.f;
  uint32_t qf[KS][4];

  for (int t = 0; t < tiles; t++) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    if (t == 0) {
#pragma unroll
      for (int s = 0; s < KS; s++)
        ldmatrix4(sQ + (warp * 16 + (lane & 15)) * kPitch + (2 * s + (lane >> 4)) * 16, qf[s]);
    }
    const int k0 = t * BK;
    if (k0 <= wEnd && k0 + BK - 1 >= wLo) {
      const uint32_t sK = sKV + (t & 1) * 2 * kTile, sV = sK + kTile;
      float s[NT][4];
#pragma unroll
      for (int n = 0; n < NT; n += 2) {
#pragma unroll
        for (int e = 0; e < 4; e++) s[n][e] = s[n + 1][e] = 0.f;
#pragma unroll
        for (int x = 0; x < KS; x++) {
          uint32_t b[4];
          ldmatrix4(sK + (n * 8 + (lane & 7) + ((lane >> 4) << 3)) * kPitch + (2 * x + ((lane >> 3) & 1)) * 16, b);
          mma16816(s[n], qf[x], b[0], b[1]);
          mma16816(s[n + 1], qf[x], b[2], b[3]);
        }
      }
      const bool masked = k0 < aLo || k0 + BK - 1 > aEnd || p.hasKeyBias;
      float corr[2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        float mx = -INFINITY;
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            float& x = s[n][2 * i + e];
            if (masked) {
              const int key = k0 + n * 8 + 2 * t4 + e;
              if (p.hasKeyBias && tileLo + key >= p.biasStart && tileLo + key < p.biasEnd) x += p.biasValue;
              if (key < lo[i] || key > end[i]) x = -INFINITY;
            }
            mx = fmaxf(mx, x);
          }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float mNew = fmaxf(m[i], mx);
        corr[i] = sm100::fast_exp2((m[i] - mNew) * kLog2e);
        m[i] = mNew;
        const float off = mNew * kLog2e;
        float sum = 0.f;
#pragma unroll
        for (int n = 0; n < NT; n++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const float pe = sm100::fast_exp2(fmaf(s[n][2 * i + e], kLog2e, -off));
            s[n][2 * i + e] = pe;
            sum += pe;
          }
        l[i] = l[i] * corr[i] + sum;
      }
#pragma unroll
      for (int c = 0; c < NC; c++)
#pragma unroll
        for (int e = 0; e < 4; e++) o[c][e] *= corr[e >> 1];
#pragma unroll
      for (int n = 0; n < NT; n += 2) {
        uint32_t pf[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const __half2 w = __floats2half2_rn(s[n + (i >> 1)][(i & 1) * 2], s[n + (i >> 1)][(i & 1) * 2 + 1]);
          pf[i] = *reinterpret_cast<const uint32_t*>(&w);
        }
#pragma unroll
        for (int c = 0; c < NC; c += 2) {
          uint32_t b[4];
          ldmatrix4_trans(sV + (n * 8 + (lane & 15)) * kPitch + (c + (lane >> 4)) * 16, b);
          mma16816(o[c], pf, b[0], b[1]);
          mma16816(o[c + 1], pf, b[2], b[3]);
        }
      }
    }
    __syncthreads();   // the tile is used up
    fill(t + 2);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (tiles == 0) __syncthreads();   // (q's copies have landed: its rows are written next)

  // Through the warp's own q rows (in registers since the first tile) to whole pieces of output rows.
  __half* __restrict__ out = static_cast<__half*>(p.out) + (int64_t)h * hd;
  unsigned char* const rows = smem + warp * 16 * kPitch;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
    l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
    const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;  // empty band -> zeros
#pragma unroll
    for (int c = 0; c < NC; c++)
      *reinterpret_cast<__half2*>(rows + (g + 8 * i) * kPitch + c * 16 + t4 * 4) =
          __floats2half2_rn(o[c][2 * i] * inv, o[c][2 * i + 1] * inv);
  }
  __syncwarp();
  using Piece = std::conditional_t<CB == 16, uint4, uint2>;
  for (int i = lane; i < 16 * W; i += 32) {
    const int r = i / W, x = (i % W) * E;
    const int64_t row = row0 + warp * 16 + r;
    if (row < rowEnd && x < hd)
      *reinterpret_cast<Piece*>(out + row * p.qHeads * hd + x) = *reinterpret_cast<const Piece*>(rows + r * kPitch + x * 2);
  }
}

template <int CB>
cudaError_t launch(const AttnParams& p, cudaStream_t s) {
  static_assert(kSmem <= 48 * 1024, "no opt-in to more shared memory");
  const int64_t perSeq = p.seqStride > 0 ? (p.seqStride + BQ - 1) / BQ : 0;
  const int64_t tiles = p.seqStride > 0 ? p.qLen / p.seqStride * perSeq : (p.qLen + BQ - 1) / BQ;
  return launch_dependent(prefill_mma_kernel<CB>, dim3((unsigned)(tiles * p.qHeads)), dim3(kThreads), kSmem, s, p, (int)perSeq);
}

int piece_bytes(const AttnParams& p) {
  const uintptr_t all = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) |
                        reinterpret_cast<uintptr_t>(p.v) | reinterpret_cast<uintptr_t>(p.out) |
                        (uintptr_t)(2 * p.hd) | (uintptr_t)(2 * p.qStride) | (uintptr_t)(2 * p.kvStride);
  return all % 16 == 0 ? 16 : all % 8 == 0 ? 8 : 0;
}

}  // namespace

// Heads of up to 32, and segments of up to 512 keys where the 64-row blocks make more than one per SM, by
// measurement against the tcgen05 kernel's 128-row blocks, us here and there, heads of 32: 39 segments
// of 512 keys, 12 heads 125 and 133, 2 heads 30 and 29; 17 of 350, 4 heads 22 and 25.  Shorter ones where
// a row has fewer than 64 bytes to move and the launch is not many blocks (heads of 20, 50 segments of 400, 2
// heads 36 and 33, 12 heads 135 and 141) and where the other kernel's blocks leave a fifth of the SMs idle, so
// that one of them is all of its time (23 of 256, 2 heads 10.2 and 9.2, 32 of 400, one head 20.5 and 15.3).  With fewer
// blocks of both: one segment of 256 7.7 and 8.6, of 500 12.5 and 12.  Where the tcgen05 kernel does not take
// the call the FP32 pipes would: 5 of 400, one head of 20: 58.
// Wider heads stay there: 8 segments of 300 keys, 8 heads of 36, in 64 padded columns 25 and 22.
bool prefill_mma_supported(const AttnParams& p, int dtype, bool other) {
  constexpr int64_t kSms = 148;
  const int64_t mine = (p.qLen + BQ - 1) / BQ * p.qHeads, theirs = (p.qLen + 127) / 128 * p.qHeads;
  const int most = !other                                ? 512
                   : mine < kSms                         ? 256
                   : theirs < 120                        ? 128
                   : p.hd <= 24 && theirs < 3 * kSms     ? 384
                                                         : 512;
  return dtype == RT_F16 && p.hd <= HDP && p.segs && p.maxSegment > 0 && p.maxSegment <= most &&
         piece_bytes(p) > 0 && p.kvLen < (1ll << 30) && p.qLen * p.qHeads < (1ll << 30);
}

cudaError_t launch_prefill_mma(const AttnParams& p, cudaStream_t s) {
  return piece_bytes(p) == 16 ? launch<16>(p, s) : launch<8>(p, s);
}

}  // namespace rt
