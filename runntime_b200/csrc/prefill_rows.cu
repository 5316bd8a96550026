// Prefill attention on the FP32 pipes in small pieces: every option of the 'attn' op, f32 or f16
// storage, any head size up to 512, any alignment.  It takes rows that see few keys and rows that
// cannot be read four elements at a time; prefill_simt.cu's tiles take the rest.
//
// A CTA owns 16 query rows of one query head, of as many sequences as they belong to, and walks the
// key tiles of the union of its rows' bands.  K and V tiles of 32 keys are staged in shared
// memory as f32; each warp owns 4 rows: lane j scores key j of the tile for
// the 4 rows, the online softmax reduces across the warp, then lane x
// accumulates output columns x, x+32, ... with the probabilities broadcast by
// shuffles.  32 columns of the head are added before they join a score, so that no f32 sum is
// long.
//
// What bounds it: the scalar FMAs and a shuffle for every four of them, which is why it is only the
// better one where a tile of 32 rows x 64 or 128 keys would be mostly masked.  Measured against the
// tile kernels at prefill_rows_better below.
//
// A value that is not finite reaches only the rows that see its key: tiles that hold one are added up
// key by key for the rows that see it.
//
// Replaces the reference's prefill routes
// (packages/runntime/src/core/kernels/attention/attn.ts:105-199,327-649 and
// attnFlash.ts:93-276); math and masking rules are theirs.
#include "common.cuh"

namespace rt {
namespace {

constexpr int BQ = 16;      // query rows per CTA
constexpr int BK = 32;      // keys per tile (one per lane)
constexpr int WARPS = 4;
constexpr int RPW = BQ / WARPS;  // rows per warp

template <typename T, int NC>  // NC = ceil(hd / 32) output columns per lane
__global__ void __launch_bounds__(WARPS * 32, NC == 1 ? 8 : NC == 2 ? 7 : NC == 4 ? 6 : NC == 8 ? 5 : 4)
prefill_rows_kernel(const AttnParams p) {
  extern __shared__ __align__(16) float smem[];
  const int hd = p.hd;
  const int ks = hd | 1;          // odd row stride: lanes read distinct banks
  const int vs = NC * 32;         // V rows padded to whole lanes, pad = 0
  float* sQ = smem;               // [hd][BQ], transposed so 4 rows load as one float4
  float* sK = sQ + hd * BQ;       // [BK][ks]
  float* sV = sK + BK * ks;       // [BK][vs]
  __shared__ int64_t sLo[BQ], sEnd[BQ];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * BQ;
  const int h = blockIdx.y;
  const int kvh = h / (p.qHeads / p.kvHeads);
  const T* __restrict__ q = static_cast<const T*>(p.q);
  const T* __restrict__ k = static_cast<const T*>(p.k) + (int64_t)kvh * hd;
  const T* __restrict__ v = static_cast<const T*>(p.v) + (int64_t)kvh * hd;

  if (tid < BQ) {
    int64_t lo = 1, end = 0;
    if (row0 + tid < p.qLen) row_band(p, row0 + tid, lo, end);
    sLo[tid] = lo;
    sEnd[tid] = end;
  }
  for (int idx = tid; idx < BQ * hd; idx += WARPS * 32) {
    const int r = idx / hd, x = idx - r * hd;
    const int64_t row = row0 + r;
    sQ[x * BQ + r] = row < p.qLen ? to_f32<T>(q[row * p.qStride + (int64_t)h * hd + x]) : 0.f;
  }
  // V pad columns stay zero for the whole kernel.
  if (vs != hd) {
    for (int idx = tid; idx < BK * (vs - hd); idx += WARPS * 32) {
      const int jj = idx / (vs - hd), x = hd + idx % (vs - hd);
      sV[jj * vs + x] = 0.f;
    }
  }
  __syncthreads();

  int64_t tileLo = INT64_MAX, tileEnd = -1;
#pragma unroll
  for (int r = 0; r < BQ; r++) {
    if (sLo[r] <= sEnd[r]) {
      tileLo = sLo[r] < tileLo ? sLo[r] : tileLo;
      tileEnd = sEnd[r] > tileEnd ? sEnd[r] : tileEnd;
    }
  }
  int64_t lo[RPW], end[RPW];
  float m[RPW], l[RPW], acc[RPW][NC];
#pragma unroll
  for (int r = 0; r < RPW; r++) {
    lo[r] = sLo[warp * RPW + r];
    end[r] = sEnd[warp * RPW + r];
    m[r] = kNegSeed;
    l[r] = 0.f;
    if (p.sinks) {
      m[r] = p.sinks[h] * 0.6931471805599453f;
      l[r] = 1.f;
    }
#pragma unroll
    for (int c = 0; c < NC; c++) acc[r][c] = 0.f;
  }

  for (int64_t k0 = tileLo; k0 <= tileEnd; k0 += BK) {
    const int nk = (int)((tileEnd - k0 + 1) < BK ? (tileEnd - k0 + 1) : BK);
    bool odd = false;   // a value that is not finite
    __syncthreads();  // previous tile fully consumed
    for (int idx = tid; idx < BK * hd; idx += WARPS * 32) {
      const int jj = idx / hd, x = idx - jj * hd;
      float kv = 0.f, vv = 0.f;
      if (jj < nk) {
        const int64_t off = (k0 + jj) * p.kvStride + x;
        kv = to_f32<T>(k[off]);
        vv = to_f32<T>(v[off]);
      }
      sK[jj * ks + x] = kv;
      sV[jj * vs + x] = vv;
      odd |= !(fabsf(vv) < INFINITY);
    }
    odd = __syncthreads_or(odd) != 0;

    // Does any of this warp's rows see any key of the tile?
    bool warpLive = false;
#pragma unroll
    for (int r = 0; r < RPW; r++) warpLive |= (lo[r] <= k0 + nk - 1) && (end[r] >= k0);
    if (!warpLive) continue;

    float s[RPW];
#pragma unroll
    for (int r = 0; r < RPW; r++) s[r] = 0.f;
    const float* kr = sK + lane * ks;
    const float4* q4 = reinterpret_cast<const float4*>(sQ) + warp;
    int x = 0;
    for (; x + 32 <= hd; x += 32) {
      float d[RPW] = {};
#pragma unroll
      for (int i = 0; i < 32; i++) {
        const float kx = kr[x + i];
        const float4 qq = q4[(x + i) * (BQ / 4)];
        d[0] = fmaf(qq.x, kx, d[0]);
        d[1] = fmaf(qq.y, kx, d[1]);
        d[2] = fmaf(qq.z, kx, d[2]);
        d[3] = fmaf(qq.w, kx, d[3]);
      }
#pragma unroll
      for (int r = 0; r < RPW; r++) s[r] += d[r];
    }
    float d[RPW] = {};
    for (; x < hd; x++) {
      const float kx = kr[x];
      const float4 qq = q4[x * (BQ / 4)];
      d[0] = fmaf(qq.x, kx, d[0]);
      d[1] = fmaf(qq.y, kx, d[1]);
      d[2] = fmaf(qq.z, kx, d[2]);
      d[3] = fmaf(qq.w, kx, d[3]);
    }
#pragma unroll
    for (int r = 0; r < RPW; r++) s[r] += d[r];
    const int64_t j = k0 + lane;
    const float bias = (p.hasKeyBias && j >= p.biasStart && j < p.biasEnd) ? p.biasValue : 0.f;
    float pr[RPW];
#pragma unroll
    for (int r = 0; r < RPW; r++) {
      const bool vis = j >= lo[r] && j <= end[r];
      const float sc = vis ? s[r] + bias : -INFINITY;
      const float mNew = fmaxf(m[r], warp_max(sc));
      const float corr = __expf(m[r] - mNew);
      const float pe = vis ? __expf(sc - mNew) : 0.f;
      l[r] = l[r] * corr + warp_sum(pe);
      m[r] = mNew;
      pr[r] = pe;
#pragma unroll
      for (int c = 0; c < NC; c++) acc[r][c] *= corr;
    }
    auto values = [&](auto guarded) {
      for (int jj = 0; jj < nk; jj++) {
        float pj[RPW];
#pragma unroll
        for (int r = 0; r < RPW; r++) pj[r] = __shfl_sync(0xffffffffu, pr[r], jj);
#pragma unroll
        for (int c = 0; c < NC; c++) {
          const float vv = sV[jj * vs + lane + 32 * c];
#pragma unroll
          for (int r = 0; r < RPW; r++)
            if (!decltype(guarded)::value || (k0 + jj >= lo[r] && k0 + jj <= end[r]))
              acc[r][c] = fmaf(pj[r], vv, acc[r][c]);
        }
      }
    };
    if (odd) values(std::true_type{});
    else values(std::false_type{});
  }

  T* __restrict__ out = static_cast<T*>(p.out);
  const int64_t qw = (int64_t)p.qHeads * hd;
#pragma unroll
  for (int r = 0; r < RPW; r++) {
    const int64_t row = row0 + warp * RPW + r;
    if (row >= p.qLen) continue;
    const float invL = l[r] > 0.f ? 1.f / l[r] : 0.f;  // empty band -> zeros
#pragma unroll
    for (int c = 0; c < NC; c++) {
      const int x = lane + 32 * c;
      if (x < hd) out[row * qw + (int64_t)h * hd + x] = from_f32<T>(acc[r][c] * invL);
    }
  }
}

template <typename T, int NC>
cudaError_t launch(const AttnParams& p, cudaStream_t s) {
  const int hd = p.hd;
  const size_t smem = sizeof(float) * ((size_t)hd * BQ + (size_t)BK * (hd | 1) + (size_t)BK * NC * 32);
  auto kern = prefill_rows_kernel<T, NC>;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  const int64_t tiles = (p.qLen + BQ - 1) / BQ;
  dim3 grid((unsigned)tiles, (unsigned)p.qHeads);
  kern<<<grid, WARPS * 32, smem, s>>>(p);
  return cudaGetLastError();
}

template <typename T>
cudaError_t dispatch_nc(const AttnParams& p, cudaStream_t s) {
  const int nc = (p.hd + 31) / 32;
  if (nc <= 1) return launch<T, 1>(p, s);
  if (nc <= 2) return launch<T, 2>(p, s);
  if (nc <= 4) return launch<T, 4>(p, s);
  if (nc <= 8) return launch<T, 8>(p, s);
  return launch<T, 16>(p, s);
}

}  // namespace

// Whether this kernel takes less time than the tile kernels (prefill_f32_tc.cu; prefill_simt.cu where that
// does not take the call).  Those give a sequence of a padded batch tiles of its own, so that one of two
// rows costs as much as one of 32, and score 64 or 128 keys at a time.  6000 rows of f32, 8 heads,
// sequences of 2 / 16 / 64 / 128, us, tiles and rows: heads of 32 779 / 105 / 69 / 61 and 27 / 26 / 40 / 63, of
// 128 1507 / 201 / 133 / 132 and 83 / 74 / 139 / 225, of 256 at sequences of 2 / 8 / 16 2138 / 562 / 307 and
// 335 / 334 / 309.  f16, heads of 80, 2 / 16 / 64: 812 / 126 / 90 and 54 / 50 / 87.  Where the blocks do not fill
// the chip, one block's time decides: four sequences, f32, heads of 64, of 16 7 and 9, of 40 17 and 9.
//
// The estimates, in us, are fitted to 1290 such pairs of up to 160 keys: here a block's chain of 32-key
// tiles, and every block's work over the chip; there waves of blocks, by head and keys.  Taking the smaller
// estimate cost 1.2 % over the better kernel on average, at worst four tenths of some 12 us.  Past 160 keys
// the tiles are the faster ones (32 segments of 250, 12 heads of 8: 178 and 229).
bool prefill_rows_better(const AttnParams& p, int dtype) {
  constexpr int64_t kSms = 148;
  int64_t seen = (int64_t)p.wl + p.wr + 1 < p.kvLen ? (int64_t)p.wl + p.wr + 1 : p.kvLen;   // by one row
  bool single = false;
  if (p.seqStride > 0) seen = seen < p.seqStride ? seen : p.seqStride;
  else if (p.segs && p.maxSegment > 0) seen = seen < p.maxSegment ? seen : p.maxSegment;
  else single = true;
  if (seen > 160) return false;
  const int64_t tiles = p.seqStride > 0 ? p.qLen / p.seqStride * ((p.seqStride + 31) / 32) : (p.qLen + 31) / 32;
  const int64_t blocks = tiles * p.qHeads;
  const bool tc = prefill_f32_tc_supported(p, dtype);
  // (one f32 sequence stays on the route that the header names for f32, 8 us for 5 where it is short,
  // unless there is much of it)
  if (tc && single && blocks <= 2 * kSms) return false;
  const double hd = p.hd, keys = (double)seen, rowBlocks = (double)((p.qLen + BQ - 1) / BQ * p.qHeads);
  // 32-key tiles of a 16-row block: sequences that are a multiple of its rows begin with it
  const bool aligned = p.seqStride > 0 && (p.seqStride % BQ == 0 || p.seqStride == p.qLen);
  const double mine = (double)((seen + (aligned ? 31 : 47)) / 32);
  const double chain = mine * (2.41 + 0.0899 * hd);
  const double work = 1e-3 * rowBlocks * (p.hd > 128 ? hd * hd * (8.62e-4 + 1.28e-3 * mine)
                                                     : 1.84 + 0.0721 * hd + mine * (0.822 + 0.115 * hd));
  const double rows = 0.5 + (chain > work ? chain + 0.47 * work : work + 0.47 * chain);
  const int padded = p.hd <= 32 ? 32 : p.hd <= 64 ? 64 : p.hd <= 128 ? 128 : 256;
  const int64_t atOnce = kSms * (tc ? (padded == 32 ? 2 : 1) : p.hd <= 64 ? 3 : p.hd <= 256 ? 2 : 1);
  const double waves = (double)((blocks + atOnce - 1) / atOnce);
  const double tile = tc ? 10.3 + 0.0125 * padded + keys * (0.0023 + 0.000054 * padded)
                         : 10.6 + 0.0219 * hd + keys * (0.013 + 0.00075 * hd);
  return rows < 0.4 + waves * tile;
}

cudaError_t launch_prefill_rows(const AttnParams& p, int dtype, cudaStream_t s) {
  return dtype == RT_F16 ? dispatch_nc<__half>(p, s) : dispatch_nc<float>(p, s);
}

}  // namespace rt
