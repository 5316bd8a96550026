// f32 prefill attention on the tensor cores (mma.sync, tf32), head sizes up to 256 that are a
// multiple of four, rows that start on 16 bytes; prefill_rows.cu takes batches of short sequences,
// prefill_simt.cu everything else.
//
// Every f32 operand x is split into hi + lo, each a tf32 number (11 bits): x = hi + lo to 2^-23, and
// a product is hi hi' + hi lo' + lo hi', 2^-22 short of exact at worst.  The tensor core adds into its
// accumulator less carefully than an FMA does, so no accumulator lives long: scores add 32 columns of
// the head before they join the f32 sum (hi hi' apart from the 2^-11 smaller cross terms), and 16 keys
// are added, their cross terms first, before they join the f32 output.  Against 64-bit
// products: 4.2e-7 to 4.8e-7 of the norm at head size 256 (1.5e-6 to 1.7e-6 for sequential f32 sums),
// 1.9e-7 to 3.0e-7 below (2.4e-7 to 9.1e-7).
//
// A CTA of eight warps owns 32 query rows of one query head and walks 128-key tiles of the union of
// its rows' bands.  For the scores a warp takes all rows and 16 of the keys, for the output all
// rows and 32 of the columns (of some of the keys, where the head has fewer than eight times 32): so
// every element of K and V is split by one warp only, for six MMAs each.  The probabilities go
// through shared memory, split once, in the order of the MMA's operands; so does q.  K comes in chunks
// of 128 keys x 32 columns and V in chunks of 16 keys per warp through a ring that cp.async fills.
//
// Why not prefill_simt.cu: two-wide FMAs with three different operands run at 48 of the
// 73 TFLOP/s, tf32 MMAs at 275, 92 in threes.
// What bounds it: instructions and latency with two warps per scheduler (8.7 instructions per MMA, the
// MMA pipe 32 % of active cycles), and the last row tiles; at head sizes up to 32 also the registers, 128 for
// two CTAs per SM, of which 356 bytes a thread spill.  8 sequences of 92..484 rows, 3 heads of
// 256 on one K/V head (2.4 GFLOP, 27 us at 92 TFLOP/s): 583 us for 16-row tiles of scalar FMAs, 155
// for prefill_simt.cu, 102 here.
//
// A product with an infinity or a NaN is NaN here (tf32.cuh), where the op's definition may have an
// infinite score that weighs nothing: a row tile with a row sum or an output that is not finite
// is computed again by whole f32 products.
#include "common.cuh"
#include "exact_row.cuh"
#include "sm100.cuh"
#include "tf32.cuh"

namespace rt {
namespace {

constexpr int BQ = 32, BK = 128, kWarps = 8, kThreads = 32 * kWarps;
constexpr int kDims = 32;                               // head columns per K chunk
// Sequences that are put in order of length.  Each block looks at all of them, and with many the launch has
// blocks enough to end evenly without: 8 heads of 32, 250 sequences of 24 rows in order 165 us, 300 of 20
// as they come 86.
constexpr int kMaxOrdered = 64;

template <int HDP>  // head size rounded up to 32, 64, 128 or 256
struct F32Tc {
  static constexpr int kColSets = HDP / 32, kKeySets = kWarps / kColSets;  // of the warps, for the output
  static constexpr int kVRows = 16 * kKeySets, kVChunks = BK / kVRows;
  // A quarter warp's 16-byte loads are two keys x 16 columns of K and four keys (every second one)
  // x two pieces of V: these pitches give them distinct banks.
  static constexpr int kKPitch = kDims + 16, kVPitch = HDP + 4;
  static constexpr int kStage = BK * kKPitch > kVRows * kVPitch ? BK * kKPitch : kVRows * kVPitch;  // floats
  static constexpr int kStages = HDP <= 64 ? 2 : 5;
  static constexpr int kQ = BQ * HDP * 2, kP = BQ * BK * 2;   // hi and lo
  static constexpr int kSmem = 4 * (kQ + kP + kStages * kStage);
  static constexpr int kCtas = HDP == 32 ? 2 : 1;             // per SM
  static_assert((kKeySets - 1) * BQ * HDP <= kStages * kStage, "the other key sets' rows fit the ring");
};

// Which row tile block number u of a padded batch takes: the tiles of the longest sequence first
// (its last rows first: under a causal mask they are the longest), those past the sequences' ends
// last.  The blocks run in about this order, so the long ones do not meet at the end
// of the launch.  Every thread of the block calls it.
__device__ __forceinline__ void ordered_tile(const AttnParams& p, int64_t u, int tilesPerSeq, int* sLen,
                                             int64_t* sTile) {
  const int batch = (int)(p.qLen / p.seqStride), tid = threadIdx.x;
  if (tid < batch) sLen[tid] = min(max(p.seqLens[tid], 0), p.seqStride);
  __syncthreads();
  if (tid < batch) {
    const int mine = sLen[tid], used = (mine + BQ - 1) / BQ;
    int before = 0, free = 0, all = 0;       // tiles of longer sequences; unused ones of those ahead
#pragma unroll 8
    for (int b = 0; b < batch; b++) {
      const int len = sLen[b], t = (len + BQ - 1) / BQ;
      all += t;
      if (len > mine || (len == mine && b < tid)) before += t;
      if (b < tid) free += tilesPerSeq - t;
    }
    if (u >= before && u < before + used) *sTile = (int64_t)tid * tilesPerSeq + used - 1 - (u - before);
    const int64_t e = u - all;               // past the used ones
    if (e >= free && e < free + tilesPerSeq - used) *sTile = (int64_t)tid * tilesPerSeq + used + (e - free);
  }
  __syncthreads();
}

template <int HDP>
__global__ void __launch_bounds__(kThreads, F32Tc<HDP>::kCtas)
prefill_f32_tc_kernel(const AttnParams p, int tilesPerSeq) {
  using S = F32Tc<HDP>;
  grid_dependency_wait();
  extern __shared__ __align__(16) float smem[];
  uint4* sQ = reinterpret_cast<uint4*>(smem);         // [16-column block][row set][hi g, hi g+8, lo g, lo g+8][lane]
  uint4* sP = reinterpret_cast<uint4*>(smem + S::kQ); // [8-key block][row set][hi, lo][lane]
  float* ring = smem + S::kQ + S::kP;                 // [kStages][kStage]
  __shared__ int64_t sLo[BQ], sEnd[BQ], sTile;
  __shared__ int sLen[kMaxOrdered];
  __shared__ float sMax[kWarps][BQ], sSum[kWarps][BQ];

  const int hd = p.hd;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int colSet = warp % S::kColSets, keySet = warp / S::kColSets;
  const int g = lane >> 2, t4 = lane & 3;    // fragment row and column
  const int h = (int)(blockIdx.x % (unsigned)p.qHeads);
  const int64_t u = blockIdx.x / (unsigned)p.qHeads;
  int64_t tile = (int64_t)(gridDim.x / (unsigned)p.qHeads) - 1 - u;   // later rows first, as in a sequence
  // In a padded batch a tile stays inside its sequence.
  int64_t row0 = tile * BQ, rowEnd = p.qLen;
  if (p.seqStride > 0) {
    if (p.qLen / p.seqStride <= kMaxOrdered) {
      ordered_tile(p, u, tilesPerSeq, sLen, &sTile);
      tile = sTile;
    }
    const int64_t b = tile / tilesPerSeq;
    row0 = b * p.seqStride + (tile - b * tilesPerSeq) * BQ;
    rowEnd = min((b + 1) * p.seqStride, row0 + BQ);
  }
  rowEnd = min(rowEnd, row0 + BQ);
  const int kvh = h / (p.qHeads / p.kvHeads);
  const float* __restrict__ q = static_cast<const float*>(p.q) + (int64_t)h * hd;
  const float* __restrict__ k = static_cast<const float*>(p.k) + (int64_t)kvh * hd;
  const float* __restrict__ v = static_cast<const float*>(p.v) + (int64_t)kvh * hd;
  float* __restrict__ out = static_cast<float*>(p.out) + (int64_t)h * hd;
  const int64_t outPitch = (int64_t)p.qHeads * hd;

  bool seen = false;
  if (tid < BQ) {
    int64_t lo = 1, end = 0;
    if (row0 + tid < rowEnd) row_band(p, row0 + tid, lo, end);
    sLo[tid] = lo;
    sEnd[tid] = end;
    seen = lo <= end;
  }
  if (!__syncthreads_or(seen)) {   // rows that see nothing: zeros
    for (int i = tid; i < BQ * (hd / 4); i += kThreads) {
      const int r = i / (hd / 4), x = (i - r * (hd / 4)) * 4;
      if (row0 + r < rowEnd) *reinterpret_cast<float4*>(out + (row0 + r) * outPitch + x) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    return;
  }
  int64_t tileLo = INT64_MAX, tileEnd = -1;     // keys some row of the CTA sees
#pragma unroll 8
  for (int r = 0; r < BQ; r++) {
    if (sLo[r] <= sEnd[r]) {
      tileLo = min(tileLo, sLo[r]);
      tileEnd = max(tileEnd, sEnd[r]);
    }
  }
  const int span = (int)(tileEnd - tileLo + 1);   // keys from here on relative to tileLo
  const int tiles = (span + BK - 1) / BK;
  const int kChunks = (hd + kDims - 1) / kDims, perTile = kChunks + S::kVChunks;

  int fillTile = 0, fillPart = 0, fillStage = 0;
  auto fill = [&]() {
    if (fillTile < tiles) {
      float* dst = ring + fillStage * S::kStage;
      const int k0 = fillTile * BK;
      if (fillPart < kChunks) {
        constexpr int W = kDims / 4;
        const int x = fillPart * kDims + (tid % W) * 4;
        const float* src = k + (tileLo + k0 + tid / W) * p.kvStride + x;
        dst += (tid / W) * S::kKPitch + (tid % W) * 4;
#pragma unroll
        for (int i = 0; i < BK * W / kThreads; i++) {
          const bool in = k0 + tid / W + i * (kThreads / W) < span && x < hd;   // zeros past the last key and column
          copy_async16(dst + i * (kThreads / W) * S::kKPitch, in ? src + i * (kThreads / W) * p.kvStride : k, in);
        }
      } else {
        constexpr int W = HDP / 4;
        const int x = (tid % W) * 4, r = k0 + (fillPart - kChunks) * S::kVRows + tid / W;
        const float* src = v + (tileLo + r) * p.kvStride + x;
        dst += (tid / W) * S::kVPitch + x;
#pragma unroll
        for (int i = 0; i < S::kVRows * W / kThreads; i++) {
          const bool in = r + i * (kThreads / W) < span && x < hd;
          copy_async16(dst + i * (kThreads / W) * S::kVPitch, in ? src + i * (kThreads / W) * p.kvStride : v, in);
        }
      }
      if (++fillPart == perTile) fillPart = 0, fillTile++;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");   // one group per chunk, empty ones at the end
    if (++fillStage == S::kStages) fillStage = 0;
  };
  int useStage = 0;
  // The next chunk has arrived for everyone, and everyone is done with the one before it,
  // whose place is filled again.
  auto advance = [&]() -> const float* {
    asm volatile("cp.async.wait_group %0;" ::"n"(S::kStages - 2) : "memory");
    __syncthreads();
    const float* at = ring + useStage * S::kStage;
    fill();
    if (++useStage == S::kStages) useStage = 0;
    return at;
  };
  for (int i = 0; i < S::kStages - 1; i++) fill();

  for (int i = tid; i < BQ * HDP / 4; i += kThreads) {
    // piece i: four columns of one row, for lane (row & 7, piece & 3)
    const int r = i / (HDP / 4), x4 = i % (HDP / 4);
    float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row0 + r < rowEnd && 4 * x4 < hd) f = *reinterpret_cast<const float4*>(q + (row0 + r) * p.qStride + 4 * x4);
    uint4 hi, lo;
    split(f.x, hi.x, lo.x), split(f.y, hi.y, lo.y), split(f.z, hi.z, lo.z), split(f.w, hi.w, lo.w);
    uint4* dst = sQ + (((x4 >> 2) * 2 + (r >> 4)) * 4 + ((r >> 3) & 1)) * 32 + (r & 7) * 4 + (x4 & 3);
    dst[0] = hi;
    dst[64] = lo;
  }

  // Rows 16 a + g + 8 i of this lane: band, running maximum, this lane's share of the row sum.
  int lo[2][2], end[2][2];
  float m[2][2], l[2][2];
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int r = 16 * a + g + 8 * i;
      const bool any = sLo[r] <= sEnd[r];
      lo[a][i] = any ? (int)(sLo[r] - tileLo) : 1;
      end[a][i] = any ? (int)(sEnd[r] - tileLo) : 0;
      m[a][i] = p.sinks ? p.sinks[h] * 0.6931471805599453f : kNegSeed;
      l[a][i] = p.sinks && warp == 0 && t4 == 0 ? 1.f : 0.f;
    }
  // o[a][j]: rows 16 a + g (0, 1) and + 8 (2, 3), columns 32 colSet + 8 t4 + j and 4 further on
  float o[2][4][4];
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int e = 0; e < 4; e++) o[a][j][e] = 0.f;

  for (int t = 0; t < tiles; t++) {
    const int key0 = t * BK + warp * 16;        // this warp's sixteen keys
    const bool live = key0 < span;

    // ---- scores of rows 16 a + g, + 8 and keys key0 + 8 n + 2 t4, + 1 ----
    float s[2][2][4], cross[2][2][4];
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
      for (int n = 0; n < 2; n++)
#pragma unroll
        for (int e = 0; e < 4; e++) s[a][n][e] = cross[a][n][e] = 0.f;
#pragma unroll 1
    for (int c = 0; c < kChunks; c++) {
      const float* sK = advance() + (warp * 16 + g) * S::kKPitch + 4 * t4;
      if (!live) continue;
      float d[2][2][4];
#pragma unroll
      for (int b = 0; b < kDims / 16; b++) {
        uint32_t kh[2][4], kl[2][4];
#pragma unroll
        for (int n = 0; n < 2; n++) {
          const float4 f = *reinterpret_cast<const float4*>(sK + n * 8 * S::kKPitch + 16 * b);
          split(f.x, kh[n][0], kl[n][0]), split(f.y, kh[n][1], kl[n][1]);
          split(f.z, kh[n][2], kl[n][2]), split(f.w, kh[n][3], kl[n][3]);
        }
#pragma unroll
        for (int a = 0; a < 2; a++) {
          const uint4* fq = sQ + ((c * (kDims / 16) + b) * 2 + a) * 128 + lane;
          const uint4 h0 = fq[0], h1 = fq[32], l0 = fq[64], l1 = fq[96];
          // column t4 of a step's operands is column 4 t4 (+ 2 in the second step) of the head,
          // column t4 + 4 the one after it
          const uint32_t hi[2][4] = {{h0.x, h1.x, h0.y, h1.y}, {h0.z, h1.z, h0.w, h1.w}};
          const uint32_t lw[2][4] = {{l0.x, l1.x, l0.y, l1.y}, {l0.z, l1.z, l0.w, l1.w}};
#pragma unroll
          for (int st = 0; st < 2; st++)
#pragma unroll
            for (int n = 0; n < 2; n++) {
              if (b == 0 && st == 0) mma_tf32_first(d[a][n], hi[st], kh[n][2 * st], kh[n][2 * st + 1]);
              else mma_tf32(d[a][n], hi[st], kh[n][2 * st], kh[n][2 * st + 1]);
              mma_tf32(cross[a][n], hi[st], kl[n][2 * st], kl[n][2 * st + 1]);
              mma_tf32(cross[a][n], lw[st], kh[n][2 * st], kh[n][2 * st + 1]);
            }
        }
      }
#pragma unroll
      for (int a = 0; a < 2; a++)
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int e = 0; e < 4; e++) s[a][n][e] += d[a][n][e];
    }

    // ---- online softmax over the tile ----
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
      for (int i = 0; i < 2; i++) {
        float mx = -INFINITY;
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const int key = key0 + 8 * n + 2 * t4 + e;
            float& x = s[a][n][2 * i + e];
            x += cross[a][n][2 * i + e];
            if (p.hasKeyBias && tileLo + key >= p.biasStart && tileLo + key < p.biasEnd) x += p.biasValue;
            if (key >= lo[a][i] && key <= end[a][i]) mx = fmaxf(mx, x);
          }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        if (t4 == 0) sMax[warp][16 * a + g + 8 * i] = mx;
      }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 2; a++) {
      uint32_t ph[2][4], pl[2][4];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        float mNew = m[a][i];
#pragma unroll
        for (int w = 0; w < kWarps; w++) mNew = fmaxf(mNew, sMax[w][16 * a + g + 8 * i]);
        const float corr = __expf(m[a][i] - mNew);
        m[a][i] = mNew;
        float sum = 0.f;
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const int key = key0 + 8 * n + 2 * t4 + e;
            const float pe = key >= lo[a][i] && key <= end[a][i] ? __expf(s[a][n][2 * i + e] - mNew) : 0.f;
            sum += pe;
            // operand columns t4 and t4 + 4 are keys 2 t4 and 2 t4 + 1
            split(pe, ph[n][i + 2 * e], pl[n][i + 2 * e]);
          }
        l[a][i] = l[a][i] * corr + sum;
#pragma unroll
        for (int j = 0; j < 4; j++) o[a][j][2 * i] *= corr, o[a][j][2 * i + 1] *= corr;
      }
#pragma unroll
      for (int n = 0; n < 2; n++) {
        uint4* dst = sP + (((warp * 2 + n) * 2 + a) * 2) * 32 + lane;
        dst[0] = make_uint4(ph[n][0], ph[n][1], ph[n][2], ph[n][3]);
        dst[32] = make_uint4(pl[n][0], pl[n][1], pl[n][2], pl[n][3]);
      }
    }

    // ---- output ----
#pragma unroll 1
    for (int c = 0; c < S::kVChunks; c++) {
      const float* sV = advance() + (keySet * 16 + 2 * t4) * S::kVPitch + 32 * colSet + 4 * g;
      const int block = c * S::kKeySets + keySet;   // sixteen keys of the tile
      if (t * BK + block * 16 >= span) continue;
      uint32_t ph[2][2][4], pl[2][2][4];   // [8 keys][row set]
      float ev[2][2][4];                   // [8 keys][key 2 t4, 2 t4 + 1]
#pragma unroll
      for (int n = 0; n < 2; n++) {
        const uint4* fp = sP + (block * 2 + n) * 128 + lane;
#pragma unroll
        for (int a = 0; a < 2; a++) {
          *reinterpret_cast<uint4*>(ph[n][a]) = fp[64 * a];
          *reinterpret_cast<uint4*>(pl[n][a]) = fp[64 * a + 32];
          *reinterpret_cast<float4*>(ev[n][a]) = *reinterpret_cast<const float4*>(sV + (n * 8 + a) * S::kVPitch);
        }
      }
      float f[2][4][4];
      // MMA column g of tile j is column 4 g + j of the warp's 32; the small products first
#pragma unroll
      for (int j = 0; j < 4; j++) {
        uint32_t vh[2][2], vl[2][2];
#pragma unroll
        for (int n = 0; n < 2; n++) split(ev[n][0][j], vh[n][0], vl[n][0]), split(ev[n][1][j], vh[n][1], vl[n][1]);
#pragma unroll
        for (int a = 0; a < 2; a++) {
          mma_tf32_first(f[a][j], pl[0][a], vh[0][0], vh[0][1]);
          mma_tf32(f[a][j], ph[0][a], vl[0][0], vl[0][1]);
          mma_tf32(f[a][j], pl[1][a], vh[1][0], vh[1][1]);
          mma_tf32(f[a][j], ph[1][a], vl[1][0], vl[1][1]);
          mma_tf32(f[a][j], ph[0][a], vh[0][0], vh[0][1]);
          mma_tf32(f[a][j], ph[1][a], vh[1][0], vh[1][1]);
        }
      }
#pragma unroll
      for (int a = 0; a < 2; a++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
          for (int e = 0; e < 4; e++) o[a][j][e] += f[a][j][e];
    }
  }

  // ---- row sums over the warps, outputs over the key sets ----
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int i = 0; i < 2; i++) {
      l[a][i] += __shfl_xor_sync(0xffffffffu, l[a][i], 1);
      l[a][i] += __shfl_xor_sync(0xffffffffu, l[a][i], 2);
      if (t4 == 0) sSum[warp][16 * a + g + 8 * i] = l[a][i];
    }
  __syncthreads();          // ... and everyone is done with the ring
  if constexpr (S::kKeySets > 1) {
    float4* box = reinterpret_cast<float4*>(ring) + colSet * 32 + lane;
    constexpr int kSet = 8 * S::kColSets * 32;
    if (keySet > 0) {
#pragma unroll
      for (int i = 0; i < 8; i++)
        box[(keySet - 1) * kSet + i * S::kColSets * 32] =
            make_float4(o[i / 4][i % 4][0], o[i / 4][i % 4][1], o[i / 4][i % 4][2], o[i / 4][i % 4][3]);
    }
    __syncthreads();
    if (keySet == 0) {
#pragma unroll
      for (int w = 0; w < S::kKeySets - 1; w++)
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const float4 f = box[w * kSet + i * S::kColSets * 32];
          o[i / 4][i % 4][0] += f.x, o[i / 4][i % 4][1] += f.y, o[i / 4][i % 4][2] += f.z, o[i / 4][i % 4][3] += f.w;
        }
    }
  }
  bool odd = false;         // something that is not finite
  if (keySet == 0) {
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int r = 16 * a + g + 8 * i;
        float sum = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; w++) sum += sSum[w][r];
        const float invL = sum > 0.f ? 1.f / sum : 0.f;  // empty band -> zeros
        odd |= !(sum < INFINITY);   // (1 / sum is not asked for a NaN sum, and 0 leaves nothing of it)
#pragma unroll
        for (int half = 0; half < 2; half++) {
          const int x = 32 * colSet + 8 * t4 + 4 * half, e = 2 * i + half;
          const float4 f = make_float4(o[a][0][e] * invL, o[a][1][e] * invL, o[a][2][e] * invL, o[a][3][e] * invL);
          if (row0 + r < rowEnd && x < hd) {
            odd |= !(fabsf(f.x) + fabsf(f.y) + fabsf(f.z) + fabsf(f.w) < INFINITY);
            *reinterpret_cast<float4*>(out + (row0 + r) * outPitch + x) = f;
          }
        }
      }
  }
  if (__syncthreads_or(odd)) {
    for (int r = warp; r < BQ; r += kWarps)
      if (row0 + r < rowEnd) exact_row<float>(p, row0 + r, h, sLo[r], sEnd[r]);
  }
}

template <int HDP>
cudaError_t launch(const AttnParams& p, cudaStream_t s) {
  auto kern = prefill_f32_tc_kernel<HDP>;
  constexpr int smem = F32Tc<HDP>::kSmem;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const int64_t perSeq = p.seqStride > 0 ? (p.seqStride + BQ - 1) / BQ : 0;
  const int64_t tiles = p.seqStride > 0 ? p.qLen / p.seqStride * perSeq : (p.qLen + BQ - 1) / BQ;
  return launch_dependent(kern, dim3((unsigned)(tiles * p.qHeads)), dim3(kThreads), smem, s, p, (int)perSeq);
}

}  // namespace

bool prefill_f32_tc_supported(const AttnParams& p, int dtype) {
  const uintptr_t bases = reinterpret_cast<uintptr_t>(p.q) | reinterpret_cast<uintptr_t>(p.k) |
                          reinterpret_cast<uintptr_t>(p.v) | reinterpret_cast<uintptr_t>(p.out);
  return dtype == RT_F32 && p.hd <= 256 && p.hd % 4 == 0 && p.qStride % 4 == 0 && p.kvStride % 4 == 0 &&
         bases % 16 == 0 && p.kvLen < (1ll << 30) && p.qLen * p.qHeads < (1ll << 30);
}

cudaError_t launch_prefill_f32_tc(const AttnParams& p, cudaStream_t s) {
  if (p.hd <= 32) return launch<32>(p, s);
  if (p.hd <= 64) return launch<64>(p, s);
  if (p.hd <= 128) return launch<128>(p, s);
  return launch<256>(p, s);
}

}  // namespace rt
