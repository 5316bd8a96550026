// Tensor-core prefill attention with two softmax warpgroups taking alternate
// key tiles of one 128-row query tile.
//
// In the other two tensor-core kernels a query tile is one serial chain
// S(j) -> softmax -> P V(j) -> S(j+1): the tensor pipe idles while a tile's
// softmax runs, and a second chain on the same SM only fills part of that gap.
// Here S has two buffers in tensor memory and P has columns of its own, so
//   - the S issuer runs ahead: S(j+1) is computed while tile j is in the softmax,
//   - warpgroup g (warps 4g..4g+3) owns tiles j = g, g+2, ...: each tile still gets a
//     whole warpgroup (one thread per query row, 128 scores in registers), but two
//     tiles are in flight, which doubles the softmax rate the tensor pipe can be fed
//     from,
//   - the P V issuer accumulates O += P(j) V(j) in tile order as the halves of P arrive.
// The running maximum is shared by the two warpgroups through shared memory: the
// reference point of a row moves only when its maximum has grown by more than 2^13
// (rare after the first tile), and the "max phases" of consecutive tiles are
// ordered by a per-warp counter, so both warpgroups always exponentiate against
// the same reference point and the accumulator is rescaled by exactly one of them.
// Up to head size 128 a tile's exponentials start before its max phase, against the
// reference point last seen, and the maximum is gathered beside them; if the point has
// moved, what was computed is computed again before anything is published.  (At head size 256
// the one S buffer makes the order of the max phases matter more, and the maximum comes first.
// Through the operator, in turn with the version before the early exponentials, the cheaper
// waits, the output through shared memory and the grid order below: 64 x 8192 rows causal, 8 heads
// of 128, 9626 -> 9323 us, the power limit being what is left there; 32 sequences of 512..2048,
// 3 heads of 256 on one, +-512 window, 180 -> 156.)
//
// Head sizes: 64 and 128 (two S buffers), 256 (the accumulator takes half of tensor
// memory, so there is ONE S buffer — free again as soon as its scores are in a warpgroup's
// registers, which is when the next S is issued — beside the two P buffers; K arrives as
// two 128-column halves and V as two 64-key halves so that every ring slot is 32 KB and
// S keeps the full-rate 128-key tile), and the narrow heads 32, 36, 52, ... (any
// multiple of 4 up to 60) padded to 64 inside the tile: K and V tiles are fetched
// with a 64-column box that starts on the 16-byte boundary at or below the head
// (the columns beside the head belong to its neighbours), Q is staged by the
// softmax threads with zeros in those columns, so the neighbours' columns add
// nothing to the scores, and the output columns they produce are dropped.
//
// Pairs (head sizes 128 and 256).  Two CTAs of a cluster, on two SMs, take two adjacent
// 128-row query tiles of the same head and run every product as ONE tcgen05.mma of
// cta_group::2 (M = 256: 128 rows per CTA, each into its own tensor memory), issued by
// the even CTA.  The B operand of such a product is split between the two CTAs' shared
// memories — each holds 64 of a K tile's 128 keys, and half of a V tile's columns — so
// each SM fetches only half of every K/V tile from the L2 (that traffic is what limits
// this kernel: it burns power at head size 128 and its latency cannot be hidden behind
// one SM's 160 KB of tile buffers at head size 256) and its ring holds twice as many
// tiles.  Everything else is per CTA as described above; the odd CTA's MMA warps idle.
// The peer's loads report to the even CTA's barriers (the cta_group::2 form of the bulk
// tensor copy), its softmax warps arrive on them remotely, and the even CTA's commits
// arrive on both CTAs' barriers.  Every copy has one destination CTA.
//
// Semantics are the 'attn' op's (see rt_attn.h); replaces attnFlash
// (packages/runntime/src/core/kernels/attention/attnFlash.ts:93-276).  Every wait is
// bounded; a wait that runs out sets the status word and the CTA winds down through
// the common exit that frees its tensor memory.
#include "common.cuh"
#include "sm100.cuh"
#include "tc_common.cuh"

namespace rt {
namespace {

using namespace sm100;
using namespace tc;

constexpr int kThreads3 = 384;
constexpr int kRegsSoftmax3 = 216, kRegsOther3 = 64;  // 2*128*216 + 128*64 <= 384*168
constexpr int BK3 = 128;
constexpr int kMaxSlots = 12;

template <int HD, bool PAIR>
struct Cfg3 {
  static constexpr int CHUNKS = HD / 64;                       // 64-column chunks of a row
  static constexpr int Q_BYTES = BM * HD * 2;
  // One CTA alone at head size 256: K and V tiles arrive in two parts (K: 128 columns each,
  // V: 64 keys each) so that a ring slot is 32 KB.  A pair holds half tiles anyway.
  static constexpr bool SPLIT = HD == 256 && !PAIR;
  static constexpr int KP = SPLIT ? 2 : 1, VP = SPLIT ? 2 : 1;  // parts per key tile
  static constexpr int K_ROWS = PAIR ? BK3 / 2 : BK3;           // keys of a K tile held by this CTA
  static constexpr int K_CHUNKS = SPLIT ? 2 : CHUNKS;           // 64-column chunks in one K part
  static constexpr int V_ROWS = SPLIT ? 64 : BK3;               // keys in one V part
  static constexpr int V_CHUNKS = PAIR ? CHUNKS / 2 : CHUNKS;   // 64-column chunks of V held here
  static constexpr int K_BYTES = K_CHUNKS * K_ROWS * 128, V_BYTES = V_CHUNKS * V_ROWS * 128;
  static constexpr int SLOT_BYTES = K_BYTES > V_BYTES ? K_BYTES : V_BYTES;
  static constexpr int SLOTS_FIT = (225 * 1024 - Q_BYTES) / SLOT_BYTES;
  static constexpr int SLOTS = SLOTS_FIT > kMaxSlots ? kMaxSlots : SLOTS_FIT;
  static constexpr int SMEM = Q_BYTES + SLOTS * SLOT_BYTES + 1024;
  // Tensor memory: S | O | P up to head size 128 (two S buffers, 2 x 64 columns of P behind
  // the accumulator); at head size 256 the accumulator takes the upper half and one S buffer
  // shares the lower half with the two P buffers.
  static constexpr int S_BUFS = HD == 256 ? 1 : 2;
  static constexpr int O_COL = 2 * BK3;
  static constexpr int P_COL = HD == 256 ? BK3 : O_COL + 128;
  static constexpr int TMEM_COLS = 512;
  static constexpr int CTAS = PAIR ? 2 : 1;
  static_assert(SLOTS >= KP + VP + 1, "ring too small");
  static_assert(O_COL + HD <= TMEM_COLS, "tensor memory budget");
  static_assert(!PAIR || HD >= 128, "a pair splits V into 64-column chunks");
};

struct Barriers3 {
  uint64_t fullQ;
  uint64_t full[kMaxSlots], empty[kMaxSlots];
  uint64_t sFull[2], sFree[2], pReady[2][2], pvDone[2];
};

// Ring sequence numbers.  The producer issues K(0); then, for every tile j, K(j+1)
// (if there is one) and V(j): K runs one tile ahead of V.
template <int KP, int VP>
__device__ __forceinline__ int seq_k(int j) { return j == 0 ? 0 : KP + (j - 1) * (KP + VP); }
template <int KP, int VP>
__device__ __forceinline__ int seq_v(int j, int n) {
  return KP + j * (KP + VP) + (j + 1 < n ? KP : 0);
}

// ---- the cta_group::2 forms (a pair of CTAs on two SMs acting as one MMA unit) ----------

// In the shared window of a cluster, bit 24 of an address tells the two CTAs of a pair
// apart: cleared it names the even CTA's copy of the same location.
constexpr uint32_t kPeerBit = 1u << 24;

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrives on a barrier anywhere in the cluster (here: the even CTA's copy).  Default
// semantics (release at CTA scope): what the consumer reads — P in this CTA's tensor memory
// — is ordered by the tcgen05 fences around the arrival, and a cluster-scope release on
// every arrival costs the arriving warp about a thousand cycles (measured).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Tiled load into this CTA's shared memory whose completion is counted on the EVEN CTA's
// barrier at the same offset (the pair's MMA issuer waits there for both halves).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y,
                                                 uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], "
      "[%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(bar & ~kPeerBit)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dstSmem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dstSmem),
               "r"(cols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols)
               : "memory");
}
// Arrives once on the barrier at `bar`'s offset in each CTA of the pair when all MMAs issued
// so far by this thread have completed in both: one commit per CTA, the second one naming
// the odd CTA's copy of the barrier (measured: as fast as a single commit naming both).
__device__ __forceinline__ void tc_commit_one(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  tc_commit_one(bar);
  tc_commit_one(bar | kPeerBit);
}
__device__ __forceinline__ void mma_f16_ss_pair(uint32_t dTmem, uint64_t aDesc, uint64_t bDesc,
                                                uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dTmem),
      "l"(aDesc), "l"(bDesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_f16_ts_pair(uint32_t dTmem, uint32_t aTmem, uint64_t bDesc,
                                                uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(dTmem),
      "r"(aTmem), "l"(bDesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Instruction descriptor of a pair's product: M = 256 over the two CTAs.
constexpr uint32_t instr_desc_pair(int n, bool bMnMajor) {
  return (instr_desc(n, bMnMajor) & ~(0x1fu << 24)) | ((uint32_t)(256 >> 4) << 24);
}

// Waits (bounded) until the counter at `addr` has reached `want`; an acquire load pairs with the
// release store of the warp that moved it.  The lanes of the warp agree on the outcome.
__device__ __forceinline__ bool counter_poll_warp(uint32_t addr, int want, volatile int* abortFlag) {
  bool reached = false;
  for (int i = 0; i < (1 << 22); i++) {
    int v;
    asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    if (v >= want) {
      reached = true;
      break;
    }
    if ((i & 63) == 63 && *abortFlag) break;
  }
  return __all_sync(0xffffffffu, reached);
}

// First and last key that four of the 128 rows from `row0` on see (lane, lane + 32, ...;
// INT_MAX and -1 if none): row_band, with the loads of all four rows ahead of the first use
// and no branch between them (row by row, each load waiting for the branch before it, this took
// 2100 cycles at the start of every unit).
__device__ __forceinline__ void rows_range(const AttnParams& p, int64_t row0, int lane, int& first, int& last) {
  constexpr int kRows = BM / 32;
  int64_t s0[kRows], s1[kRows];
  if (p.segs) {
    float a[kRows], b[kRows];
#pragma unroll
    for (int i = 0; i < kRows; i++) {
      const int64_t row = min(row0 + lane + 32 * i, p.qLen - 1);
      a[i] = p.segs[2 * row];
      b[i] = p.segs[2 * row + 1];
    }
#pragma unroll
    for (int i = 0; i < kRows; i++) s0[i] = (int64_t)a[i], s1[i] = (int64_t)b[i] - 1;
  } else if (p.seqStride > 0) {
    int len[kRows];
#pragma unroll
    for (int i = 0; i < kRows; i++) {
      const uint32_t row = (uint32_t)min(row0 + lane + 32 * i, p.qLen - 1);   // (qLen is below 2^31)
      const uint32_t b = row / (uint32_t)p.seqStride;
      s0[i] = (int64_t)b * p.seqStride;
      len[i] = p.seqLens[b];
    }
#pragma unroll
    for (int i = 0; i < kRows; i++)
      s1[i] = row0 + lane + 32 * i - s0[i] < len[i] ? s0[i] + len[i] - 1 : -1;
  } else {
#pragma unroll
    for (int i = 0; i < kRows; i++) s0[i] = 0, s1[i] = p.kvLen - 1;
  }
  first = INT_MAX;
  last = -1;
#pragma unroll
  for (int i = 0; i < kRows; i++) {
    const int64_t row = row0 + lane + 32 * i, pos = p.qPosOffset + row;
    const int64_t lo = max(max(pos - p.wl, s0[i]), (int64_t)0);
    const int64_t end = min(min(pos + p.wr, s1[i]), p.kvLen - 1);
    if (row < p.qLen && lo <= end) first = min(first, (int)lo), last = max(last, (int)end);
  }
}

// PADDED: the head is narrower than the 64 columns the tile holds (see the file header);
// p.hd is the real size, `shift` = (kvh * hd) & 7 the head's first column inside the box.
// PAIR: two CTAs of a cluster share every K/V tile (see the file header).
template <int HD, bool PADDED, bool PAIR>
__global__ void __launch_bounds__(kThreads3, 1)
prefill_tc3_kernel(const __grid_constant__ CUtensorMap mapQ, const __grid_constant__ CUtensorMap mapK,
                   const __grid_constant__ CUtensorMap mapV, const __grid_constant__ CUtensorMap mapO,
                   const AttnParams p, int* status) {
  using C = Cfg3<HD, PAIR>;
  constexpr int BK = BK3, KP = C::KP, VP = C::VP, NS = C::SLOTS;
  static_assert(!PADDED || (HD == 64 && !PAIR), "narrow heads are padded to 64 columns, one CTA");
  extern __shared__ unsigned char smemRaw[];
  __shared__ Barriers3 bars;
  __shared__ uint32_t sTmemBase;
  __shared__ int sAbort;
  __shared__ int sLoMin[8], sEndMax[8];   // a pair's range of keys, by warp
  __shared__ int sUnit[2];                // one CTA alone: first key tile and number of key tiles
  __shared__ float sMref[BM];          // the rows' reference points (log2 domain)
  __shared__ float sL[2][BM];          // the warpgroups' row sums, for the epilogue
  __shared__ volatile int sMaxDone[4];  // per warp of a warpgroup: tiles whose max phase is over

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  TC_TRACE_DECL
  // Long rows first under a causal mask; the two CTAs of a pair take adjacent row tiles.
  const int cta = PAIR ? (int)cluster_ctarank() : 0;
  // One CTA alone: the query heads that share a kv head are neighbours in the grid, so that a K
  // or V tile comes from memory once for all of them: 4 causal sequences of 4096 rows, 3 heads of
  // 256 on one, 101 -> 91.5 us; 8 of 512..2048 rows both ways 53.5 -> 49.2; in a window of +-512
  // the tiles are few and it is even.  One query head per kv head takes no division: with it, 8
  // heads of 128 x 8192 rows took 269 us for 262.
  int unit = (int)(gridDim.x / C::CTAS) - 1 - (int)(blockIdx.x / C::CTAS);
  int h = blockIdx.y, kvh = h;
  if (p.qHeads != p.kvHeads) {
    const int group = p.qHeads / p.kvHeads;
    if constexpr (PAIR) {
      kvh = h / group;
    } else {
      const int fromEnd = (int)(gridDim.x - 1 - blockIdx.x);
      unit = fromEnd / group;
      h = h * group + fromEnd - unit * group;
      kvh = blockIdx.y;
    }
  }
  const int qTile = unit * C::CTAS + cta;
  const bool leader = cta == 0;
  const int64_t row0 = (int64_t)qTile * BM;
  const int hd = PADDED ? p.hd : HD;
  const int shift = PADDED ? ((kvh * hd) & 7) : 0;

  const uint32_t smemBase = (smem_u32(smemRaw) + 1023u) & ~1023u;
  const uint32_t sQ = smemBase;
  const uint32_t sRing = sQ + C::Q_BYTES;

  const int xKV = PADDED ? ((kvh * hd) & ~7) : kvh * HD;

  // One CTA alone: the producer warp works the unit's key range out by itself (four rows per
  // lane) and starts the copies of Q and of the first K tile before the rest of the set-up —
  // tensor memory, the rows' bands — instead of after the barrier that ends it: the first S of
  // a unit at head size 128 is there 4340 cycles after the block's start, 5020 before (of 24000
  // for nine key tiles).
  if (!PAIR && warp == 8) {
    if (lane == 0) {
      if (!PADDED) prefetch_tensormap(&mapQ);
      prefetch_tensormap(&mapK);
      prefetch_tensormap(&mapV);
      mbar_init(smem_u32(&bars.fullQ), 1);
      for (int s = 0; s < kMaxSlots; s++) {
        mbar_init(smem_u32(&bars.full[s]), 1);
        mbar_init(smem_u32(&bars.empty[s]), 1);
      }
      fence_barrier_init();
    }
    grid_dependency_wait();
    int wl, we;
    rows_range(p, row0, lane, wl, we);
    wl = __reduce_min_sync(0xffffffffu, wl);
    we = __reduce_max_sync(0xffffffffu, we);
    if (lane == 0) {
      const int first = we >= 0 ? wl / BK : 0;
      sUnit[0] = first;
      sUnit[1] = we >= 0 ? we / BK - first + 1 : 0;
      if (we >= 0) {   // (in a padded batch the units past a sequence's end ask for nothing)
        if (!PADDED) {
          mbar_expect_tx(smem_u32(&bars.fullQ), C::Q_BYTES);
          for (int c = 0; c < C::CHUNKS; c++)
            tma_load_2d(sQ + c * (BM * 128), &mapQ, h * HD + c * 64, (int)row0, smem_u32(&bars.fullQ));
        }
        for (int part = 0; part < KP; part++) {
          mbar_expect_tx(smem_u32(&bars.full[part]), C::K_BYTES);
          for (int c = 0; c < C::K_CHUNKS; c++)
            tma_load_2d(sRing + part * C::SLOT_BYTES + c * (C::K_ROWS * 128), &mapK,
                        xKV + (part * C::K_CHUNKS + c) * 64, first * BK, smem_u32(&bars.full[part]));
        }
      }
    }
    __syncwarp();
  }
  if (tid == 0) {
    sAbort = 0;
    if (PAIR) {
      mbar_init(smem_u32(&bars.fullQ), 1);
      for (int s = 0; s < kMaxSlots; s++) {
        mbar_init(smem_u32(&bars.full[s]), 1);
        mbar_init(smem_u32(&bars.empty[s]), 1);
      }
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(smem_u32(&bars.sFull[b]), 1);
      // one arrival per warp of the warpgroup — of both CTAs' warpgroups in a pair, whose
      // arrivals all go to the even CTA, where the MMA issuers wait
      mbar_init(smem_u32(&bars.sFree[b]), 4 * C::CTAS);
      mbar_init(smem_u32(&bars.pReady[b][0]), 4 * C::CTAS);
      mbar_init(smem_u32(&bars.pReady[b][1]), 4 * C::CTAS);
      mbar_init(smem_u32(&bars.pvDone[b]), 1);
    }
    fence_barrier_init();
  }
  if (warp == 9) {
    if (PAIR) {
      tmem_alloc_pair(smem_u32(&sTmemBase), C::TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(smem_u32(&sTmemBase), C::TMEM_COLS);
      tmem_relinquish();
    }
  }

  // Band of this thread's row.  The two CTAs of a pair walk the same key tiles, so each works
  // the range out for both — warps 0-3 from its own rows, warps 4-7 from the other CTA's.
  const int rowInTile = tid & 127;
  int lo = 1, end = 0;  // empty
  if (warp < 8 || PAIR) grid_dependency_wait();   // (the producer has waited by itself where it loads before here)
  if (warp < 8) {
    // Q of a narrow head by hand: 16-byte units of the swizzled K-major layout, the head's
    // columns at [shift, shift + hd), zeros beside them and in rows past the end.  A head
    // starts on four elements of the tile, so a unit is two quads that are inside or outside
    // as a whole; they are read as such (as pairs where q's rows start on four bytes only),
    // all of a thread's before the first is used: element by element, after the barrier, this
    // took 4000 of a unit's 26000 cycles (head size 52, nine key tiles).
    constexpr int kUnits = PADDED ? BM * 8 / 256 : 1;
    uint2 v[kUnits][2];
    if (PADDED) {
      const __half* qg = static_cast<const __half*>(p.q) + (int64_t)h * hd;
      const bool quads = (reinterpret_cast<uintptr_t>(p.q) & 7u) == 0 && p.qStride % 4 == 0;
      auto load = [&](auto read) {
#pragma unroll
        for (int i = 0; i < kUnits; i++) {
          const int u = tid + 256 * i, c0 = (u & 7) * 8 - shift;
          const int64_t row = row0 + (u >> 3);
#pragma unroll
          for (int e = 0; e < 2; e++) {
            const int c = c0 + 4 * e;
            v[i][e] = make_uint2(0u, 0u);
            if (row < p.qLen && c >= 0 && c < hd) v[i][e] = read(qg + row * p.qStride + c);
          }
        }
      };
      if (quads) load([](const __half* src) { return *reinterpret_cast<const uint2*>(src); });
      else
        load([](const __half* src) {
          const uint32_t* w = reinterpret_cast<const uint32_t*>(src);
          return make_uint2(w[0], w[1]);
        });
    }
    const int64_t row = row0 + rowInTile;
    if (row < p.qLen) {
      int64_t l64, e64;
      row_band(p, row, l64, e64);
      if (l64 <= e64) {
        lo = (int)l64;
        end = (int)e64;
      }
    }
    if (PADDED) {
#pragma unroll
      for (int i = 0; i < kUnits; i++) {
        const int u = tid + 256 * i, r = u >> 3;
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sQ + r * 128 + (((u & 7) ^ (r & 7)) << 4)),
                     "r"(v[i][0].x), "r"(v[i][0].y), "r"(v[i][1].x), "r"(v[i][1].y)
                     : "memory");
      }
      fence_proxy_async();  // generic-proxy stores -> visible to the tensor core after the barrier
    }
    if (PAIR) {
      int olo = lo, oend = end;   // the row this thread contributes to the pair's range
      if (warp >= 4) {
        const int64_t other = (int64_t)(unit * 2 + (1 - cta)) * BM + rowInTile;
        olo = 1, oend = 0;
        if (other < p.qLen) {
          int64_t l64, e64;
          row_band(p, other, l64, e64);
          if (l64 <= e64) olo = (int)l64, oend = (int)e64;
        }
      }
      const int wl = __reduce_min_sync(0xffffffffu, olo <= oend ? olo : INT_MAX);
      const int we = __reduce_max_sync(0xffffffffu, olo <= oend ? oend : -1);
      if (lane == 0) {
        sLoMin[warp] = wl;
        sEndMax[warp] = we;
      }
    }
    if (warp < 4) {
      if (lane == 0) sMaxDone[warp] = 0;
      sMref[rowInTile] = p.sinks ? p.sinks[h] : kNegSeed;  // sinks arrive in the log2 domain
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (PAIR) cluster_sync_all();   // both CTAs' barriers exist before either is signalled from afar
  tc_fence_after_sync();
  TC_TRACE(99, 0);
  const uint32_t tmem = sTmemBase;
  int kt0, nTiles;
  if (PAIR) {
    int tileLo = INT_MAX, tileEnd = -1;
#pragma unroll
    for (int w8 = 0; w8 < 8; w8++) {
      tileLo = min(tileLo, sLoMin[w8]);
      tileEnd = max(tileEnd, sEndMax[w8]);
    }
    kt0 = tileEnd >= 0 ? tileLo / BK : 0;
    nTiles = tileEnd >= 0 ? tileEnd / BK - kt0 + 1 : 0;
  } else {
    kt0 = sUnit[0];
    nTiles = sUnit[1];
  }

  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther3));
    if (warp == 8) {
      // ------------------------------ TMA producer ------------------------------
      // In a pair every CTA loads its own Q tile and its halves of the K/V tiles into its
      // own ring (which both CTAs walk in step: same sequence numbers, same slots); all
      // completions are counted on the even CTA's barriers, where the byte counts expected
      // are the pair's.
      if (lane == 0 && nTiles > 0) {
        auto load = [&](uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
          if (PAIR) tma_load_2d_pair(dst, map, x, y, bar);
          else tma_load_2d(dst, map, x, y, bar);
        };
        if (PAIR) {
          prefetch_tensormap(&mapQ);
          prefetch_tensormap(&mapK);
          prefetch_tensormap(&mapV);
          if (leader) mbar_expect_tx(smem_u32(&bars.fullQ), C::CTAS * C::Q_BYTES);
          for (int c = 0; c < C::CHUNKS; c++)
            load(sQ + c * (BM * 128), &mapQ, h * HD + c * 64, (int)row0, smem_u32(&bars.fullQ));
        }
        int seq = PAIR ? 0 : KP;   // (one CTA alone: K(0) is on its way)
        bool ok = true;
        auto slot_for = [&](int& slot) {  // claims the next ring slot, waiting for its release
          slot = seq % NS;
          if (seq >= NS) ok = mbar_poll(smem_u32(&bars.empty[slot]), ((seq / NS) - 1) & 1, &sAbort);
          seq++;
          return ok;
        };
        auto load_k = [&](int j) {
          const int key0 = (kt0 + j) * BK + cta * C::K_ROWS;   // a pair: 64 keys each
          for (int part = 0; part < KP && ok; part++) {
            int slot;
            if (!slot_for(slot)) return;
            const uint32_t bar = smem_u32(&bars.full[slot]), dst = sRing + slot * C::SLOT_BYTES;
            if (leader) mbar_expect_tx(bar, C::CTAS * C::K_BYTES);
            for (int c = 0; c < C::K_CHUNKS; c++)
              load(dst + c * (C::K_ROWS * 128), &mapK, xKV + (part * C::K_CHUNKS + c) * 64, key0, bar);
          }
        };
        auto load_v = [&](int j) {
          const int key0 = (kt0 + j) * BK;
          const int x0 = xKV + cta * C::V_CHUNKS * 64;          // a pair: half of the columns each
          for (int part = 0; part < VP && ok; part++) {
            int slot;
            if (!slot_for(slot)) return;
            const uint32_t bar = smem_u32(&bars.full[slot]), dst = sRing + slot * C::SLOT_BYTES;
            if (leader) mbar_expect_tx(bar, C::CTAS * C::V_BYTES);
            for (int c = 0; c < C::V_CHUNKS; c++)
              load(dst + c * (C::V_ROWS * 128), &mapV, x0 + c * 64, key0 + part * C::V_ROWS, bar);
          }
        };
        if (PAIR) load_k(0);
        for (int j = 0; j < nTiles && ok; j++) {
          if (j + 1 < nTiles) load_k(j + 1);
          if (ok) load_v(j);
        }
        if (!ok) sAbort = 1;
      }
    } else if (warp == 9 && leader) {
      // ------------------------------ MMA issuer: S = Q K^T ----------------------
      // The whole warp walks the loop (waits included); the tensor-core instructions
      // run in one elected lane, which keeps their operands in uniform registers.
      if (nTiles > 0) {
        constexpr uint32_t idescS = PAIR ? instr_desc_pair(BK, false) : instr_desc(BK, false);
        constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);  // SBO, version, SW128
        constexpr uint32_t kLboK = (16u >> 4) << 16;
        auto desc = [](uint32_t lo32) { return ((uint64_t)kDescHi << 32) | lo32; };
        auto wait = [&](uint64_t* bar, int parity) {
          return mbar_poll_warp(smem_u32(bar), (uint32_t)parity, &sAbort);
        };
        // descriptors carry the 18-bit offset inside the CTA's window, not the CTA's rank bits
        const uint32_t aLo = ((sQ & 0x3ffffu) >> 4) | kLboK;
        const int kSteps = PADDED ? (shift + hd + 15) / 16 : HD / 16;  // K = 16 per instruction
        bool ok = PADDED || wait(&bars.fullQ, 0);   // (a narrow head's Q was staged before the barrier)
#pragma unroll 1
        for (int j = 0; j < nTiles && ok; j++) {
          const int b = j & 1;
          const uint32_t sBuf = C::S_BUFS == 2 ? b * BK : 0;
          const int s0 = seq_k<KP, VP>(j);
          TC_TRACE(10, j);
#pragma unroll
          for (int part = 0; part < KP; part++) {
            const int slot = (s0 + part) % NS;
            ok = wait(&bars.full[slot], ((s0 + part) / NS) & 1);
            // The S buffer is free once its previous contents are in the registers of the
            // warpgroup that took them: S(j-2) with two buffers, S(j-1) with one.
            if (ok && part == 0 && j >= C::S_BUFS) {
              const int jp = j - C::S_BUFS;
              ok = wait(&bars.sFree[jp & 1], (jp >> 1) & 1);
            }
            if (!ok) break;
            tc_fence_after_sync();
            TC_TRACE(11, j);
            if (elect_one()) {
              const uint32_t bLo = (((sRing + slot * C::SLOT_BYTES) & 0x3ffffu) >> 4) | kLboK;
              constexpr int kPerPart = C::K_CHUNKS * 4;  // K = 16 steps in one part
#pragma unroll
              for (int k2 = 0; k2 < kPerPart; k2++) {
                const int kk = part * kPerPart + k2;
                if (PADDED && k2 >= kSteps) break;
                const uint32_t aOff = (kk >> 2) * ((BM * 128) >> 4) + (kk & 3) * 2;
                const uint32_t bOff = (k2 >> 2) * ((C::K_ROWS * 128) >> 4) + (k2 & 3) * 2;
                if (PAIR) mma_f16_ss_pair(tmem + sBuf, desc(aLo + aOff), desc(bLo + bOff), idescS, kk > 0);
                else mma_f16_ss(tmem + sBuf, desc(aLo + aOff), desc(bLo + bOff), idescS, kk > 0);
              }
              if (PAIR) {
                tc_commit_pair(smem_u32(&bars.empty[slot]));
                if (part == KP - 1) tc_commit_pair(smem_u32(&bars.sFull[b]));
              } else {
                tc_commit(smem_u32(&bars.empty[slot]));
                if (part == KP - 1) tc_commit(smem_u32(&bars.sFull[b]));
              }
            }
            __syncwarp();
            TC_TRACE(12, j);
          }
        }
        if (!ok) sAbort = 1;
      }
    } else if (warp == 10 && leader) {
      // ------------------------------ MMA issuer: O += P V ------------------------
      if (nTiles > 0) {
        constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
        constexpr uint32_t kLboV = ((uint32_t)(C::V_ROWS * 128) >> 4) << 16;  // next 64 columns of hd
        auto desc = [](uint32_t lo32) { return ((uint64_t)kDescHi << 32) | lo32; };
        auto wait = [&](uint64_t* bar, int parity) {
          return mbar_poll_warp(smem_u32(bar), (uint32_t)parity, &sAbort);
        };
        const uint32_t idescO = PAIR ? instr_desc_pair(HD, true)
                                     : instr_desc(PADDED ? ((shift + hd + 15) & ~15) : HD, true);
        bool ok = true;
#pragma unroll 1
        for (int j = 0; j < nTiles && ok; j++) {
          const int b = j & 1;
          const int s0 = seq_v<KP, VP>(j, nTiles);
          const uint32_t pCol = tmem + C::P_COL + b * 64;
#pragma unroll
          for (int half = 0; half < 2; half++) {
            const int part = VP == 2 ? half : 0;
            const int slot = (s0 + part) % NS;
            TC_TRACE(13 + 3 * half, j);
            if (VP == 2 || half == 0) ok = wait(&bars.full[slot], ((s0 + part) / NS) & 1);
            TC_TRACE(14 + 3 * half, j);
            if (ok) ok = wait(&bars.pReady[b][half], (j >> 1) & 1);
            if (!ok) break;
            tc_fence_after_sync();
            TC_TRACE(15 + 3 * half, j);
            if (elect_one()) {
              const uint32_t bLo = (((sRing + slot * C::SLOT_BYTES) & 0x3ffffu) >> 4) | kLboV;
#pragma unroll
              for (int k2 = 0; k2 < 4; k2++) {
                const int kk = half * 4 + k2;              // 16 keys per step
                const int kLocal = VP == 2 ? k2 : kk;       // within this part's rows
                const uint32_t acc = (j > 0 || kk > 0) ? 1u : 0u;
                if (PAIR) mma_f16_ts_pair(tmem + C::O_COL, pCol + kk * 8, desc(bLo + kLocal * (2048 >> 4)), idescO, acc);
                else mma_f16_ts(tmem + C::O_COL, pCol + kk * 8, desc(bLo + kLocal * (2048 >> 4)), idescO, acc);
              }
              if (PAIR) {
                if (half == 1) {
                  tc_commit_pair(smem_u32(&bars.empty[slot]));
                  tc_commit_pair(smem_u32(&bars.pvDone[b]));
                }
              } else {
                if (VP == 2 || half == 1) tc_commit(smem_u32(&bars.empty[slot]));
                if (half == 1) tc_commit(smem_u32(&bars.pvDone[b]));
              }
            }
            __syncwarp();
          }
        }
        if (!ok) sAbort = 1;
      }
    }
  } else {
    // ------------------------------ softmax + epilogue ------------------------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax3));
    const int g = warp >> 2, w = warp & 3;
    const uint32_t laneBase = (uint32_t)(w * 32) << 16;
    const uint32_t sCol = tmem + laneBase + (C::S_BUFS == 2 ? g * BK : 0);
    const uint32_t pCol = tmem + laneBase + C::P_COL + g * 64;
    const uint32_t oCol = tmem + laneBase + C::O_COL;
    // where the MMA issuers wait for this warp: this CTA, or the even CTA of the pair
    auto arrive = [&](uint64_t* bar) {
      if (PAIR && !leader) mbar_arrive_cluster(smem_u32(bar) & ~kPeerBit);
      else mbar_arrive(smem_u32(bar));
    };
    bool ok = true;

    float seen = p.sinks ? p.sinks[h] : kNegSeed;  // the reference point this thread's l is relative to
    float l = (p.sinks && g == 0) ? 1.f : 0.f;
#pragma unroll 1
    for (int j = g; j < nTiles && ok; j += 2) {
      const int key0 = (kt0 + j) * BK;
      TC_TRACE(0, j);
      ok = mbar_poll_warp(smem_u32(&bars.sFull[g]), (j >> 1) & 1, &sAbort);
      if (!ok) break;  // the whole warp leaves together
      tc_fence_after_sync();
      TC_TRACE(1, j);
      uint32_t sv[BK];
#pragma unroll
      for (int c = 0; c < BK; c += 32)
        tmem_ld32(sCol + c, *reinterpret_cast<uint32_t(*)[32]>(&sv[c]));
      tmem_wait_ld();
      TC_TRACE(2, j);
      // S(j) is in registers: its buffer may take the next S
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) arrive(&bars.sFree[g]);
      TC_TRACE(20, j);
      const bool fullTile = lo <= key0 && end >= key0 + BK - 1;
      if (p.hasKeyBias) {
        const int b0 = p.biasStart - key0, b1 = p.biasEnd - key0;
#pragma unroll
        for (int c = 0; c < BK; c++) {
          const float s = __uint_as_float(sv[c]);
          sv[c] = __float_as_uint((c >= b0 && c < b1) ? s + p.biasValue : s);
        }
      }
      if (!fullTile) {
        // visible columns of this row are the interval [c0, c0 + span]
        const int c0 = lo <= end ? lo - key0 : (1 << 30);
        const unsigned span = lo <= end ? (unsigned)(end - lo) : 0u;
#pragma unroll
        for (int c = 0; c < BK; c++)
          sv[c] = ((unsigned)(c - c0) <= span) ? sv[c] : 0xff800000u;  // -inf
      }
      // Row maximum: four independent chains of 3-input max, gathered while the special-
      // function unit works on the first half's exponentials.
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      float2 sum2[4];
      uint32_t pk[32];
      auto foldMax = [&](int c) {  // columns c .. c+7
#pragma unroll
        for (int u = 0; u < 4; u++)
          mx4[u] = max3(mx4[u], __uint_as_float(sv[c + 2 * u]), __uint_as_float(sv[c + 2 * u + 1]));
      };
      auto clearSums = [&]() {
#pragma unroll
        for (int u = 0; u < 4; u++) sum2[u] = make_float2(0.f, 0.f);
      };
      auto expHalf = [&](int half, bool withMax) {
        const float2 scale2 = make_float2(kLog2e, kLog2e), shift2 = make_float2(-seen, -seen);
#pragma unroll
        for (int c = 0; c < 64; c += 2) {
          const int cc = half * 64 + c;
          const float2 t = fma2(make_float2(__uint_as_float(sv[cc]), __uint_as_float(sv[cc + 1])),
                                scale2, shift2);
          const float2 pe = exp2_pair(t, c >> 1);
          sum2[(c >> 1) & 3] = add2(sum2[(c >> 1) & 3], pe);
          const __half2 hp = __floats2half2_rn(pe.x, pe.y);
          pk[c / 2] = *reinterpret_cast<const uint32_t*>(&hp);
          if (withMax && (c & 3) == 0) foldMax(2 * c);  // 16 steps x 8 columns = all 128
        }
      };
      clearSums();
      // The exponentials of a warpgroup's first tile wait for a reference point; later tiles
      // start against the one last seen, and the half is computed again if it has moved.
      const bool early = HD < 256 && j > 1;
      if (early) {
        expHalf(0, true);
      } else {
#pragma unroll
        for (int c = 0; c < BK; c += 8) foldMax(c);
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * kLog2e;
      TC_TRACE(21, j);

      // ---- max phase, in tile order across the two warpgroups ----
      if (j > 0) {
        // (an acquire load pairs with the release store below: what the other warpgroup's
        // warp wrote before it — reference points, its rescale of O — is visible after it)
        ok = counter_poll_warp(smem_u32(const_cast<int*>(&sMaxDone[w])), j, &sAbort);
        if (!ok) break;
        tc_fence_after_sync();
      }
      TC_TRACE(22, j);
      float mref = sMref[rowInTile];
      const bool grow = mx > mref + kRescaleThreshold;
      if (__any_sync(0xffffffffu, grow || mref != seen || !early)) {
        if (mref != seen) {  // the other warpgroup moved the reference point since this one last looked
          l *= fast_exp2(seen - mref);
          seen = mref;
        }
        if (__any_sync(0xffffffffu, grow)) {
          // A row whose reference point is still the seed has seen no key in any tile so far:
          // its accumulator row is exactly zero and needs no pass (the rows of a band's first,
          // partly masked tile meet their first keys in the second one).  When only such rows
          // have grown, they alone move; the pass over O, when there is one, moves every row.
          const bool pass = j > 0 && __any_sync(0xffffffffu, grow && mref != kNegSeed);
          const float mnew = (pass || j == 0 || mref == kNegSeed) ? fmaxf(mref, mx) : mref;
          const float f = fast_exp2(mref - mnew);
          if (pass) {
            // O holds the tiles up to j-1 once P V(j-1) has landed (the products complete in order)
            ok = mbar_poll_warp(smem_u32(&bars.pvDone[(j - 1) & 1]), ((j - 1) >> 1) & 1, &sAbort);
            if (!ok) break;
            tc_fence_after_sync();
            constexpr int oCols = PADDED ? 64 : HD;
#pragma unroll
            for (int c = 0; c < oCols; c += 32) {
              tmem_ld32(oCol + c, pk);
              tmem_wait_ld();
#pragma unroll
              for (int x = 0; x < 32; x++) pk[x] = __float_as_uint(__uint_as_float(pk[x]) * f);
              tmem_st32(oCol + c, pk);
            }
            tmem_wait_st();
            tc_fence_before_sync();
          }
          l *= f;
          mref = seen = mnew;
          sMref[rowInTile] = mnew;
        }
        clearSums();
        __syncwarp();
        if (lane == 0)
          asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(
                           smem_u32(const_cast<int*>(&sMaxDone[w]))),
                       "r"(j + 1)
                       : "memory");
        expHalf(0, false);
      } else if (lane == 0) {
        asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(
                         smem_u32(const_cast<int*>(&sMaxDone[w]))),
                     "r"(j + 1)
                     : "memory");
      }
      TC_TRACE(3, j);

      // ---- P in two halves ----
      // P's own columns were last read by P V(j-2).
      if (j >= 2) {
        ok = mbar_poll_warp(smem_u32(&bars.pvDone[g]), ((j >> 1) - 1) & 1, &sAbort);
        if (!ok) break;
      }
      TC_TRACE(6, j);
      auto publish = [&](int half) {
        tmem_st32(pCol + half * 32, pk);
        tmem_wait_st();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) arrive(&bars.pReady[g][half]);
        TC_TRACE(4 + half, j);
      };
      publish(0);
      expHalf(1, false);
      publish(1);
      const float2 s01 = add2(add2(sum2[0], sum2[1]), add2(sum2[2], sum2[3]));
      l += s01.x + s01.y;
    }

    if (!ok) sAbort = 1;

    // ---- epilogue: both warpgroups, half of the output columns each ----
    // (every softmax thread passes the barriers, also after a failed wait)
    named_barrier_sync(2, 256);
    {
      const float mfin = sMref[rowInTile];
      if (mfin != seen) l *= fast_exp2(seen - mfin);
      sL[g][rowInTile] = l;
    }
    named_barrier_sync(2, 256);
    l = sL[0][rowInTile] + sL[1][rowInTile];
    // The unit's rows go out through the Q tile's shared memory, which the last S has left:
    // one bulk tensor store per 64 columns (rows past the end are outside the map), or, for
    // a narrow head, whose columns start on eight bytes, quads in the order of memory.  A
    // thread that stores its own row sends each piece of 32 bytes to another row's sectors:
    // 2000 cycles a unit at head size 128, 3500 at 256, 3900 in 4-byte pieces at 52.
    bool good = ok && !sAbort;
    if (nTiles > 0) {
      if (good) {
        good = mbar_poll(smem_u32(&bars.pvDone[(nTiles - 1) & 1]), ((nTiles - 1) >> 1) & 1, &sAbort);
        if (!good) sAbort = 1;
      }
      good = __all_sync(0xffffffffu, good);
      if (good) {
        tc_fence_after_sync();
        const float invL = (l > 0.f && lo <= end) ? 1.f / l : 0.f;  // a row that saw no key: zeros
        constexpr int perGroup = (PADDED ? 64 : HD) / 2;
#pragma unroll
        for (int c = 0; c < perGroup; c += 32) {
          const int col = g * perGroup + c;
          uint32_t o[32];
          tmem_ld32(oCol + col, o);
          tmem_wait_ld();
          uint32_t wds[16];
#pragma unroll
          for (int x = 0; x < 32; x += 2) {
            const __half2 hp = __floats2half2_rn(__uint_as_float(o[x]) * invL,
                                                 __uint_as_float(o[x + 1]) * invL);
            wds[x / 2] = *reinterpret_cast<const uint32_t*>(&hp);
          }
          if (PADDED) {
            const uint32_t base = sQ + rowInTile * (hd * 2);
#pragma unroll
            for (int x = 0; x < 32; x += 4) {
              const int at = col + x - shift;   // a quad is inside the head or outside as a whole
              if (at >= 0 && at < hd)
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(base + at * 2), "r"(wds[x / 2]),
                             "r"(wds[x / 2 + 1])
                             : "memory");
            }
          } else {
            const uint32_t base = sQ + (col >> 6) * (BM * 128) + rowInTile * 128;
#pragma unroll
            for (int v = 0; v < 4; v++)
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(
                               base + (((((col & 63) >> 3) + v) ^ (rowInTile & 7)) << 4)),
                           "r"(wds[4 * v]), "r"(wds[4 * v + 1]), "r"(wds[4 * v + 2]), "r"(wds[4 * v + 3])
                           : "memory");
          }
        }
        if (!PADDED) fence_proxy_async();
      }
      // At head sizes of 128 and more a warpgroup stores the chunks it has written itself.
      constexpr bool own = !PADDED && HD >= 128;
      if (own) named_barrier_sync(3 + g, 128);
      else named_barrier_sync(2, 256);
      if (!PADDED && good && w == 0 && (own || g == 0) && elect_one()) {
        constexpr int chunks = own ? C::CHUNKS / 2 : C::CHUNKS;
#pragma unroll
        for (int c = 0; c < chunks; c++) {
          const int chunk = (own ? g * chunks : 0) + c;
          tma_store_2d(&mapO, sQ + chunk * (BM * 128), h * HD + chunk * 64, (int)row0);
        }
        bulk_commit();
        bulk_wait_read<0>();
      }
    }
    if (PADDED && good) {
      // (zeros where no row of the unit sees a key)
      __half* base = static_cast<__half*>(p.out) + (int64_t)h * hd;
      const int64_t pitch = (int64_t)p.qHeads * hd;
      const bool quads = (reinterpret_cast<uintptr_t>(p.out) & 7u) == 0;
      const int perRow = hd / 4;
      for (int u = tid; u < BM * perRow; u += 256) {
        const int r = u / perRow, c = (u - r * perRow) * 4;
        if (row0 + r < p.qLen) {
          uint2 v = make_uint2(0u, 0u);
          if (nTiles > 0)
            asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(sQ + u * 8));
          __half* dst = base + (row0 + r) * pitch + c;
          if (quads) {
            *reinterpret_cast<uint2*>(dst) = v;
          } else {
            reinterpret_cast<uint32_t*>(dst)[0] = v.x;
            reinterpret_cast<uint32_t*>(dst)[1] = v.y;
          }
        }
      }
    } else if (nTiles == 0) {
      // No row of this unit sees a key (in a padded batch: every unit past a sequence's end):
      // 16-byte stores, consecutive threads on consecutive pieces of a row.
      constexpr int kPerRow = HD / 8;
      __half* base = static_cast<__half*>(p.out) + row0 * ((int64_t)p.qHeads * HD) + (int64_t)h * HD;
      for (int i = tid; i < BM * kPerRow; i += 256) {
        const int r = i / kPerRow, c = i - r * kPerRow;
        if (row0 + r < p.qLen)
          reinterpret_cast<uint4*>(base + (int64_t)r * p.qHeads * HD)[c] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
  }

  // Common exit: every role arrives here, then the allocating warp frees TMEM.  In a pair
  // neither CTA leaves while the other may still read its shared memory or signal it.
  tc_fence_before_sync();
  __syncthreads();
  if (PAIR) cluster_sync_all();
  if (tid == 0 && sAbort) atomicOr(status, kStatusWaitTimeout);
  if (warp == 9) {
    tc_fence_after_sync();
    if (PAIR) tmem_dealloc_pair(tmem, C::TMEM_COLS);
    else tmem_dealloc(tmem, C::TMEM_COLS);
  }
}

template <int HD, bool PADDED, bool PAIR>
cudaError_t launch3(const AttnParams& p, int* status, cudaStream_t s, std::string* err) {
  using C = Cfg3<HD, PAIR>;
  CUtensorMap mq, mk, mv, mo;
  // The narrow-head form reads Q with plain loads; its K/V maps span the real columns,
  // so a box that runs past the last head reads zeros there.
  const int64_t qCols = (int64_t)p.qHeads * p.hd, kvCols = (int64_t)p.kvHeads * p.hd;
  if ((!PADDED && !make_map(&mq, p.q, p.qLen, qCols, p.qStride, BM, err)) ||
      !make_map(&mk, p.k, p.kvLen, kvCols, p.kvStride, C::K_ROWS, err) ||
      !make_map(&mv, p.v, p.kvLen, kvCols, p.kvStride, C::V_ROWS, err))
    return cudaErrorInvalidValue;
  if (PADDED) mq = mo = mk;  // unused by the kernel; valid maps all the same
  else if (!make_map(&mo, p.out, p.qLen, qCols, qCols, BM, err)) return cudaErrorInvalidValue;
  auto kern = prefill_tc3_kernel<HD, PADDED, PAIR>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
  if (e != cudaSuccess) return e;
  const unsigned tiles = (unsigned)((p.qLen + BM - 1) / BM);
  cudaLaunchConfig_t cfg{};
  const unsigned group = PAIR ? 1u : (unsigned)(p.qHeads / p.kvHeads);
  cfg.gridDim = dim3((tiles + C::CTAS - 1) / C::CTAS * C::CTAS * group, (unsigned)p.qHeads / group);
  cfg.blockDim = dim3(kThreads3);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C::CTAS;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = PAIR ? attr : attr + 1;
  cfg.numAttrs = PAIR ? 2 : 1;
  e = cudaLaunchKernelEx(&cfg, kern, mq, mk, mv, mo, p, status);
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

bool prefill_tc3_supported(const AttnParams& p, int dtype) {
  if (dtype != RT_F16) return false;
  const bool wide = p.hd == 64 || p.hd == 128 || p.hd == 256;
  const bool narrow = p.hd >= 4 && p.hd <= 60 && p.hd % 4 == 0;
  if (!wide && !narrow) return false;
  if (p.qLen < 2 || p.qLen >= (1ll << 31) - 256 || p.kvLen >= (1ll << 31) - 256) return false;
  auto al = [](const void* ptr, uintptr_t a) { return (reinterpret_cast<uintptr_t>(ptr) & (a - 1)) == 0; };
  // TMA: 16-byte aligned bases and row pitches (Q of a narrow head is read with plain
  // loads and written back in 4-byte pairs)
  if (!al(p.k, 16) || !al(p.v, 16) || (p.kvStride * 2) % 16) return false;
  if (wide && (!al(p.q, 16) || !al(p.out, 16) || (p.qStride * 2) % 16)) return false;
  if (narrow && (!al(p.q, 4) || !al(p.out, 4) || p.qStride % 2)) return false;
  if (!encode_fn()) return false;
  return true;
}

// Pairs of CTAs need two row tiles of the same head and one of the head sizes whose V tile
// splits into 64-column chunks.
bool prefill_tc3_pair_supported(const AttnParams& p, int dtype) {
  return prefill_tc3_supported(p, dtype) && (p.hd == 128 || p.hd == 256) && p.qLen > BM;
}

cudaError_t launch_prefill_tc3(const AttnParams& p, bool pair, int* status, cudaStream_t s,
                               std::string* err) {
  if (pair) {
    return p.hd == 128 ? launch3<128, false, true>(p, status, s, err)
                       : launch3<256, false, true>(p, status, s, err);
  }
  switch (p.hd) {
    case 64: return launch3<64, false, false>(p, status, s, err);
    case 128: return launch3<128, false, false>(p, status, s, err);
    case 256: return launch3<256, false, false>(p, status, s, err);
  }
  return launch3<64, true, false>(p, status, s, err);
}

}  // namespace rt
