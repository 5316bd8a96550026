// Single-token decode attention over KV caches: bandwidth-bound split-KV.
//
// Grid = (key splits, sequences, head blocks).  A CTA streams its slice of one
// sequence's K and V cache rows through a shared-memory ring filled by bulk
// async copies (TMA, 16-byte aligned, whole rows so every DRAM sector fetched is
// used), issued by a producer warp and signalled through mbarriers.  The 256
// consumer threads are laid out as (key slot, query head): each thread runs a
// private online softmax over the keys of its slot in f32 registers.  At the
// end the slots of a head are merged with a log-sum-exp; with more than one
// split the per-split (m, l, acc) partials go to scratch and the last CTA to
// arrive for the sequence merges them, without waiting, or, where they are more than
// one CTA reads in a few microseconds, a second launch does (see plan_decode).
//
// f16 caches with several query heads per kv head, or many wide heads and few keys, are read by
// eight warps on the tensor cores instead (decode_mma_kernel).
//
// The KV-cache append is fused: the new K/V row is stored to the cache by the
// CTA of split 0 and attended to straight from its source.
//
// Replaces packages/runntime/src/core/kernels/attention/attnDecode.ts:81-187
// (decode), :263-424 (decodeSplit + merge) and the writeRows dispatches that
// precede them (packages/runntime/src/core/kernels/shape/rows.ts:143-162).
#include <mutex>

#include "common.cuh"
#include "sm100.cuh"

namespace rt {
namespace {

using namespace sm100;

// Optional per-CTA timeline for kernel development (off unless the translation unit is
// compiled with RT_DEC_TRACE): thread 0 of every CTA stores the global timer at a few points.
#ifdef RT_DEC_TRACE
constexpr int kDecTraceCtas = 8192, kDecTracePoints = 8;
__device__ unsigned long long gDecTrace[kDecTraceCtas * kDecTracePoints];
#define DEC_TRACE(i)                                                                        \
  do {                                                                                      \
    if (threadIdx.x == 0) {                                                                 \
      const unsigned id_ = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;  \
      if (id_ < kDecTraceCtas) {                                                            \
        unsigned long long t_;                                                              \
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_));                              \
        gDecTrace[id_ * kDecTracePoints + (i)] = t_;                                        \
      }                                                                                     \
    }                                                                                       \
  } while (0)
#else
#define DEC_TRACE(i) \
  do {               \
  } while (0)
#endif

constexpr int kConsumers = 256;
constexpr int kConsumerWarps = kConsumers / 32;
constexpr int kMaxStages = 8;
// Heads up to 64 wide fit two CTAs per SM (registers and shared memory), so that one
// CTA's set-up, pipeline fill and merge overlap the other's streaming; wider heads get
// the whole SM.
constexpr size_t kSmemBudget = 200 * 1024;
constexpr size_t kSmemBudgetTwoPerSm = 108 * 1024;
constexpr size_t kSmemBudgetMma = 220 * 1024;   // three stages of 16 keys, 8 heads of 128

__host__ __device__ constexpr int q_stride(int hdp) { return ((hdp / 4) & 1) ? hdp : hdp + 4; }

template <typename T, int VEC>
struct Loader;

// 8 halves per 16-byte load
template <>
struct Loader<__half, 8> {
  static __device__ __forceinline__ void load(const __half* p, float (&f)[8]) {
    const uint4 w = *reinterpret_cast<const uint4*>(p);
    const __half2* h = reinterpret_cast<const __half2*>(&w);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const float2 t = __half22float2(h[i]);
      f[2 * i] = t.x;
      f[2 * i + 1] = t.y;
    }
  }
};
template <>
struct Loader<__half, 4> {
  static __device__ __forceinline__ void load(const __half* p, float (&f)[4]) {
    const uint2 w = *reinterpret_cast<const uint2*>(p);
    const __half2* h = reinterpret_cast<const __half2*>(&w);
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const float2 t = __half22float2(h[i]);
      f[2 * i] = t.x;
      f[2 * i + 1] = t.y;
    }
  }
};
template <>
struct Loader<float, 4> {
  static __device__ __forceinline__ void load(const float* p, float (&f)[4]) {
    const float4 w = *reinterpret_cast<const float4*>(p);
    f[0] = w.x; f[1] = w.y; f[2] = w.z; f[3] = w.w;
  }
};
template <typename T>
struct Loader<T, 1> {
  static __device__ __forceinline__ void load(const T* p, float (&f)[1]) { f[0] = to_f32<T>(*p); }
};

// Rows whose pitch is a multiple of 128 bytes (head size 64 or 128) put the same column of
// every key into the same bank: threads that walk their rows in step would collide on every
// load (eight ways for 16-byte loads; measured 1.0 TB/s at head size 128).  Such a thread
// starts at chunk `rot` of its row and wraps around instead: a dot product does not care
// about the order, q is fetched from the same rotated position, and the accumulator keeps
// its chunks in rotated order until it is written out (acc chunk i = row chunk
// (i + rot) mod chunks).
template <int HDP, bool EXACT, int VEC>
struct Rotated {
  static constexpr bool value = EXACT && VEC > 1 && (HDP == 64 || HDP == 128);
};

// One key for one head: score, online-softmax update, accumulate p*v.
// kp/vp may point at shared memory (cache tile) or global memory (appended row).
template <typename T, int HDP, bool EXACT, int VEC, bool QSMEM>
__device__ __forceinline__ void process_key(const T* kp, const T* vp, const float* qv, int hd,
                                            float& m, float& l, float (&acc)[HDP], int rot) {
  constexpr bool ROT = Rotated<HDP, EXACT, VEC>::value;
  constexpr int NCH = HDP / VEC;
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
  for (int i = 0; i < HDP / VEC; i++) {
    if (EXACT || i * VEC < hd) {
      const int ci = ROT ? ((i + rot) & (NCH - 1)) : i;
      float f[VEC];
      Loader<T, VEC>::load(kp + ci * VEC, f);
      if (ROT) {
        // q chunk from the same position: 16-byte loads (the q rows are 16-byte aligned)
        float qf[VEC];
#pragma unroll
        for (int e = 0; e < VEC; e += 4) {
          const float4 t = *reinterpret_cast<const float4*>(qv + ci * VEC + e);
          qf[e] = t.x, qf[e + 1] = t.y, qf[e + 2] = t.z, qf[e + 3] = t.w;
        }
#pragma unroll
        for (int e = 0; e < VEC; e += 4) {
          s0 = fmaf(qf[e], f[e], s0);
          s1 = fmaf(qf[e + 1], f[e + 1], s1);
          s2 = fmaf(qf[e + 2], f[e + 2], s2);
          s3 = fmaf(qf[e + 3], f[e + 3], s3);
        }
      } else {
#pragma unroll
        for (int e = 0; e < VEC; e++) {
          if ((i * VEC + e) & 1) s1 = fmaf(qv[i * VEC + e], f[e], s1);
          else s0 = fmaf(qv[i * VEC + e], f[e], s0);
        }
      }
    }
  }
  const float s = ((s0 + s1) + (s2 + s3)) * kLog2e;  // log2 domain
  if (s > m) {
    const float c = fast_exp2(m - s);
    l *= c;
#pragma unroll
    for (int x = 0; x < HDP; x++) acc[x] *= c;
    m = s;
  }
  const float pe = fast_exp2(s - m);
  l += pe;
#pragma unroll
  for (int i = 0; i < HDP / VEC; i++) {
    if (EXACT || i * VEC < hd) {
      const int ci = ROT ? ((i + rot) & (NCH - 1)) : i;
      float f[VEC];
      Loader<T, VEC>::load(vp + ci * VEC, f);
#pragma unroll
      for (int e = 0; e < VEC; e++) acc[i * VEC + e] = fmaf(pe, f[e], acc[i * VEC + e]);
    }
  }
}

// Two keys of one head at once (heads without a rotation: 36 and 52 columns): q is read once for
// both, and their two dot products and updates are independent instruction streams, which a block
// alone on its SM has too few warps to do without.
template <typename T, int HDP, int VEC>
__device__ __forceinline__ void process_two(const T* ka, const T* va, const T* kb, const T* vb, const float* qv,
                                            float& m, float& l, float (&acc)[HDP]) {
  static_assert(VEC == 4, "q in pieces of four");
  float a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
#pragma unroll
  for (int i = 0; i < HDP / VEC; i++) {
    float fa[VEC], fb[VEC];
    Loader<T, VEC>::load(ka + i * VEC, fa);
    Loader<T, VEC>::load(kb + i * VEC, fb);
    const float4 q = *reinterpret_cast<const float4*>(qv + i * VEC);
    a0 = fmaf(q.x, fa[0], a0), a1 = fmaf(q.y, fa[1], a1), a0 = fmaf(q.z, fa[2], a0), a1 = fmaf(q.w, fa[3], a1);
    b0 = fmaf(q.x, fb[0], b0), b1 = fmaf(q.y, fb[1], b1), b0 = fmaf(q.z, fb[2], b0), b1 = fmaf(q.w, fb[3], b1);
  }
  const float sa = (a0 + a1) * kLog2e, sb = (b0 + b1) * kLog2e;  // log2 domain
  const float mn = fmaxf(sa, sb);
  if (mn > m) {
    const float c = fast_exp2(m - mn);
    l *= c;
#pragma unroll
    for (int x = 0; x < HDP; x++) acc[x] *= c;
    m = mn;
  }
  const float pa = fast_exp2(sa - m), pb = fast_exp2(sb - m);
  l += pa + pb;
#pragma unroll
  for (int i = 0; i < HDP / VEC; i++) {
    float fa[VEC], fb[VEC];
    Loader<T, VEC>::load(va + i * VEC, fa);
    Loader<T, VEC>::load(vb + i * VEC, fb);
#pragma unroll
    for (int e = 0; e < VEC; e++) acc[i * VEC + e] = fmaf(pa, fa[e], fmaf(pb, fb[e], acc[i * VEC + e]));
  }
}

// The same for a thread that owns W = hd / R columns of the (key, head) pair, R = 2 or 4
// adjacent lanes sharing the pair (head size 64 and 128: a whole 128-wide row per thread
// costs 512 bytes of every stage and 128 accumulator registers, so few keys fit a tile
// and the threads' long dependent chains leave the SM idle — measured 2.5 TB/s).  The
// partial scores are added across the R lanes by shuffles restricted to the group; m
// and l then evolve identically in all of them.  q lives in registers, loaded once in
// the same rotated chunk order as the row is walked (see Rotated).
template <typename T, int W, int VEC, int R>
__device__ __forceinline__ void process_key_sub(const T* kp, const T* vp, const float (&q)[W],
                                                float& m, float& l, float (&acc)[W], int rot,
                                                unsigned groupMask) {
  constexpr int NCH = W / VEC;
  float s0 = 0.f, s1 = 0.f;
#pragma unroll
  for (int i = 0; i < NCH; i++) {
    const int ci = (i + rot) & (NCH - 1);
    float f[VEC];
    Loader<T, VEC>::load(kp + ci * VEC, f);
#pragma unroll
    for (int e = 0; e < VEC; e += 2) {
      s0 = fmaf(q[i * VEC + e], f[e], s0);
      s1 = fmaf(q[i * VEC + e + 1], f[e + 1], s1);
    }
  }
  float s = s0 + s1;
#pragma unroll
  for (int o = 1; o < R; o <<= 1) s += __shfl_xor_sync(groupMask, s, o);
  s *= kLog2e;  // log2 domain
  if (s > m) {
    const float c = fast_exp2(m - s);
    l *= c;
#pragma unroll
    for (int x = 0; x < W; x++) acc[x] *= c;
    m = s;
  }
  const float pe = fast_exp2(s - m);
  l += pe;
#pragma unroll
  for (int i = 0; i < NCH; i++) {
    const int ci = (i + rot) & (NCH - 1);
    float f[VEC];
    Loader<T, VEC>::load(vp + ci * VEC, f);
#pragma unroll
    for (int e = 0; e < VEC; e++) acc[i * VEC + e] = fmaf(pe, f[e], acc[i * VEC + e]);
  }
}

// Two keys at once for the same thread: the two dot products, their shuffles and the two
// accumulations are independent instruction streams, which a thread with one key at a time
// does not have (nine warps per SM hide little latency).
template <typename T, int W, int VEC, int R>
__device__ __forceinline__ void process_key_pair(const T* ka, const T* va, const T* kb, const T* vb,
                                                 const float (&q)[W], float& m, float& l,
                                                 float (&acc)[W], int rot, unsigned groupMask) {
  constexpr int NCH = W / VEC;
  float a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
#pragma unroll
  for (int i = 0; i < NCH; i++) {
    const int ci = (i + rot) & (NCH - 1);
    float fa[VEC], fb[VEC];
    Loader<T, VEC>::load(ka + ci * VEC, fa);
    Loader<T, VEC>::load(kb + ci * VEC, fb);
#pragma unroll
    for (int e = 0; e < VEC; e += 2) {
      a0 = fmaf(q[i * VEC + e], fa[e], a0);
      a1 = fmaf(q[i * VEC + e + 1], fa[e + 1], a1);
      b0 = fmaf(q[i * VEC + e], fb[e], b0);
      b1 = fmaf(q[i * VEC + e + 1], fb[e + 1], b1);
    }
  }
  float sa = a0 + a1, sb = b0 + b1;
#pragma unroll
  for (int o = 1; o < R; o <<= 1) {
    sa += __shfl_xor_sync(groupMask, sa, o);
    sb += __shfl_xor_sync(groupMask, sb, o);
  }
  sa *= kLog2e, sb *= kLog2e;  // log2 domain
  const float mn = fmaxf(sa, sb);
  if (mn > m) {
    const float c = fast_exp2(m - mn);
    l *= c;
#pragma unroll
    for (int x = 0; x < W; x++) acc[x] *= c;
    m = mn;
  }
  const float pa = fast_exp2(sa - m), pb = fast_exp2(sb - m);
  l += pa + pb;
#pragma unroll
  for (int i = 0; i < NCH; i++) {
    const int ci = (i + rot) & (NCH - 1);
    float fa[VEC], fb[VEC];
    Loader<T, VEC>::load(va + ci * VEC, fa);
    Loader<T, VEC>::load(vb + ci * VEC, fb);
#pragma unroll
    for (int e = 0; e < VEC; e++) acc[i * VEC + e] = fmaf(pa, fa[e], fmaf(pb, fb[e], acc[i * VEC + e]));
  }
}

// Cross-GPU hand-over, called by the consumer threads of the block that wrote the final
// rows of (sequence b, head block) into this rank's staging buffer.  The rows go to the one
// rank that merges sequence b (its owner): plain, coalesced stores into that rank's
// exchange buffer — peer memory unless the owner is this rank.  The block then counts
// itself in for that owner; the last block to do so fences at system scope and publishes
// this rank's step in the owner's arrival word (one release store), so an owner is told as
// soon as its rows are complete, while the other owners' sequences are still being
// attended.  The last owner group to finish moves this rank's step counter for the merge
// kernel and the next launch.
__device__ __forceinline__ void exchange_rows(const DecodeParams& p, int b, int hq, int h0, int tid,
                                              uint32_t epoch, int headBlocks) {
  const int stride = 2 + p.hd;
  const int owner = owner_of(b, p.batch, p.xWorld), bl = b - owner_first(owner, p.batch, p.xWorld);
  const float* src = p.xStage + ((int64_t)b * p.qHeads + h0) * stride;  // this block's rows: contiguous
  float* dst = p.xPartials[owner] +
               ((((int64_t)(epoch & 1u) * p.xWorld + p.xRank) * p.xPer + bl) * p.qHeads + h0) * stride;
  const int n = hq * stride;
  named_barrier_sync(1, kConsumers);   // the rows this block's threads wrote are visible to all of them
  for (int i = tid; i < n; i += kConsumers) dst[i] = __ldcg(src + i);
  __threadfence();                     // each thread's stores, before the block is counted in
  named_barrier_sync(1, kConsumers);
  if (tid != 0) return;
  unsigned* counts = p.xStep + 2;      // [world] blocks arrived per owner, then owners done
  const int owned = owner_count(owner, p.batch, p.xWorld);
  if (atomicAdd(counts + owner, 1u) != (unsigned)(owned * headBlocks) - 1u) return;
  counts[owner] = 0;                   // ready for the next launch
  __threadfence_system();
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p.xFlags[owner] + p.xRank), "r"(epoch)
               : "memory");
  if (atomicAdd(counts + p.xWorld, 1u) != (unsigned)p.xWorld - 1u) return;   // every rank owns some
  counts[p.xWorld] = 0;
  __threadfence();
  *reinterpret_cast<volatile uint32_t*>(p.xStep) = epoch;
}

// The last block's merge of the splits' partials (rows of (m, l, acc) in log2 units) for `heads`
// consecutive query heads, by the consumer threads.  The weights of all splits go to shared memory
// first, a warp per head; after that every load of an accumulator is independent of the
// others, a run of consecutive columns per warp and sixteen splits of it in flight.  (Each thread
// walking its own columns split by split, weight and all, waited for L2 a few hundred times: 45 us
// more for eight sequences of 4096 keys, 32 heads of 128, 18 splits.)
template <typename T>
__device__ __noinline__ void merge_splits(int hd, int splits, int qHeads, const float* base, T* out, float* partials,
                                          int heads, float* smem, int smemFloats) {
  const int tid = threadIdx.x, lane = tid & 31, stride = 2 + hd;
  const int64_t ss = (int64_t)qHeads * stride;     // between splits
  const int atOnce = min(heads, smemFloats / (splits + 1));
  float* sInv = smem;                              // [atOnce]
  float* sW = smem + atOnce;                       // [atOnce][splits]
  for (int h0 = 0; h0 < heads; h0 += atOnce) {
    const int n = min(atOnce, heads - h0);
    const float* rows = base + (int64_t)h0 * stride;
    if (h0) named_barrier_sync(1, kConsumers);     // the heads before are done with the weights
    for (int hl = tid >> 5; hl < n; hl += kConsumerWarps) {
      float m[2], l[2];                            // splits lane and lane + 32
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int s = lane + 32 * i;
        m[i] = s < splits ? __ldcg(rows + hl * stride + s * ss) : kNegSeed;
        l[i] = s < splits ? __ldcg(rows + hl * stride + s * ss + 1) : 0.f;
      }
      const float M = warp_max(fmaxf(m[0], m[1]));
      const float w0 = fast_exp2(m[0] - M), w1 = fast_exp2(m[1] - M);
      const float L = warp_sum(fmaf(l[0], w0, l[1] * w1));
      if (lane < splits) sW[hl * splits + lane] = w0;
      if (lane + 32 < splits) sW[hl * splits + lane + 32] = w1;
      if (lane == 0) {
        sInv[hl] = L > 0.f ? 1.f / L : 0.f;
        if (partials) {
          partials[(h0 + hl) * stride] = L > 0.f ? M * 0.6931471805599453f : kNegSeed;
          partials[(h0 + hl) * stride + 1] = L;
        }
      }
    }
    named_barrier_sync(1, kConsumers);
    auto sum = [&](int i, auto zero) {             // column (or column pair) i of the n * hd
      using V = decltype(zero);
      constexpr int N = sizeof(V) / 4;
      const int at = i * N, hl = at / hd, x = at - hl * hd;
      const float* src = rows + hl * stride + 2 + x;
      const float* w = sW + hl * splits;
      float o[N] = {};
      for (int s0 = 0; s0 < splits; s0 += 16) {
        V v[16];
#pragma unroll
        for (int s = 0; s < 16; s++)
          if (s0 + s < splits) v[s] = __ldcg(reinterpret_cast<const V*>(src + (s0 + s) * ss));
#pragma unroll
        for (int s = 0; s < 16; s++)
          if (s0 + s < splits) {
#pragma unroll
            for (int e = 0; e < N; e++) o[e] = fmaf(reinterpret_cast<const float*>(&v[s])[e], w[s0 + s], o[e]);
          }
      }
#pragma unroll
      for (int e = 0; e < N; e++) {
        if (partials) partials[(h0 + hl) * stride + 2 + x + e] = o[e];
        else out[(int64_t)(h0 + hl) * hd + x + e] = from_f32<T>(o[e] * sInv[hl]);
      }
    };
    if (hd % 2 == 0) {                             // rows start on eight bytes
      for (int i = tid; i < n * hd / 2; i += kConsumers) sum(i, float2{});
    } else {
      for (int i = tid; i < n * hd; i += kConsumers) sum(i, float{});
    }
  }
}

template <typename T, int HDP, bool EXACT, int VEC, bool BULK, int R = 1>
__global__ void __launch_bounds__(BULK ? kConsumers + 32 : kConsumers, HDP / R <= 64 ? 2 : 1)
decode_kernel(const DecodeParams p) {
  constexpr bool QSMEM = true;
  constexpr int W = HDP / R;   // columns of a head per thread (R lanes share a (key, head) pair)
  static_assert(R == 1 || (EXACT && BULK && VEC > 1 && (W % VEC) == 0), "sub-row threads: exact bulk path only");
  constexpr int QS = q_stride(HDP);
  extern __shared__ __align__(128) unsigned char smemRaw[];
  __shared__ int sAbort;
  __shared__ int sAbortSeen;
  __shared__ int sIsLast;
  __shared__ float sHeadTop[kConsumers], sHeadSum[kConsumers];
  __shared__ __align__(8) uint64_t sFull[kMaxStages], sEmpty[kMaxStages];

  const int tid = threadIdx.x;
  DEC_TRACE(0);
  // Launched as a programmatic dependent of the kernel before it in the stream (see
  // launch_one): the blocks may become resident while that kernel's last blocks finish, and
  // wait here until all of its writes are visible.  Nothing above reads memory.
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int split = blockIdx.x, zb = blockIdx.z;
  const int by = blockIdx.y;   // unique per (attention, sequence): indexes scratch and counters
  int b = by;
  if (p.xWorld > 1) {   // the sequences this rank merges itself come last
    b += p.xRot;
    if (b >= p.batch) b -= p.batch;
  }
  // The second attention of the launch (cross-attention) takes blocks [batch, 2*batch).
  const bool sec = p.hasSecond && by >= p.batch;
  if (sec) b = by - p.batch;
  const void* aQ = sec ? p.s2.q : p.q;
  void* aOut = sec ? p.s2.out : p.out;
  const int32_t* aLens = sec ? p.s2.kvLens : p.kvLens;
  const int64_t aSeqStride = sec ? p.s2.cacheSeqStride : p.cacheSeqStride;
  const int64_t aQStride = sec ? p.s2.qRowStride : p.qRowStride;
  const int aCacheRows = sec ? p.s2.cacheRows : p.cacheRows;
  const int aKvLen = sec ? p.s2.kvLen : p.kvLen;
  const int aWl = sec ? p.s2.wl : p.wl;
  const int hd = p.hd;
  const int group = p.qHeads / p.kvHeads;
  const int kvh0 = zb * p.kvPerCta;
  const int nkv = min(p.kvPerCta, p.kvHeads - kvh0);
  const int hqReal = nkv * group;           // query heads of this CTA
  const int hqMax = p.kvPerCta * group * R;  // thread columns: (head, lane of the head's group)
  const int hq = hqReal * R;
  const int KS = p.keySlots;
  const int sliceElems = nkv * hd;
  const int rowElems = p.kvHeads * hd;
  // Where the final (m, l, acc) rows go, if not into `out`: the caller's buffer, or —
  // with the cross-GPU exchange — this rank's staging buffer, from where exchange_rows
  // sends them to the rank that merges the sequence.  The step now starting is one past
  // the rank's step counter, which only the last block of this launch moves, so all
  // blocks read the same value.
  float* partialsOut = p.partialsOut;
  uint32_t epoch = 0;
  if (p.xWorld > 0) {
    epoch = *reinterpret_cast<volatile uint32_t*>(p.xStep) + 1u;
    partialsOut = p.xStage;
  }

  // Key range of this sequence that lives in the cache.
  // L: visible rows of this cache; Lg: the sequence's length (the two differ only when the
  // cache is one rank's shard of the sequence).
  int64_t lo, end, L = 0, Lg = 0;
  bool hasNew = p.kNew != nullptr && !sec;
  // This sequence's caches: its slice of the slab, or its own allocation.
  const void* const* kPtrs = sec ? p.s2.kPtrs : p.kPtrs;
  const void* const* vPtrs = sec ? p.s2.vPtrs : p.vPtrs;
  const T* kSeq = kPtrs ? static_cast<const T*>(kPtrs[b])
                        : static_cast<const T*>(sec ? p.s2.kCache : p.kCache) + (int64_t)b * aSeqStride;
  const T* vSeq = vPtrs ? static_cast<const T*>(vPtrs[b])
                        : static_cast<const T*>(sec ? p.s2.vCache : p.vCache) + (int64_t)b * aSeqStride;
  // What a consumer thread stages — q and, in split 0, the appended K/V row — is loaded into
  // registers before the sequence's length is looked at: the length decides where the rows
  // go, not where they come from, and under a saturated memory system every load that has
  // to wait for another costs microseconds of set-up.
  constexpr int kPre = 4;   // elements per thread held in registers; longer rows finish in a loop
  const T* qg = static_cast<const T*>(aQ) + (int64_t)b * aQStride;
  const bool roped = p.ropeCos != nullptr && !p.useRange && !sec;
  const bool pre = R == 1 && !roped && tid < kConsumers;
  const bool preNew = pre && hasNew && split == 0 && !p.useRange;
  const T* kn = hasNew ? static_cast<const T*>(p.kNew) + (int64_t)b * p.kNewRowStride + kvh0 * hd : nullptr;
  const T* vn = hasNew ? static_cast<const T*>(p.vNew) + (int64_t)b * p.vNewRowStride + kvh0 * hd : nullptr;
  T qPre[kPre], knPre[kPre], vnPre[kPre];
#pragma unroll
  for (int i = 0; i < kPre; i++) {
    const int idx = tid + i * kConsumers;
    qPre[i] = knPre[i] = vnPre[i] = from_f32<T>(0.f);
    if (pre && idx < hqReal * hd) qPre[i] = qg[kvh0 * group * hd + idx];   // the CTA's heads are contiguous
    if (preNew && idx < sliceElems) {
      knPre[i] = kn[idx];
      vnPre[i] = vn[idx];
    }
  }
  // (a separately allocated cache is only known here: the bulk copies need 16-byte alignment)
  const bool misaligned = kPtrs && BULK &&
                          ((reinterpret_cast<uintptr_t>(kSeq) | reinterpret_cast<uintptr_t>(vSeq)) & 15u);
  if (p.useRange) {
    lo = p.lo;
    end = p.end;
  } else {
    Lg = L = aLens ? aLens[b] : aKvLen;
    if (misaligned || (!p.kvSharded && L > aCacheRows)) {
      // A length past the cache's capacity (the host checks only the scalar kvLen; this one
      // lives on the device): writeRows would refuse it ('rows exceed dst capacity').  The
      // sequence is treated as empty — nothing appended, nothing read, zeros out — and the
      // status word reports it.  The same for a cache pointer the bulk copies cannot take,
      // whether the cache holds the whole sequence or a shard of it.
      if (tid == 0) atomicOr(p.status, kStatusBadState);
      Lg = L = 0;
      hasNew = false;
    } else if (p.kvSharded) {
      // This cache holds rows [shardStart, shardStart + cacheRows) of the sequence: it sees
      // what falls inside, and takes the appended row (global row Lg-1) only if that is one
      // of its own.
      const int64_t local = Lg - p.shardStart;
      hasNew = hasNew && local >= 1 && local <= p.cacheRows;
      L = local < 0 ? 0 : local > p.cacheRows ? p.cacheRows : local;
    }
    end = L - 1;
    lo = Lg - 1 - aWl - p.shardStart;
    if (lo < 0) lo = 0;
    if (hasNew) end -= 1;  // row L-1 is the appended one, taken from kNew/vNew
    if (L <= 0) { lo = 1; end = -1; }
  }
  const int64_t n = end >= lo ? end - lo + 1 : 0;
  int64_t chunk = (n + p.splits - 1) / p.splits;
  chunk = (chunk + KS - 1) / KS * KS;
  int64_t s0 = lo + (int64_t)split * chunk, s1 = s0 + chunk;
  if (s1 > end + 1) s1 = end + 1;
  const int ntiles = s1 > s0 ? (int)((s1 - s0 + KS - 1) / KS) : 0;

  const T* kBase = kSeq + kvh0 * hd;
  const T* vBase = vSeq + kvh0 * hd;

  // Shared-memory carve-up: [q][appended K, V slices][ring: stages x (K tile, V tile)];
  // the ring is reused for the slot merge at the end.
  float* sQ = reinterpret_cast<float*>(smemRaw);
  // (threads that own a slice of a head keep q in registers and read the appended row back
  // from the cache: no staging areas)
  const int qBytes = R == 1 ? ((hqMax * QS * 4 + 127) / 128) * 128 : 0;
  const int newBytes = (R == 1 && p.kNew != nullptr) ? ((p.kvPerCta * hd * (int)sizeof(T) + 127) / 128) * 128 : 0;
  T* sKn = reinterpret_cast<T*>(smemRaw + qBytes);           // appended K slice
  T* sVn = reinterpret_cast<T*>(smemRaw + qBytes + newBytes);  // appended V slice
  unsigned char* ring = smemRaw + qBytes + 2 * newBytes;
  const int tileBytes = ((KS * p.kvPerCta * hd * (int)sizeof(T) + 127) / 128) * 128;
  const int stages = BULK ? p.stages : 1;

  if (tid == 0) {
    sAbort = 0;
    sIsLast = 0;
    if (BULK) {
      for (int s = 0; s < stages; s++) {
        mbar_init(smem_u32(&sFull[s]), 1);
        mbar_init(smem_u32(&sEmpty[s]), kConsumerWarps);
      }
      fence_barrier_init();
    }
  }
  __syncthreads();

  if (BULK && tid >= kConsumers) {
    // ---------------- producer warp ----------------
    const int lane = tid - kConsumers;
    const bool flat = (nkv == p.kvHeads);
    for (int it = 0; it < ntiles; it++) {
      const int s = it % stages;
      if (it >= stages) {
        if (!mbar_park(smem_u32(&sEmpty[s]), ((it / stages) - 1) & 1, &sAbort)) {
          sAbort = 1;
          break;
        }
      }
      const int64_t k0 = s0 + (int64_t)it * KS;
      const int nk = (int)min((int64_t)KS, s1 - k0);
      const uint32_t bar = smem_u32(&sFull[s]);
      const uint32_t dK = smem_u32(ring + (size_t)s * 2 * tileBytes);
      const uint32_t dV = dK + tileBytes;
      const uint32_t rowBytes = (uint32_t)sliceElems * sizeof(T);
      if (lane == 0) mbar_expect_tx(bar, 2u * nk * rowBytes);
      __syncwarp();
      if (flat) {
        if (lane == 0) {
          bulk_g2s(dK, kBase + k0 * rowElems, nk * rowBytes, bar);
          bulk_g2s(dV, vBase + k0 * rowElems, nk * rowBytes, bar);
        }
      } else {
        for (int r = lane; r < nk; r += 32) {
          bulk_g2s(dK + r * rowBytes, kBase + (k0 + r) * rowElems, rowBytes, bar);
          bulk_g2s(dV + r * rowBytes, vBase + (k0 + r) * rowElems, rowBytes, bar);
        }
      }
    }
    return;
  }

  // ---------------- consumers ----------------
  const int hv = tid % hqMax;        // thread column
  const int hl = hv / R;             // query head within the CTA
  const int sub = hv % R;            // which W columns of the head
  const int slot = tid / hqMax;
  const bool active = slot < KS && hv < hq;
  const int h = kvh0 * group + hl;   // query head
  const int kvl = hl / group;        // kv head within the CTA's slice
  const unsigned groupMask = R == 1 ? 0u : (((1u << R) - 1u) << ((tid & 31) & ~(R - 1)));

  // Stage q (f32) and, in split 0, the appended K/V slices; with rope tables q and
  // the new K row are rotated here and rounded to T as the separate rope dispatch
  // stores them.  The new row goes to the cache from the same threads (what
  // writeRows would do) and is attended from shared memory after the cache keys.
  const bool appendHere = hasNew && split == 0 && !p.useRange && L >= 1;
  const float* qv = sQ + hl * QS;
  const int64_t ropeRow = p.ropeByPos ? (Lg >= 1 ? Lg - 1 : 0) : b;
  const float* rc = roped ? p.ropeCos + ropeRow * hd : nullptr;
  const float* rs = roped ? p.ropeSin + ropeRow * hd : nullptr;
  {
    if (R > 1) {
      // q goes straight to registers below
    } else if (roped) {
      const int hp = hd >> 1;
      for (int idx = tid; idx < hqReal * hp; idx += kConsumers) {
        const int hh = idx / hp, x = (idx - hh * hp) * 2;
        const T* src = qg + (kvh0 * group + hh) * hd + x;
        float r0, r1;
        rope_pair(to_f32<T>(src[0]), to_f32<T>(src[1]), rc[x], rs[x], r0, r1);
        sQ[hh * QS + x] = to_f32<T>(from_f32<T>(r0));
        sQ[hh * QS + x + 1] = to_f32<T>(from_f32<T>(r1));
      }
    } else {
#pragma unroll
      for (int i = 0; i < kPre; i++) {
        const int idx = tid + i * kConsumers;
        if (idx < hqReal * hd) {
          const int hh = idx / hd, x = idx - hh * hd;
          sQ[hh * QS + x] = to_f32<T>(qPre[i]);
        }
      }
      for (int idx = tid + kPre * kConsumers; idx < hqReal * hd; idx += kConsumers) {
        const int hh = idx / hd, x = idx - hh * hd;
        sQ[hh * QS + x] = to_f32<T>(qg[(kvh0 * group + hh) * hd + x]);
      }
    }
    if (appendHere) {
      T* kc = const_cast<T*>(kBase) + (L - 1) * rowElems;
      T* vc = const_cast<T*>(vBase) + (L - 1) * rowElems;
      // Loads kBatch at a time before any of their stores: the compiler cannot move a load over a
      // store to the cache, and one element at a time a row of 4096 took 30 us under the streams.
      constexpr int kBatch = 8;
      if (roped) {
        const int hp = hd >> 1;
        for (int i0 = tid; i0 < nkv * hp; i0 += kBatch * kConsumers) {
          T k0[kBatch], k1[kBatch];
          float c[kBatch], sn[kBatch];
#pragma unroll
          for (int i = 0; i < kBatch; i++) {
            const int idx = i0 + i * kConsumers, x = idx % hp * 2;
            if (idx < nkv * hp) k0[i] = kn[2 * idx], k1[i] = kn[2 * idx + 1], c[i] = rc[x], sn[i] = rs[x];
          }
#pragma unroll
          for (int i = 0; i < kBatch; i++) {
            const int at = 2 * (i0 + i * kConsumers);
            if (at >= nkv * hd) break;
            float r0, r1;
            rope_pair(to_f32<T>(k0[i]), to_f32<T>(k1[i]), c[i], sn[i], r0, r1);
            const T t0 = from_f32<T>(r0), t1 = from_f32<T>(r1);
            if (R == 1) sKn[at] = t0, sKn[at + 1] = t1;
            kc[at] = t0, kc[at + 1] = t1;
          }
        }
      }
      if (preNew) {
#pragma unroll
        for (int i = 0; i < kPre; i++) {
          const int x = tid + i * kConsumers;
          if (x < sliceElems) {
            sKn[x] = knPre[i], kc[x] = knPre[i];
            sVn[x] = vnPre[i], vc[x] = vnPre[i];
          }
        }
      }
      for (int x0 = tid + (preNew ? kPre * kConsumers : 0); x0 < sliceElems; x0 += kBatch * kConsumers) {
        T t[kBatch], u[kBatch];
#pragma unroll
        for (int i = 0; i < kBatch; i++) {
          const int x = x0 + i * kConsumers;
          if (x < sliceElems) {
            u[i] = vn[x];
            if (!roped) t[i] = kn[x];
          }
        }
#pragma unroll
        for (int i = 0; i < kBatch; i++) {
          const int x = x0 + i * kConsumers;
          if (x >= sliceElems) break;
          if (!roped) {
            if (R == 1) sKn[x] = t[i];
            kc[x] = t[i];
          }
          if (R == 1) sVn[x] = u[i];
          vc[x] = u[i];
        }
      }
    }
    named_barrier_sync(1, kConsumers);
  }
  DEC_TRACE(1);

  float m = kNegSeed, l = 0.f;
  float acc[W];
  constexpr bool ROT = R > 1 || Rotated<HDP, EXACT, VEC>::value;
  // Threads whose rows start in the same bank take different rotations (see Rotated):
  // with 64-byte slices every second thread does.
  constexpr int kSameBank = (W * (int)sizeof(T) >= 128) ? 1 : 128 / (W * (int)sizeof(T));
  const int rot = ROT ? ((tid / kSameBank) & (W / VEC - 1)) : 0;
#pragma unroll
  for (int x = 0; x < W; x++) acc[x] = 0.f;
  float qr[R > 1 ? W : 1];
  if (R > 1) {
    // This thread's W columns of q, rotated like the rows it will walk, with the rope applied
    // and rounded to T as the separate rope dispatch would store them.
#pragma unroll
    for (int x = 0; x < (R > 1 ? W : 1); x++) qr[x] = 0.f;
    if (hv < hq) {
      const T* src = qg + (int64_t)h * hd + sub * W;
#pragma unroll
      for (int i = 0; i < W / VEC; i++) {
        const int ci = (i + rot) & (W / VEC - 1);
        float f[VEC];
        Loader<T, VEC>::load(src + ci * VEC, f);
#pragma unroll
        for (int e = 0; e < VEC; e += 2) {
          float r0 = f[e], r1 = f[e + 1];
          if (roped) {
            const int x = sub * W + ci * VEC + e;
            rope_pair(f[e], f[e + 1], rc[x], rs[x], r0, r1);
            r0 = to_f32<T>(from_f32<T>(r0));
            r1 = to_f32<T>(from_f32<T>(r1));
          }
          qr[(i * VEC + e) % (R > 1 ? W : 1)] = r0;
          qr[(i * VEC + e + 1) % (R > 1 ? W : 1)] = r1;
        }
      }
    }
  }
  if (active && slot == 0 && split == 0 && p.sinks) {
    m = p.sinks[h];  // sinks are log2-space: sink * ln2 * log2e
    l = 1.f;
  }

  bool ok = true;
  int it = 0;
  // (f32 tiles are too large for a ring of four of them)
  constexpr bool PAIRS = BULK && (R > 1 || (EXACT && !ROT && VEC == 4 && sizeof(T) == 2));
  if constexpr (PAIRS) {
    // Tiles two at a time while the ring is deep enough to keep copies in flight behind them.
    if (stages >= 4) {
      for (; it + 1 < ntiles; it += 2) {
        const int sa = it % stages, sb = (it + 1) % stages;
        if (!mbar_park(smem_u32(&sFull[sa]), (it / stages) & 1, &sAbort) ||
            !mbar_park(smem_u32(&sFull[sb]), ((it + 1) / stages) & 1, &sAbort)) {
          ok = false;
          break;
        }
        const T* aK = reinterpret_cast<const T*>(ring + (size_t)sa * 2 * tileBytes);
        const T* bK = reinterpret_cast<const T*>(ring + (size_t)sb * 2 * tileBytes);
        const int nkb = (int)min((int64_t)KS, s1 - (s0 + (int64_t)(it + 1) * KS));  // tile `it` is full
        if (active) {
          const int off = slot * sliceElems + kvl * hd + sub * W;
          const int vOff = tileBytes / (int)sizeof(T);
          if constexpr (R == 1) {
            if (slot < nkb)
              process_two<T, HDP, VEC>(aK + off, aK + vOff + off, bK + off, bK + vOff + off, qv, m, l, acc);
            else
              process_key<T, HDP, EXACT, VEC, QSMEM>(aK + off, aK + vOff + off, qv, hd, m, l, acc, rot);
          } else if (slot < nkb)
            process_key_pair<T, W, VEC, R>(aK + off, aK + vOff + off, bK + off, bK + vOff + off, qr, m,
                                           l, acc, rot, groupMask);
          else
            process_key_sub<T, W, VEC, R>(aK + off, aK + vOff + off, qr, m, l, acc, rot, groupMask);
        }
        __syncwarp();
        if ((tid & 31) == 0) {
          mbar_arrive(smem_u32(&sEmpty[sa]));
          mbar_arrive(smem_u32(&sEmpty[sb]));
        }
      }
    }
  }
  for (; it < ntiles && ok; it++) {
    const int64_t k0 = s0 + (int64_t)it * KS;
    const int nk = (int)min((int64_t)KS, s1 - k0);
    const int s = BULK ? it % stages : 0;
    T* tK = reinterpret_cast<T*>(ring + (size_t)s * 2 * tileBytes);
    T* tV = reinterpret_cast<T*>(ring + (size_t)s * 2 * tileBytes + tileBytes);
    if (BULK) {
      if (!mbar_park(smem_u32(&sFull[s]), (it / stages) & 1, &sAbort)) { ok = false; break; }
      if (it == 0) DEC_TRACE(2);
    } else {
      named_barrier_sync(1, kConsumers);
      for (int idx = tid; idx < nk * sliceElems; idx += kConsumers) {
        const int jj = idx / sliceElems, x = idx - jj * sliceElems;
        tK[idx] = kBase[(k0 + jj) * rowElems + x];
        tV[idx] = vBase[(k0 + jj) * rowElems + x];
      }
      named_barrier_sync(1, kConsumers);
    }
    if (active && slot < nk) {
      const int off = slot * sliceElems + kvl * hd + sub * W;
      if constexpr (R > 1) process_key_sub<T, W, VEC, R>(tK + off, tV + off, qr, m, l, acc, rot, groupMask);
      else process_key<T, HDP, EXACT, VEC, QSMEM>(tK + off, tV + off, qv, hd, m, l, acc, rot);
    }
    if (BULK) {
      __syncwarp();
      if ((tid & 31) == 0) mbar_arrive(smem_u32(&sEmpty[s]));
    }
  }

  if (!ok) sAbort = 1;
  DEC_TRACE(3);
  // This block has streamed its keys: once every block has, the next kernel's blocks may
  // take the freed slots (they wait for this grid to finish before they read anything).
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // Fused append: split 0 attends to the new row it staged (and stored) above.
  if (appendHere && active && slot == 0) {
    const int off = kvl * hd + sub * W;
    // (sub-row threads read the row this block stored to the cache before the barrier above)
    if constexpr (R > 1)
      process_key_sub<T, W, VEC, R>(kBase + (L - 1) * rowElems + off, vBase + (L - 1) * rowElems + off, qr,
                                    m, l, acc, rot, groupMask);
    else process_key<T, HDP, EXACT, VEC, QSMEM>(sKn + off, sVn + off, qv, hd, m, l, acc, rot);
  }

  // Every consumer is through its tiles (or has given up): the ring is free.  Whether a wait
  // ran out is decided once for the whole block — a thread that finished its tiles before
  // another one's wait ran out must not go on to barriers the other will never reach.
  named_barrier_sync(1, kConsumers);
  if (tid == 0) sAbortSeen = sAbort;
  named_barrier_sync(1, kConsumers);
  if (sAbortSeen) {
    // A wait ran out: record it, let copies in flight land, leave.
    if (tid == 0) {
      atomicOr(p.status, kStatusWaitTimeout);
      // (the arrival counter, which the blocks leave alone then, and which is cleared with the status
      // word: the merge launch writes nothing for these heads)
      if (p.mergeAfter) p.counters[by * gridDim.z + zb] = 1;
    }
    for (int i = 0; i < 64; i++) __nanosleep(4000);
    return;
  }

  // ---- merge the key slots of each head (log-sum-exp) ----
  // Every thread brings its own sums to its head's maximum before they meet in shared memory, so
  // that a column of the result is a plain sum over the slots; consecutive threads take
  // consecutive columns of the block's heads.  (With the weights worked out anew for every column and
  // the columns dealt out by slot: 2.4 to 3.3 us of every launch.)
  constexpr int MS = 1 + W;                          // l, columns: an odd pitch, distinct banks
  float* sTop = reinterpret_cast<float*>(ring);      // [KS][hqMax] maxima
  float* sM = sTop + KS * hqMax;                     // [KS][hqMax][MS]
  if (active) sTop[slot * hqMax + hv] = m;
  named_barrier_sync(1, kConsumers);
  if (active) {
    float top = m;
#pragma unroll 8
    for (int s = 0; s < KS; s++) top = fmaxf(top, sTop[s * hqMax + hv]);
    const float w = fast_exp2(m - top);
    float* r = sM + (slot * hqMax + hv) * MS;
    r[0] = l * w;
#pragma unroll
    for (int i = 0; i < W / VEC; i++) {
      float* dst = r + 1 + (ROT ? ((i + rot) & (W / VEC - 1)) : i) * VEC;
#pragma unroll
      for (int e = 0; e < VEC; e++) dst[e] = acc[i * VEC + e] * w;
    }
    if (slot == 0 && sub == 0) sHeadTop[hl] = top;
  }
  named_barrier_sync(1, kConsumers);
  for (int hh = tid; hh < hqReal; hh += kConsumers) {
    float sum = 0.f;
#pragma unroll 8
    for (int s = 0; s < KS; s++) sum += sM[(s * hqMax + hh * R) * MS];
    sHeadSum[hh] = sum;
  }
  named_barrier_sync(1, kConsumers);

  const int stride = 2 + hd;  // partials row in global memory
  const bool whole = p.splits == 1;
  const int64_t head0 = (int64_t)b * p.qHeads + kvh0 * group;
  float* rowF = !whole ? p.scratch + (((int64_t)by * p.splits + split) * p.qHeads + kvh0 * group) * stride
                       : partialsOut ? partialsOut + head0 * stride : nullptr;
  T* rowT = static_cast<T*>(aOut) + head0 * hd;
  if (rowF) {
    for (int hh = tid; hh < hqReal; hh += kConsumers) {
      // finished rows carry the maximum in natural-log units, split rows in log2 units
      const float top = sHeadTop[hh], sum = sHeadSum[hh];
      rowF[hh * stride] = !whole ? top : sum > 0.f ? top * 0.6931471805599453f : kNegSeed;
      rowF[hh * stride + 1] = sum;
    }
  }
  const int cols = EXACT ? HDP : hd;   // (a constant to divide by, where there is one)
  for (int i = tid; i < hqReal * cols; i += kConsumers) {
    const int hh = i / cols, x = i - hh * cols;
    const float* r = sM + (hh * R + x / W) * MS + 1 + x % W;
    float o = 0.f;
#pragma unroll 8
    for (int s = 0; s < KS; s++) o += r[s * hqMax * MS];
    if (rowF) {
      rowF[hh * stride + 2 + x] = o;
    } else {
      const float sum = sHeadSum[hh];
      rowT[i] = from_f32<T>(o * (sum > 0.f ? 1.f / sum : 0.f));
    }
  }
  DEC_TRACE(4);
  if (p.splits == 1) {
    if (p.xWorld > 0) exchange_rows(p, b, hqReal, kvh0 * group, tid, epoch, gridDim.z);
    DEC_TRACE(5);
    return;
  }

  if (p.mergeAfter) return;   // a launch of its own merges the splits

  // ---- last CTA of the sequence merges the splits ----
  __threadfence();
  named_barrier_sync(1, kConsumers);
  if (tid == 0) {
    const unsigned old = atomicAdd(&p.counters[by * gridDim.z + zb], 1u);
    sIsLast = (old == (unsigned)p.splits - 1);
  }
  named_barrier_sync(1, kConsumers);
  if (!sIsLast) return;
  __threadfence();
  merge_splits<T>(hd, p.splits, p.qHeads, p.scratch + ((int64_t)by * p.splits * p.qHeads + kvh0 * group) * stride,
                  static_cast<T*>(aOut) + ((int64_t)b * p.qHeads + kvh0 * group) * hd,
                  partialsOut ? partialsOut + ((int64_t)b * p.qHeads + kvh0 * group) * stride : nullptr,
                  hqReal, sM, KS * hqMax * MS);
  if (tid == 0) p.counters[by * gridDim.z + zb] = 0;  // ready for the next launch
  if (p.xWorld > 0) exchange_rows(p, b, hqReal, kvh0 * group, tid, epoch, gridDim.z);
}

// ---- f16 on the tensor cores -------------------------------------------------------------
// A warp takes one kv head and 16 or 32 keys of the tile at a time: S = q K^T with the (up to
// eight) query heads of the kv head as the rows of an m16n8k16 and the keys as its columns, then
// O = P V with S's fragments as the A operand.  The order of a contraction is free, so a thread's
// operands are 8 or 16 contiguous bytes of a key's row: columns for the scores, key pairs (by
// byte permutes) for the output.
// The tensor core adds f32 sums up by cutting off what an FMA would round, so little is left to it:
//   - q is split in two (rows g and g + 8), and no more than 16 columns go into one accumulator;
//   - a probability, p = exp(s - m) in f32 as on the FP32 pipes, is scaled by a power of two to the top of
//     a half's range and held as hi + lo (rows g and g + 8 again), 22 to 24 bits of it; the scale is
//     the block of keys' own, and what is smaller than its largest one by 2^28 or more waits for another pass,
//     so small ones keep as many bits as large ones;
//   - no more than 16 keys go into one accumulator, the rest is f32;
//   - a sink joins the sums at their end, so that a dominating one takes no bits from the keys.
// Error of the f32 partials (2-norm, against 64 bits; the FP32 pipes / here): 32 heads of 128 on 8, 50 / 487 /
// 4000 keys 1.9 / 4.8 / 13 e-7 and 1.4 / 2.0 / 3.8 e-7, scores four times as steep 3.2 / 6.2 / 18 and
// 2.3 / 3.7 / 6.1, a sink of e^20 4.5 / 15 / 76 and 4.6 / 5.2 / 6.2; the log of the sum within the same
// few e-7 of both.  What stays larger: all-positive values of heads of 36 or 52, four on each of 8 kv heads, over
// 4000 keys (2.0 and 2.4), whose keys the other kernel deals out to more threads.
// What bounds the FP32-pipe form with several query heads per kv head is that every key is read
// and converted once per query head, by two warps per scheduler: 16 sequences of 2000 keys, 32
// heads of 128 on 8, take 75.9 us among launches; here 34.9 (mma_better has more of both sides).  What bounds
// this form is the latency of nine warps, once per SM at heads of 128 (that case: DRAM 51 % busy, issue slots
// 35 %, per issue 1.5 warps waiting for shared memory, 1.4 for the pipe, 1.2 for global loads), and its instructions at
// heads of up to 64, twice per SM (96 registers a thread, 64 to 84 bytes of them spilled).
template <int HD>
struct Mma {
  static constexpr int VEC = HD % 8 == 0 ? 8 : 4;               // halves per load
  static constexpr int STEPS = (HD + 15) / 16;                  // of the scores' contraction
  static constexpr int CHUNKS = (HD + 8 * VEC - 1) / (8 * VEC); // of 8 * VEC output columns
  static constexpr int NB = HD <= 64 ? 2 : 1;                   // blocks of 16 keys at a time
  static constexpr int KEYS = 16 * NB;
};
// A probability in two halves: p * 2^e rounded, between 2^-14 (the least normal half) and 2^kPTop, and what
// that left of it times kPLow.
constexpr int kPTop = 14;
constexpr float kPLeast = 1.f / 16384, kPLow = 4096.f;

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// VEC halves as 32-bit words, zeros where `there` is false.
template <int VEC>
__device__ __forceinline__ void load_words(const __half* p, bool there, uint32_t (&w)[VEC / 2]) {
#pragma unroll
  for (int i = 0; i < VEC / 2; i++) w[i] = 0u;
  if (there) {
    if constexpr (VEC == 8) {
      const uint4 v = *reinterpret_cast<const uint4*>(p);
      w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
    } else {
      const uint2 v = *reinterpret_cast<const uint2*>(p);
      w[0] = v.x, w[1] = v.y;
    }
  }
}

// A thread's part of q, the columns its K loads will cover.  An element's upper six bits go to row g of
// the A operand and the other five to row g + 8, so that products of 17 and 16 bits are what the tensor
// core adds up and cuts off.  Heads of 128 hold both (8 sequences of 8000 keys, 8 heads of 128 on one: 54.4
// us split at each use, 52.5); narrower ones have no registers for that (64 x 8000, 8 of 52 on 2 56.9
// held, 53.9).
template <int HD>
struct MmaQuery {
  static constexpr bool HELD = HD > 64;
  uint32_t upper[Mma<HD>::STEPS][2], lower[HELD ? Mma<HD>::STEPS : 1][2];
  static __device__ __forceinline__ uint32_t high(uint32_t q) { return q & 0xffe0ffe0u; }
  static __device__ __forceinline__ uint32_t rest(uint32_t q) {
    const uint32_t h = high(q);
    const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&q), *reinterpret_cast<const __half2*>(&h));
    return *reinterpret_cast<const uint32_t*>(&d);
  }
  __device__ __forceinline__ MmaQuery(const __half* q, bool there, int t) {
    constexpr int VEC = Mma<HD>::VEC;
#pragma unroll
    for (int st = 0; st < Mma<HD>::STEPS; st++)
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const int col = VEC == 8 ? 32 * (st >> 1) + 8 * t + 4 * (st & 1) + 2 * r : 16 * st + 4 * t + 2 * r;
        const uint32_t v = there && col < HD ? *reinterpret_cast<const uint32_t*>(q + col) : 0u;
        upper[st][r] = HELD ? high(v) : v;
        if constexpr (HELD) lower[st][r] = rest(v);
      }
  }
  __device__ __forceinline__ uint32_t up(int st, int r) const { return HELD ? upper[st][r] : high(upper[st][r]); }
  __device__ __forceinline__ uint32_t low(int st, int r) const {
    if constexpr (HELD) return lower[st][r];
    else return rest(upper[st][r]);
  }
};

// KEYS keys from k and v on, `pitch` elements apart, of which the first nk count.
template <int HD>
__device__ __forceinline__ void mma_keys(const __half* k, const __half* v, int pitch, int nk, int g, int t,
                                         const MmaQuery<HD>& qa, float& m, float& l,
                                         float (&o)[Mma<HD>::CHUNKS][Mma<HD>::VEC][2]) {
  using C = Mma<HD>;
  constexpr int VEC = C::VEC, NB = C::NB, PER = VEC / 4;   // steps per load
  float sc[2 * NB][2];
#pragma unroll
  for (int i = 0; i < 2 * NB; i++) {
    const __half* row = k + (8 * i + g) * pitch + VEC * t;
    float part[4][2] = {};   // of 32 columns each
#pragma unroll
    for (int st = 0; st < C::STEPS; st += PER) {
      uint32_t w[VEC / 2];
      load_words<VEC>(row + 16 * st, VEC == 8 || 16 * st + 4 * t < HD, w);
#pragma unroll
      for (int e = 0; e < PER; e++) {
        float c[4] = {0.f, 0.f, 0.f, 0.f};
        mma_16816(c, qa.up(st + e, 0), qa.low(st + e, 0), qa.up(st + e, 1), qa.low(st + e, 1), w[2 * e], w[2 * e + 1]);
        part[(st + e) / 2][0] += c[0] + c[2];
        part[(st + e) / 2][1] += c[1] + c[3];
      }
    }
#pragma unroll
    for (int e = 0; e < 2; e++)
      sc[i][e] = C::STEPS > 4 ? (part[0][e] + part[1][e]) + (part[2][e] + part[3][e]) : part[0][e] + part[1][e];
  }
  // this thread: head g, keys 8 i + 2 t and + 1
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < 2 * NB; i++)
#pragma unroll
    for (int e = 0; e < 2; e++) {
      sc[i][e] = 8 * i + 2 * t + e < nk ? sc[i][e] : -INFINITY;
      mx = fmaxf(mx, sc[i][e]);
    }
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
  mx *= kLog2e;
  const float top = fmaxf(m, mx);
  float alpha = fast_exp2(m - top);
  m = top;
  l *= alpha;
#pragma unroll
  for (int i = 0; i < 2 * NB; i++) {
    sc[i][0] = fast_exp2(fmaf(sc[i][0], kLog2e, -top)), sc[i][1] = fast_exp2(fmaf(sc[i][1], kLog2e, -top));
    l += sc[i][0] + sc[i][1];
  }
  // The largest of these probabilities goes to the top of a half's range; those that would be below its
  // normal numbers wait for another pass, 28 powers of two further down.
  int at = kPTop + (int)fminf(top - mx, 100.f);
  for (bool more = true; more; alpha = 1.f) {
    const float up = __int_as_float((at + 127) << 23), down = __int_as_float((127 - at) << 23);
    uint32_t hi[2 * NB], lo[2 * NB];
    bool small = false;
#pragma unroll
    for (int i = 0; i < 2 * NB; i++) {
      float y[2];
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const float x = sc[i][e] * up;
        const bool later = __float_as_uint(x) - 1u < __float_as_uint(kPLeast) - 1u;   // 0 < x < kPLeast
        small |= later;
        y[e] = later ? 0.f : x;
        sc[i][e] = later ? sc[i][e] : 0.f;
      }
      const __half2 h = __floats2half2_rn(y[0], y[1]);
      const float2 f = __half22float2(h);
      const __half2 r = __floats2half2_rn((y[0] - f.x) * kPLow, (y[1] - f.y) * kPLow);
      hi[i] = *reinterpret_cast<const uint32_t*>(&h);
      lo[i] = *reinterpret_cast<const uint32_t*>(&r);
    }
    more = __any_sync(0xffffffffu, small && at < 126);   // (the same in all lanes: at most five passes)
    at = min(at + 28, 126);
#pragma unroll
    for (int c = 0; c < C::CHUNKS; c++) {
      const int col = c * 8 * VEC + VEC * g;
      uint32_t w[NB][4][VEC / 2];
#pragma unroll
      for (int b = 0; b < NB; b++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int key = 16 * b + 2 * t + (j & 1) + 8 * (j >> 1);
          load_words<VEC>(v + key * pitch + col, key < nk && (HD % (8 * VEC) == 0 || col < HD), w[b][j]);
        }
#pragma unroll
      for (int e = 0; e < VEC; e++) {
        const uint32_t sel = e & 1 ? 0x7632u : 0x5410u;
        float x0 = 0.f, x1 = 0.f;
#pragma unroll
        for (int b = 0; b < NB; b++) {
          float d[4] = {0.f, 0.f, 0.f, 0.f};
          mma_16816(d, hi[2 * b], lo[2 * b], hi[2 * b + 1], lo[2 * b + 1],
                    __byte_perm(w[b][0][e / 2], w[b][1][e / 2], sel), __byte_perm(w[b][2][e / 2], w[b][3][e / 2], sel));
          x0 += fmaf(d[2], 1.f / kPLow, d[0]);
          x1 += fmaf(d[3], 1.f / kPLow, d[1]);
        }
        o[c][e][0] = fmaf(o[c][e][0], alpha, x0 * down);
        o[c][e][1] = fmaf(o[c][e][1], alpha, x1 * down);
      }
    }
  }
}

// One head over the keys [k0, k0 + n) and, if `kn` is given, an appended row, key by key: what the
// tensor cores cannot give where a value is infinite (hi * inf + lo * inf is NaN).  The warp's
// lanes share the columns; the row goes to r = (l, columns), the maximum is returned.
template <int HD>
__device__ __noinline__ float exact_head(const __half* q, const __half* k, const __half* v, int64_t pitch, int64_t s0,
                                         int64_t s1, int tile, int off, const __half* kn, const __half* vn, float m,
                                         float l, float* r) {
  constexpr int kCols = (HD + 31) / 32;
  const int lane = threadIdx.x & 31;
  float acc[kCols];
#pragma unroll
  for (int c = 0; c < kCols; c++) acc[c] = 0.f;
  auto key = [&](const __half* kr, const __half* vr) {
    float s = 0.f;
    for (int x = lane; x < HD; x += 32) s = fmaf(__half2float(q[x]), __half2float(kr[x]), s);
    s = warp_sum(s) * kLog2e;
    if (s > m) {
      const float c = fast_exp2(m - s);
      l *= c;
#pragma unroll
      for (int i = 0; i < kCols; i++) acc[i] *= c;
      m = s;
    }
    const float pe = fast_exp2(s - m);
    l += pe;
#pragma unroll
    for (int i = 0; i < kCols; i++)
      if (lane + 32 * i < HD) acc[i] = fmaf(pe, __half2float(vr[lane + 32 * i]), acc[i]);
  };
  for (int64_t at = s0 + off; at < s1; at += tile)   // this warp's keys of every tile
    for (int64_t j = at; j < s1 && j < at + Mma<HD>::KEYS; j++) key(k + j * pitch, v + j * pitch);
  if (kn) key(kn, vn);
  if (lane == 0) r[0] = l;
#pragma unroll
  for (int i = 0; i < kCols; i++)
    if (lane + 32 * i < HD) r[1 + lane + 32 * i] = acc[i];
  __syncwarp();
  return m;
}

// ---- f16 on the tensor cores: the kernel ---------------------------------------------------
// The same streaming as decode_kernel — producer warp, ring of bulk copies, append by split 0, last
// CTA or a second launch merges the splits — with eight consumer warps that each take a kv head
// and KEYS keys of every tile (slots = 8 / kvPerCta warps share a head).  The appended row is
// attended to from the cache row the block has just stored.
template <int HD>
__global__ void __launch_bounds__(kConsumers + 32, HD <= 64 ? 2 : 1) decode_mma_kernel(const DecodeParams p) {
  using T = __half;
  using M = Mma<HD>;
  constexpr int MS = 1 + HD;   // a row of the block's merge: l, columns
  extern __shared__ __align__(128) unsigned char smemRaw[];
  __shared__ int sAbort, sAbortSeen, sIsLast;
  __shared__ float sHeadTop[kConsumers], sHeadSum[kConsumers];
  __shared__ __align__(8) uint64_t sFull[kMaxStages], sEmpty[kMaxStages];

  const int tid = threadIdx.x;
  DEC_TRACE(0);
  asm volatile("griddepcontrol.wait;" ::: "memory");   // (launched as a programmatic dependent)
  const int split = blockIdx.x, zb = blockIdx.z, by = blockIdx.y;
  int b = by;
  if (p.xWorld > 1) {   // the sequences this rank merges itself come last
    b += p.xRot;
    if (b >= p.batch) b -= p.batch;
  }
  const bool sec = p.hasSecond && by >= p.batch;   // the second attention's blocks
  if (sec) b = by - p.batch;
  const int group = p.qHeads / p.kvHeads, kvh0 = zb * p.kvPerCta, hq = p.kvPerCta * group;
  const int KS = p.keySlots, sliceElems = p.kvPerCta * HD, rowElems = p.kvHeads * HD;
  const int32_t* lens = sec ? p.s2.kvLens : p.kvLens;
  const int64_t seqStride = sec ? p.s2.cacheSeqStride : p.cacheSeqStride;
  const void* const* kPtrs = sec ? p.s2.kPtrs : p.kPtrs;
  const void* const* vPtrs = sec ? p.s2.vPtrs : p.vPtrs;
  const T* kBase = kPtrs ? static_cast<const T*>(kPtrs[b])
                         : static_cast<const T*>(sec ? p.s2.kCache : p.kCache) + (int64_t)b * seqStride;
  const T* vBase = vPtrs ? static_cast<const T*>(vPtrs[b])
                         : static_cast<const T*>(sec ? p.s2.vCache : p.vCache) + (int64_t)b * seqStride;
  const bool misaligned =
      kPtrs && ((reinterpret_cast<uintptr_t>(kBase) | reinterpret_cast<uintptr_t>(vBase)) & 15u);
  kBase += kvh0 * HD;
  vBase += kvh0 * HD;
  const T* qg = static_cast<const T*>(sec ? p.s2.q : p.q) + (int64_t)b * (sec ? p.s2.qRowStride : p.qRowStride) +
                kvh0 * group * HD;
  // (finished rows that the exchange between GPUs sends on are staged; see decode_kernel)
  float* partialsOut = p.partialsOut;
  uint32_t epoch = 0;
  if (p.xWorld > 0) {
    epoch = *reinterpret_cast<volatile uint32_t*>(p.xStep) + 1u;
    partialsOut = p.xStage;
  }

  // L: visible rows of this cache; Lg: the sequence's length (see decode_kernel).
  int64_t lo, end, L = 0, Lg = 0;
  bool hasNew = p.kNew != nullptr && !sec;
  if (p.useRange) {
    lo = p.lo;
    end = p.end;
  } else {
    Lg = L = lens ? lens[b] : sec ? p.s2.kvLen : p.kvLen;
    if (misaligned || (!p.kvSharded && L > (sec ? p.s2.cacheRows : p.cacheRows))) {
      if (tid == 0) atomicOr(p.status, kStatusBadState);
      Lg = L = 0;
      hasNew = false;
    } else if (p.kvSharded) {
      const int64_t local = Lg - p.shardStart;
      hasNew = hasNew && local >= 1 && local <= p.cacheRows;
      L = local < 0 ? 0 : local > p.cacheRows ? p.cacheRows : local;
    }
    end = L - 1;
    lo = Lg - 1 - (sec ? p.s2.wl : p.wl) - p.shardStart;
    if (lo < 0) lo = 0;
    if (hasNew) end -= 1;  // row L-1 is the appended one
    if (L <= 0) { lo = 1; end = -1; }
  }
  const int64_t n = end >= lo ? end - lo + 1 : 0;
  int64_t chunk = (n + p.splits - 1) / p.splits;
  chunk = (chunk + KS - 1) / KS * KS;
  const int64_t s0 = lo + (int64_t)split * chunk, s1 = min(s0 + chunk, end + 1);
  const int ntiles = s1 > s0 ? (int)((s1 - s0 + KS - 1) / KS) : 0;

  // Shared memory: q, the ring (used again for the merge at the end).
  T* sQ = reinterpret_cast<T*>(smemRaw);
  unsigned char* ring = smemRaw + ((hq * HD * (int)sizeof(T) + 127) / 128) * 128;
  const int tileBytes = ((KS * sliceElems * (int)sizeof(T) + 127) / 128) * 128, stages = p.stages;
  if (tid == 0) {
    sAbort = 0;
    sIsLast = 0;
    for (int s = 0; s < stages; s++) {
      mbar_init(smem_u32(&sFull[s]), 1);
      mbar_init(smem_u32(&sEmpty[s]), kConsumerWarps);
    }
    fence_barrier_init();
  }
  __syncthreads();

  if (tid >= kConsumers) {
    // ---------------- producer warp ----------------
    const int lane = tid - kConsumers;
    const uint32_t rowBytes = (uint32_t)sliceElems * sizeof(T);
    for (int it = 0; it < ntiles; it++) {
      const int s = it % stages;
      if (it >= stages && !mbar_park(smem_u32(&sEmpty[s]), ((it / stages) - 1) & 1, &sAbort)) {
        sAbort = 1;
        break;
      }
      const int64_t k0 = s0 + (int64_t)it * KS;
      const int nk = (int)min((int64_t)KS, s1 - k0);
      const uint32_t bar = smem_u32(&sFull[s]);
      const uint32_t dK = smem_u32(ring + (size_t)s * 2 * tileBytes), dV = dK + tileBytes;
      if (lane == 0) mbar_expect_tx(bar, 2u * nk * rowBytes);
      __syncwarp();
      if (sliceElems == rowElems) {
        if (lane == 0) {
          bulk_g2s(dK, kBase + k0 * rowElems, nk * rowBytes, bar);
          bulk_g2s(dV, vBase + k0 * rowElems, nk * rowBytes, bar);
        }
      } else {
        for (int r = lane; r < nk; r += 32) {
          bulk_g2s(dK + r * rowBytes, kBase + (k0 + r) * rowElems, rowBytes, bar);
          bulk_g2s(dV + r * rowBytes, vBase + (k0 + r) * rowElems, rowBytes, bar);
        }
      }
    }
    return;
  }

  // ---------------- consumers ----------------
  // q and, in split 0, the appended row: rotated and rounded to f16 as the separate rope dispatch
  // stores them; the row goes to the cache.
  const bool roped = p.ropeCos != nullptr && !p.useRange && !sec;
  const bool appendHere = hasNew && split == 0 && !p.useRange && L >= 1;
  const int64_t ropeRow = p.ropeByPos ? (Lg >= 1 ? Lg - 1 : 0) : b;
  const float* rc = roped ? p.ropeCos + ropeRow * HD : nullptr;
  const float* rs = roped ? p.ropeSin + ropeRow * HD : nullptr;
  for (int idx = tid; idx < hq * (HD / 2); idx += kConsumers) {
    T r0 = qg[2 * idx], r1 = qg[2 * idx + 1];
    if (roped) {
      const int x = idx % (HD / 2) * 2;
      float f0, f1;
      rope_pair(to_f32<T>(r0), to_f32<T>(r1), rc[x], rs[x], f0, f1);
      r0 = from_f32<T>(f0), r1 = from_f32<T>(f1);
    }
    sQ[2 * idx] = r0;
    sQ[2 * idx + 1] = r1;
  }
  if (appendHere) {
    const T* kn = static_cast<const T*>(p.kNew) + (int64_t)b * p.kNewRowStride + kvh0 * HD;
    const T* vn = static_cast<const T*>(p.vNew) + (int64_t)b * p.vNewRowStride + kvh0 * HD;
    T* kc = const_cast<T*>(kBase) + (L - 1) * rowElems;
    T* vc = const_cast<T*>(vBase) + (L - 1) * rowElems;
    constexpr int kBatch = 4;   // loads ahead of any of their stores, which may alias them for the compiler
    for (int i0 = tid; i0 < sliceElems / 2; i0 += kBatch * kConsumers) {
      T k0[kBatch], k1[kBatch], v0[kBatch], v1[kBatch];
      float c[kBatch], sn[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; i++) {
        const int idx = i0 + i * kConsumers, x = idx % (HD / 2) * 2;
        if (idx < sliceElems / 2) {
          k0[i] = kn[2 * idx], k1[i] = kn[2 * idx + 1];
          v0[i] = vn[2 * idx], v1[i] = vn[2 * idx + 1];
          if (roped) c[i] = rc[x], sn[i] = rs[x];
        }
      }
#pragma unroll
      for (int i = 0; i < kBatch; i++) {
        const int at = 2 * (i0 + i * kConsumers);
        if (at >= sliceElems) break;
        if (roped) {
          float r0, r1;
          rope_pair(to_f32<T>(k0[i]), to_f32<T>(k1[i]), c[i], sn[i], r0, r1);
          k0[i] = from_f32<T>(r0), k1[i] = from_f32<T>(r1);
        }
        kc[at] = k0[i], kc[at + 1] = k1[i];
        vc[at] = v0[i], vc[at + 1] = v1[i];
      }
    }
  }
  named_barrier_sync(1, kConsumers);
  DEC_TRACE(1);

  const int lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int kvl = (tid >> 5) % p.kvPerCta, slot = (tid >> 5) / p.kvPerCta, slots = kConsumerWarps / p.kvPerCta;
  const bool sink = slot == 0 && split == 0 && p.sinks, append = appendHere && slot == 0;
  const int64_t newRow = (L - 1) * rowElems + kvl * HD;
  const MmaQuery<HD> qa(sQ + (kvl * group + g) * HD, g < group, t);
  float m = kNegSeed, l = 0.f, o[M::CHUNKS][M::VEC][2];
#pragma unroll
  for (int c = 0; c < M::CHUNKS; c++)
#pragma unroll
    for (int e = 0; e < M::VEC; e++) o[c][e][0] = o[c][e][1] = 0.f;
  bool ok = true;
  for (int it = 0; it < ntiles; it++) {
    const int s = it % stages;
    ok = __all_sync(0xffffffffu, mbar_park(smem_u32(&sFull[s]), (it / stages) & 1, &sAbort));
    if (!ok) break;   // the whole warp leaves together
    if (it == 0) DEC_TRACE(2);
    const int first = slot * M::KEYS, nk = (int)min((int64_t)KS, s1 - (s0 + (int64_t)it * KS)) - first;
    const T* tK = reinterpret_cast<const T*>(ring + (size_t)s * 2 * tileBytes) + first * sliceElems + kvl * HD;
    if (nk > 0) mma_keys<HD>(tK, tK + tileBytes / (int)sizeof(T), sliceElems, nk, g, t, qa, m, l, o);
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&sEmpty[s]));
  }
  if (!ok) sAbort = 1;
  DEC_TRACE(3);
  // (this block has streamed its keys: the next kernel's blocks may take the freed slots)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (append && ok) mma_keys<HD>(kBase + newRow, vBase + newRow, 0, 1, g, t, qa, m, l, o);
  // A sink joins the finished sums: as the first reference point a dominating one would leave the
  // probabilities no bits.
  if (sink && g < group) {
    const float x = p.sinks[(kvh0 + kvl) * group + g];   // log2-space: sink * ln2 * log2e
    const float top = m > x ? m : x, f = fast_exp2(m - top);   // (a NaN stays one)
    l = l * f + (t == 0 ? fast_exp2(x - top) : 0.f);     // (a head's sum is spread over the four threads of a row)
    m = top;
#pragma unroll
    for (int c = 0; c < M::CHUNKS; c++)
#pragma unroll
      for (int e = 0; e < M::VEC; e++) o[c][e][0] *= f, o[c][e][1] *= f;
  }

  // Whether a wait ran out is decided once for the whole block.
  named_barrier_sync(1, kConsumers);
  if (tid == 0) sAbortSeen = sAbort;
  named_barrier_sync(1, kConsumers);
  if (sAbortSeen) {
    if (tid == 0) {
      atomicOr(p.status, kStatusWaitTimeout);
      if (p.mergeAfter) p.counters[by * gridDim.z + zb] = 1;
    }
    for (int i = 0; i < 64; i++) __nanosleep(4000);
    return;
  }

  // ---- merge the warps that share a head (log-sum-exp), as decode_kernel merges its slots ----
  float* sTop = reinterpret_cast<float*>(ring);   // [slots][hq] maxima
  float* sM = sTop + slots * hq;                  // [slots][hq][MS]
  l += __shfl_xor_sync(0xffffffffu, l, 1);
  l += __shfl_xor_sync(0xffffffffu, l, 2);
  // An output that is not finite is computed again, key by key.
  float probe = 0.f;
#pragma unroll
  for (int c = 0; c < M::CHUNKS; c++)
#pragma unroll
    for (int e = 0; e < M::VEC; e++)
#pragma unroll
      for (int x = 0; x < 2; x++)
        if (c * 8 * M::VEC + M::VEC * (2 * t + x) + e < HD) probe = fmaf(o[c][e][x], 0.f, probe);
  const bool redo = __any_sync(0xffffffffu, g < group && probe != 0.f);
  if (redo) {
    for (int hh = kvl * group; hh < (kvl + 1) * group; hh++) {
      const int at = slot * hq + hh;
      const float top = exact_head<HD>(sQ + hh * HD, kBase + kvl * HD, vBase + kvl * HD, rowElems, s0, s1, KS,
                                       slot * M::KEYS, append ? kBase + newRow : nullptr, vBase + newRow,
                                       sink ? p.sinks[kvh0 * group + hh] : kNegSeed, sink ? 1.f : 0.f, sM + at * MS);
      if (lane == 0) sTop[at] = top;
    }
  } else if (g < group && t == 0) {
    sTop[slot * hq + kvl * group + g] = m;
  }
  named_barrier_sync(1, kConsumers);
  auto top_of = [&](int hh) {
    float top = kNegSeed;
    for (int s = 0; s < slots; s++) top = fmaxf(top, sTop[s * hq + hh]);
    return top;
  };
  if (redo) {
    for (int hh = kvl * group; hh < (kvl + 1) * group; hh++) {
      const float top = top_of(hh), w = fast_exp2(sTop[slot * hq + hh] - top);
      float* r = sM + (slot * hq + hh) * MS;
      for (int x = lane; x < MS; x += 32) r[x] *= w;
      if (slot == 0 && lane == 0) sHeadTop[hh] = top;
    }
  } else if (g < group) {
    const int hh = kvl * group + g;
    const float top = top_of(hh), w = fast_exp2(m - top);
    float* r = sM + (slot * hq + hh) * MS;
    if (t == 0) r[0] = l * w;
#pragma unroll
    for (int c = 0; c < M::CHUNKS; c++)
#pragma unroll
      for (int e = 0; e < M::VEC; e++)
#pragma unroll
        for (int x = 0; x < 2; x++) {
          const int col = c * 8 * M::VEC + M::VEC * (2 * t + x) + e;
          if (col < HD) r[1 + col] = o[c][e][x] * w;
        }
    if (slot == 0 && t == 0) sHeadTop[hh] = top;
  }
  named_barrier_sync(1, kConsumers);

  constexpr int stride = 2 + HD;  // partials row in global memory
  const bool whole = p.splits == 1;
  const int64_t head0 = (int64_t)b * p.qHeads + kvh0 * group;
  float* rowF = !whole ? p.scratch + (((int64_t)by * p.splits + split) * p.qHeads + kvh0 * group) * stride
                       : partialsOut ? partialsOut + head0 * stride : nullptr;
  T* rowT = static_cast<T*>(sec ? p.s2.out : p.out) + head0 * HD;
  for (int hh = tid; hh < hq; hh += kConsumers) {
    const float top = sHeadTop[hh];
    float sum = 0.f;
    for (int s = 0; s < slots; s++) sum += sM[(s * hq + hh) * MS];
    sHeadSum[hh] = sum;
    if (rowF) {
      // finished rows carry the maximum in natural-log units, split rows in log2 units
      rowF[hh * stride] = !whole ? top : sum > 0.f ? top * 0.6931471805599453f : kNegSeed;
      rowF[hh * stride + 1] = sum;
    }
  }
  named_barrier_sync(1, kConsumers);
  for (int i = tid; i < hq * HD; i += kConsumers) {
    const int hh = i / HD, x = i - hh * HD;
    const float* r = sM + hh * MS + 1 + x;
    float v = 0.f;
    for (int s = 0; s < slots; s++) v += r[s * hq * MS];
    if (rowF) {
      rowF[hh * stride + 2 + x] = v;
    } else {
      const float sum = sHeadSum[hh];
      rowT[i] = from_f32<T>(v * (sum > 0.f ? 1.f / sum : 0.f));
    }
  }
  DEC_TRACE(4);
  if (whole) {
    if (p.xWorld > 0) exchange_rows(p, b, hq, kvh0 * group, tid, epoch, gridDim.z);
    return;
  }
  if (p.mergeAfter) return;   // a launch of its own merges the splits
  __threadfence();
  named_barrier_sync(1, kConsumers);
  if (tid == 0) sIsLast = atomicAdd(&p.counters[by * gridDim.z + zb], 1u) == (unsigned)p.splits - 1;
  named_barrier_sync(1, kConsumers);
  if (!sIsLast) return;
  __threadfence();
  merge_splits<T>(HD, p.splits, p.qHeads, p.scratch + ((int64_t)by * p.splits * p.qHeads + kvh0 * group) * stride,
                  rowT, partialsOut ? partialsOut + head0 * stride : nullptr, hq, sM, slots * hq * MS);
  if (tid == 0) p.counters[by * gridDim.z + zb] = 0;  // ready for the next launch
  if (p.xWorld > 0) exchange_rows(p, b, hq, kvh0 * group, tid, epoch, gridDim.z);
}

// The merge of the splits as a launch of its own, one block per (sequence, query head):
// what the last block of a sequence does when there is little of it.
constexpr int kMergeThreads = 128;
template <typename T>
__global__ void __launch_bounds__(kMergeThreads)
merge_kernel(const DecodeParams p) {
  __shared__ float sW[64], sInv;
  const int h = blockIdx.x, b = blockIdx.y, hd = p.hd, stride = 2 + hd, splits = p.splits;
  const int zBlocks = (p.kvHeads + p.kvPerCta - 1) / p.kvPerCta;
  const int zb = h / (p.qHeads / p.kvHeads) / p.kvPerCta;
  asm volatile("griddepcontrol.wait;" ::: "memory");   // the attention's partials are complete
  if (__ldcg(p.counters + b * zBlocks + zb) != 0) return;   // a block gave up: its rows are no partials
  const int64_t row = (int64_t)b * p.qHeads + h;
  const float* src = p.scratch + ((int64_t)b * splits * p.qHeads + h) * stride;
  const int64_t ss = (int64_t)p.qHeads * stride;       // between splits
  float* partials = p.partialsOut ? p.partialsOut + row * stride : nullptr;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const bool a = lane < splits, c = lane + 32 < splits;
    const float m0 = a ? __ldcg(src + lane * ss) : kNegSeed, l0 = a ? __ldcg(src + lane * ss + 1) : 0.f;
    const float m1 = c ? __ldcg(src + (lane + 32) * ss) : kNegSeed, l1 = c ? __ldcg(src + (lane + 32) * ss + 1) : 0.f;
    const float M = warp_max(fmaxf(m0, m1));
    const float w0 = fast_exp2(m0 - M), w1 = fast_exp2(m1 - M);
    const float L = warp_sum(fmaf(l0, w0, l1 * w1));
    sW[lane] = w0, sW[lane + 32] = w1;
    if (lane == 0) {
      sInv = L > 0.f ? 1.f / L : 0.f;
      if (partials) partials[0] = L > 0.f ? M * 0.6931471805599453f : kNegSeed, partials[1] = L;
    }
  }
  __syncthreads();
  const int x = threadIdx.x;
  if (x >= hd) return;
  float o = 0.f;
#pragma unroll 16
  for (int s = 0; s < splits; s++) o = fmaf(__ldcg(src + s * ss + 2 + x), sW[s], o);
  if (partials) partials[2 + x] = o;
  else static_cast<T*>(p.out)[row * hd + x] = from_f32<T>(o * sInv);
}

template <typename T>
cudaError_t launch_merge(const DecodeParams& p, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.qHeads, p.batch);
  cfg.blockDim = dim3(kMergeThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, merge_kernel<T>, p);
}

size_t smem_bytes(const DecodeParams& p, int esize, int hdp, bool bulk) {
  const int group = p.qHeads / p.kvHeads;
  const int hqMax = p.kvPerCta * group;
  const bool staged = p.lanesPerRow <= 1;   // see the kernel's carve-up
  const size_t qBytes = p.mma   ? (((size_t)hqMax * p.hd * esize + 127) / 128) * 128
                        : staged ? (((size_t)hqMax * q_stride(hdp) * 4 + 127) / 128) * 128
                                 : 0;
  const size_t tileBytes = (((size_t)p.keySlots * p.kvPerCta * p.hd * esize + 127) / 128) * 128;
  const size_t ringBytes = (size_t)(bulk ? p.stages : 1) * 2 * tileBytes;
  const int lanes = p.lanesPerRow > 1 ? p.lanesPerRow : 1;
  const int slots = p.mma ? kConsumerWarps / p.kvPerCta : p.keySlots;
  const size_t mergeBytes = (size_t)slots * hqMax * lanes * (2 + hdp / lanes) * 4;
  const size_t newBytes = (staged && p.kNew && !p.mma) ? 2 * ((((size_t)p.kvPerCta * p.hd * esize) + 127) / 128) * 128 : 0;
  return qBytes + newBytes + (ringBytes > mergeBytes ? ringBytes : mergeBytes);
}

int padded_hd(int hd) { return hd <= 32 ? 32 : hd <= 64 ? 64 : 128; }
bool exact_hd(int hd) { return hd == 36 || hd == 52 || hd == 64 || hd == 128; }

bool aligned16(const void* ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 15u) == 0; }

// The bulk (TMA) path needs 16-byte aligned rows and slices.
bool bulk_ok(const DecodeParams& p, int esize) {
  if (!exact_hd(p.hd)) return false;
  const int64_t rowBytes = (int64_t)p.kvHeads * p.hd * esize;
  const int64_t sliceBytes = (int64_t)p.kvPerCta * p.hd * esize;
  if (rowBytes % 16 || sliceBytes % 16) return false;
  // (separately allocated caches are checked by the kernel, sequence by sequence)
  if (!p.kPtrs && ((p.cacheSeqStride * esize) % 16 || !aligned16(p.kCache) || !aligned16(p.vCache)))
    return false;
  if (p.hasSecond && !p.s2.kPtrs &&
      ((p.s2.cacheSeqStride * esize) % 16 || !aligned16(p.s2.kCache) || !aligned16(p.s2.vCache)))
    return false;
  if (p.kvHeads % p.kvPerCta) return false;  // a ragged last block changes the slice size
  return true;
}

cudaError_t launch_kernel(void (*kern)(DecodeParams), bool bulk, const DecodeParams& p, size_t smem, cudaStream_t s) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int zBlocks = (p.kvHeads + p.kvPerCta - 1) / p.kvPerCta;
  dim3 grid(p.splits, p.batch * (p.hasSecond ? 2 : 1), zBlocks);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(bulk ? kConsumers + 32 : kConsumers);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, p);
}

template <typename T, int HDP, bool EXACT, int VEC, bool BULK, int R = 1>
cudaError_t launch_one(const DecodeParams& p, size_t smem, cudaStream_t s) {
  return launch_kernel(decode_kernel<T, HDP, EXACT, VEC, BULK, R>, BULK, p, smem, s);
}

template <typename T>
cudaError_t launch_typed(const DecodeParams& p, cudaStream_t s) {
  constexpr int esize = sizeof(T);
  constexpr int V = sizeof(T) == 2 ? 8 : 4;   // widest vector for the exact paths
  if (bulk_ok(p, esize)) {
    const size_t smem = smem_bytes(p, esize, p.hd, true);
    if (p.mma) {
      switch (p.hd) {
        case 36: return launch_kernel(decode_mma_kernel<36>, true, p, smem, s);
        case 52: return launch_kernel(decode_mma_kernel<52>, true, p, smem, s);
        case 64: return launch_kernel(decode_mma_kernel<64>, true, p, smem, s);
        case 128: return launch_kernel(decode_mma_kernel<128>, true, p, smem, s);
      }
    }
    switch (p.hd) {
      case 36: return launch_one<T, 36, true, 4, true>(p, smem, s);
      case 52: return launch_one<T, 52, true, 4, true>(p, smem, s);
      case 64:
        return p.lanesPerRow == 2 ? launch_one<T, 64, true, V, true, 2>(p, smem, s)
                                  : launch_one<T, 64, true, V, true>(p, smem, s);
      case 128:
        return p.lanesPerRow == 4 ? launch_one<T, 128, true, V, true, 4>(p, smem, s)
                                  : launch_one<T, 128, true, V, true>(p, smem, s);
    }
  }
  if (p.lanesPerRow > 1 || p.mma) return cudaErrorInvalidValue;   // the plan promised the bulk path
  const int hdp = padded_hd(p.hd);
  const size_t smem = smem_bytes(p, esize, hdp, false);
  if (hdp == 32) return launch_one<T, 32, false, 1, false>(p, smem, s);
  if (hdp == 64) return launch_one<T, 64, false, 1, false>(p, smem, s);
  return launch_one<T, 128, false, 1, false>(p, smem, s);
}

// Which f16 calls go to the tensor cores, by measurement (B200, us among launches, FP32 pipes / tensor cores).
// With several query heads on a kv head the FP32 pipes read and convert every key once per query
// head: 16 sequences of 2000 keys, 32 heads of 128 on 8: 75.9 / 34.9; 64 x 100, 8 of 128 on one: 14.2 / 6.8;
// 64 x 2000, 32 of 64 on 8: 112.8 / 64.3; 64 x 448, 64 of 36 on 8: 46.6 / 27.1.
//   - Heads of less than 64 need four query heads on a warp's kv head, or two where a block's warps
//     share kv heads: 64 x 2000, 16 of 36 on 8 43.6 / 52.7, of 52 51.0 / 59.7; 8 of 52 on 4 30.2 / 32.3, 64 x 100 8.4 / 7.9.
//     At worst 16 x 448, 32 of 36 on 8: 14.5 / 16.9, 16 of 64 on 8, one of 448 11.4 / 12.4.
//   - With one query head each, wide heads and many of them gain from tiles of 16 keys and 8 heads where the
//     other kernel's hold all heads of two to four keys: up to 64 MB (32 heads of 128, 64 x 50 keys
//     29.4 / 22.9, 4 x 400 19.6 / 15.8; 16 heads up to 48), and up to 160 where the blocks are few (4 x 2500 40.7 / 40.4, 64 heads, 4 x 800
//     34.8 / 30.9) or fill the chip once or twice (32 x 256 33.1 / 32.2, 64 x 160 48.4 / 43.8).  Else a wave of them is half
//     empty (24 x 256 28.7 / 31.9, 16 x 600 37.5 / 41.2), or long rows stream as well (16 x 2000 87.7 / 88).
bool mma_better(const DecodeParams& p, int group) {
  if (group > 8 || (p.kvHeads % 8 && p.kvHeads != 4 && p.kvHeads != 2 && p.kvHeads != 1)) return false;
  const int heads = p.kvHeads < 8 ? p.kvHeads : 8;   // kv heads of a block
  if (p.hd < 64) return group > 1 && group * (8 / heads) >= 4;
  if (group > 1) return true;
  if (p.hd != 128 || p.kvHeads <= 8) return false;
  constexpr int64_t kSms = 148;
  const int64_t blocks = (int64_t)p.batch * (p.kvHeads / heads) * (p.hasSecond ? 2 : 1);
  const int64_t rows = p.useRange ? p.end - p.lo + 1 : p.kvLen, bytes = p.batch * rows * p.kvHeads * p.hd * 4;
  const bool fills = blocks <= 2 * kSms && blocks * 20 >= (blocks + kSms - 1) / kSms * kSms * 17;   // 85 %
  const bool wide = p.kvHeads >= 32;
  return bytes <= ((wide ? 64ll : 48ll) << 20) || (bytes <= (160ll << 20) && (blocks <= (wide ? 48 : 8) || fills));
}

}  // namespace

bool plan_decode(DecodeParams& p, int dtype, int smCount, std::string* err, bool tensorCores) {
  const int esize = dtype == RT_F16 ? 2 : 4;
  const int group = p.qHeads / p.kvHeads;
  if (group > kConsumers) {
    *err = "decode: more than 256 query heads per kv head";
    return false;
  }
  const int hdp = padded_hd(p.hd);
  // Head size 64 and 128: 2 or 4 threads share a (key, head) pair, 32 columns each (see
  // process_key_sub); that needs the bulk path, so fall back to whole rows without it.
  int lanes = p.hd == 128 ? 4 : p.hd == 64 ? 2 : 1;
  if (group * lanes > kConsumers) lanes = 1;
  // One geometry for a given shared-memory budget per CTA.
  struct Geom {
    int kvPerCta, keySlots, stages;
    size_t tile;
    bool fits;
  };
  auto geometry = [&](size_t budgetTotal, int lanesNow) {
    const int wdp = hdp / lanesNow;   // columns per thread
    Geom g{};
    g.kvPerCta = p.kvHeads;
    while (g.kvPerCta * group * lanesNow > kConsumers) g.kvPerCta = (g.kvPerCta + 1) / 2;
    // Key slots per tile: 256 threads' worth, fewer when two stages of that many keys do not
    // fit.  The heads stay together as long as a handful of key slots fit (wide heads then
    // leave some threads idle): a CTA that owns all the heads fetches a tile with one bulk
    // copy per tensor, while one that owns a single head needs a copy of hd elements per
    // key — measured 1.0 TB/s at 32 heads x 128, the copy engine's rate for 256-byte copies.
    constexpr int kMinKeySlots = 4;
    size_t budget;
    for (;;) {
      const size_t qBytes = lanesNow > 1 ? 128 :   // sub-row threads stage neither q nor the new row
                            (size_t)g.kvPerCta * group * q_stride(hdp) * 4 + 128 +
                            (p.kNew ? 2 * ((size_t)g.kvPerCta * p.hd * esize + 128) : 0);
      budget = budgetTotal > qBytes ? budgetTotal - qBytes : 0;
      g.keySlots = kConsumers / (g.kvPerCta * group * lanesNow);
      const size_t perSlot = 2ull * g.kvPerCta * p.hd * esize;            // K+V bytes of one key
      const size_t mergePerSlot = (size_t)g.kvPerCta * group * lanesNow * (2 + wdp) * 4;
      const size_t capTile = budget / 2 > 256 ? (budget / 2 - 256) / perSlot : 0;   // two stages must fit
      const size_t capMerge = budget / mergePerSlot;
      const size_t cap = capTile < capMerge ? capTile : capMerge;
      if (cap < (size_t)(g.keySlots < kMinKeySlots ? g.keySlots : kMinKeySlots) && g.kvPerCta > 1) {
        g.kvPerCta = (g.kvPerCta + 1) / 2;
        continue;
      }
      g.fits = cap >= 1;
      if (g.fits && (size_t)g.keySlots > cap) g.keySlots = (int)cap;
      break;
    }
    g.tile = ((2ull * g.keySlots * g.kvPerCta * p.hd * esize + 255) / 256) * 256 + 256;
    const int stages = g.fits ? (int)(budget / g.tile) : 0;
    g.stages = stages < 2 ? 2 : stages > kMaxStages ? kMaxStages : stages;
    return g;
  };
  // Up to 64 columns per thread, two CTAs fit an SM (registers), each with half of the
  // shared memory: one's set-up and merge overlap the other's streaming.  Sub-row threads
  // with only a few sequences to work on do better with one CTA per SM and a deep ring
  // (fewer, longer key splits; two tiles per barrier round): measured at 32 heads x 128,
  // KV 4096, 8 / 16 / 32 / 64 sequences: 147 / 195 / 261 / 249 us with one against
  // 270 / 286 / 234 / 248 us with two; the same crossing at 8 heads and at head size 64.
  Geom g{};
  int ctasPerSm = 1;
  // f16 on the tensor cores: eight warps deal with eight kv heads, or with fewer of them and more
  // keys.
  auto mma_geometry = [&](size_t budget) {
    Geom of{};
    of.kvPerCta = p.kvHeads % 8 == 0 ? 8 : p.kvHeads;
    const int slots = kConsumerWarps / of.kvPerCta;
    of.keySlots = (p.hd <= 64 ? 32 : 16) * slots;
    of.tile = 2ull * of.kvPerCta * p.hd * esize * of.keySlots + 256;
    const size_t qBytes = (size_t)of.kvPerCta * group * p.hd * esize + 128;
    const size_t rest = budget > qBytes ? budget - qBytes : 0;
    of.stages = (int)(rest / of.tile);
    if (of.stages > kMaxStages) of.stages = kMaxStages;
    of.fits = of.stages >= 3 && (size_t)slots * of.kvPerCta * group * (2 + p.hd) * 4 <= rest;
    return of;
  };
  p.mma = 0;
  if (tensorCores && dtype == RT_F16 && exact_hd(p.hd) && mma_better(p, group)) {
    g = mma_geometry(kSmemBudgetMma);
    p.kvPerCta = g.kvPerCta;
    if (g.fits && bulk_ok(p, esize)) {
      p.mma = 1;
      p.lanesPerRow = 1;
      const Geom two = mma_geometry(kSmemBudgetTwoPerSm);
      if (p.hd <= 64 && two.fits && (int64_t)p.batch * (p.kvHeads / g.kvPerCta) * (p.hasSecond ? 2 : 1) > smCount) {
        g = two;
        ctasPerSm = 2;
      }
    }
  }
  for (; !p.mma; lanes = 1) {
    const bool twoFit = hdp / lanes <= 64;
    const Geom one = geometry(kSmemBudget, lanes);
    g = one;
    ctasPerSm = 1;
    if (twoFit) {
      const Geom two = geometry(kSmemBudgetTwoPerSm, lanes);
      const int64_t seqCtas = (int64_t)p.batch * ((p.kvHeads + one.kvPerCta - 1) / one.kvPerCta);
      // Fewer blocks than SMs (a decode step of a small batch): a block alone on its SM takes
      // the whole shared memory for a ring twice as deep or more, and a block's copy rate is
      // what its ring keeps in flight over the memory latency (measured: 63 GB/s with two
      // 36 KB stages).
      const bool alone = seqCtas * (p.hasSecond ? 2 : 1) <= smCount;
      const bool fewSequences = one.fits && ((lanes > 1 && seqCtas * 8 <= smCount) || alone);
      if (two.fits && !fewSequences) {
        g = two;
        ctasPerSm = 2;
      }
    }
    p.kvPerCta = g.kvPerCta;
    p.lanesPerRow = lanes;
    if (lanes > 1 && !(g.fits && bulk_ok(p, esize))) continue;   // once more with whole rows
    if (!g.fits) {
      *err = "decode: heads too wide for shared memory";
      return false;
    }
    break;
  }
  const int kvPerCta = g.kvPerCta, keySlots = g.keySlots;
  p.kvPerCta = kvPerCta;
  p.keySlots = keySlots;
  p.stages = g.stages;

  if (p.splits <= 0) {
    const int zBlocks = (p.kvHeads + kvPerCta - 1) / kvPerCta;
    const int64_t ctas = (int64_t)p.batch * (p.hasSecond ? 2 : 1) * zBlocks;
    int64_t nmax = p.useRange ? (p.end >= p.lo ? p.end - p.lo + 1 : 0) : p.kvLen;
    if (p.hasSecond && p.s2.kvLen > nmax) nmax = p.s2.kvLen;
    if (p.kvSharded) {   // the longest stretch of a sequence this shard can hold
      nmax -= p.shardStart;
      nmax = nmax < 1 ? 1 : nmax > p.cacheRows ? p.cacheRows : nmax;
    }
    if (!p.useRange && p.wl < nmax) nmax = (int64_t)p.wl + 1;
    // At least one full tile per split, or, for the tensor cores' tiles of 16 keys and more, a begun one:
    // a few keys over a whole number of tiles else make two of every split (100 keys, 16 heads of 128 on 8,
    // 16.1 us in six splits of up to two tiles, 10.7 in seven of one).
    int64_t maxS = (nmax + (p.mma ? keySlots - 1 : 0)) / keySlots;
    if (maxS > 64) maxS = 64;
    if (maxS < 1) maxS = 1;
    // Cost in eighths of one tile's streaming time: every CTA pays a fixed set-up,
    // pipeline-fill and merge cost (about three tiles' worth, measured), CTAs run in
    // waves of `resident` at a time, and splitting adds the partials pass, three tiles and an
    // eighth per split.  Measured on B200: with at least one wave of sequences, not splitting is
    // fastest; alone, a sequence of 415 keys takes 12.9 / 10.2 / 9.1 us in 1 / 3 / 13 splits, one of
    // 1250 keys 28.3 / 10.4 / 12.2 in 1 / 20 / 39, one of 4096 keys x 32 heads of 128 50 / 35 in
    // 32 / 64.
    const int64_t resident = (int64_t)smCount * ctasPerSm;
    int best = 1;
    int64_t bestCost = INT64_MAX;
    for (int s = 1; s <= maxS; s++) {
      const int64_t tilesPerCta = (nmax + (int64_t)s * keySlots - 1) / ((int64_t)s * keySlots);
      const int64_t waves = (ctas * s + resident - 1) / resident;
      const int64_t cost = 8 * waves * (3 + tilesPerCta) + (s > 1 ? 24 + s : 0);
      if (cost < bestCost) {
        bestCost = cost;
        best = s;
      }
    }
    p.splits = best;
  }
  // One block reads a sequence's partials at about 11 GB/s (latency: 24 us for 18 splits of 32 heads
  // of 128), a launch of its own takes 3 us whatever there is to read.  The exchange between GPUs
  // sends the merged rows on from the attention's own blocks, and a layer's two attentions
  // promise to be one launch.
  constexpr int64_t kMergeFloats = 8192;
  p.mergeAfter = p.splits > 1 && p.xWorld == 0 && !p.hasSecond && (int64_t)p.splits * p.qHeads * p.hd > kMergeFloats;
  return true;
}

cudaError_t launch_decode(const DecodeParams& p, int dtype, cudaStream_t s) {
  const cudaError_t e = dtype == RT_F16 ? launch_typed<__half>(p, s) : launch_typed<float>(p, s);
  if (e != cudaSuccess || !p.mergeAfter) return e;
  return dtype == RT_F16 ? launch_merge<__half>(p, s) : launch_merge<float>(p, s);
}

}  // namespace rt

// ---- decode without any allocation ---------------------------------------------
//
// Some hosts of this library must not allocate device memory when they call it:
// a real-time audio or serving loop that has pinned its memory budget up front,
// a plugin that runs inside another framework's memory pool, or code that runs
// while the device allocator is locked.  rt_attn_decode needs a context, and a
// context allocates (its stream, its status word, and the split scratch that
// grows on demand).  This entry point runs the same decode kernel with no
// context: the split scratch, the arrival counters and the status word live in
// the fixed-size device array below, which every GPU that loads the library
// holds until the process exits.
namespace rt {
namespace {

constexpr size_t kStaticScratchFloats = 1u << 20;   // 4 MiB of (m, l, acc) partials
constexpr size_t kStaticCounters = 4096;            // one per (sequence, head block)

struct StaticDecodeArea {
  float partials[kStaticScratchFloats];
  unsigned counters[kStaticCounters];
  int status;
};

static __device__ __align__(256) StaticDecodeArea gStaticDecodeArea;

constexpr int kMaxDevices = 64;
std::mutex gStaticMutex;
StaticDecodeArea* gStaticAddr[kMaxDevices];  // device address of the area, per device
int gStaticSmCount[kMaxDevices];

// Recorded where rt_last_error(NULL) finds it: this entry point has no context.
int static_fail(int code, const std::string& msg) {
  set_thread_error(msg.c_str());
  return code;
}

// The current device's copy of the area.  Set-up, once per device, with that device
// current: in host code the array's name is only a handle, the kernel needs its device
// address.
int static_area(StaticDecodeArea** area, int* smCount) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess)
    return static_fail(RT_EXECUTION_FAILED, std::string("cudaGetDevice: ") + cudaGetErrorString(e));
  if (device < 0 || device >= kMaxDevices)
    return static_fail(RT_UNSUPPORTED_DEVICE, "rt_attn_decode_noalloc: device ordinal " +
                                                  std::to_string(device) + " is past the " +
                                                  std::to_string(kMaxDevices) +
                                                  " devices this entry point keeps an address for");
  std::lock_guard<std::mutex> lock(gStaticMutex);
  if (!gStaticAddr[device]) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, gStaticDecodeArea);
    if (e != cudaSuccess || !ptr)
      return static_fail(RT_EXECUTION_FAILED,
                         std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    int sms = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e != cudaSuccess || sms < 1)
      return static_fail(RT_EXECUTION_FAILED,
                         std::string("cudaDeviceGetAttribute: ") + cudaGetErrorString(e));
    gStaticSmCount[device] = sms;
    gStaticAddr[device] = static_cast<StaticDecodeArea*>(ptr);
  }
  *area = gStaticAddr[device];
  *smCount = gStaticSmCount[device];
  return RT_OK;
}

}  // namespace
}  // namespace rt

extern "C" {

int rt_attn_decode_noalloc_status(void* cuda_stream) {
  using namespace rt;
  StaticDecodeArea* area;
  int smCount;
  if (int s = static_area(&area, &smCount)) return s;
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  cudaError_t e = cudaStreamSynchronize(stream);
  int status = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&status, &area->status, sizeof(int), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess)
    return static_fail(RT_EXECUTION_FAILED,
                       std::string("rt_attn_decode_noalloc_status: ") + cudaGetErrorString(e));
  if (status == 0) return RT_OK;
  cudaMemset(&area->status, 0, sizeof(int));
  return static_fail(RT_EXECUTION_FAILED,
                     (status & kStatusWaitTimeout)
                         ? "rt_attn_decode_noalloc: a bounded device-side wait ran out"
                         : "rt_attn_decode_noalloc: a kvLens entry exceeds cacheRows");
}

int rt_attn_decode_noalloc(const rt_decode_args* a, void* cuda_stream) {
  using namespace rt;
  if (!a) return static_fail(RT_INVALID_ARGUMENT, "rt_attn_decode_noalloc: args is NULL");
  if (!a->q || (!a->kCache && !a->kCachePtrs) || (!a->vCache && !a->vCachePtrs) ||
      (!a->out && !a->partialsOut))
    return static_fail(RT_INVALID_ARGUMENT,
                       "rt_attn_decode_noalloc: q, kCache, vCache and out (or partialsOut) must be "
                       "device pointers");
  if (a->dtype != RT_F32 && a->dtype != RT_F16)
    return static_fail(RT_INVALID_ARGUMENT, "rt_attn_decode_noalloc: dtype is neither f32 nor f16");
  if (a->exchange)
    return static_fail(RT_INVALID_ARGUMENT,
                       "rt_attn_decode_noalloc: the cross-GPU exchange needs rt_attn_decode");
  if (a->batch < 1 || a->batch > 65535 || a->cacheRows < 1 || a->qHeads < 1 || a->headDim < 1 ||
      a->headDim > 128 || a->kvHeads < 1 || a->qHeads % a->kvHeads != 0 || a->kvLen < 0 ||
      (!a->kvSharded && a->kvLen > a->cacheRows) || (!a->kvLens && a->kvLen < 1) || a->windowLeft < 0 ||
      a->splits < 0 || a->splits > 64 || (a->kNew == nullptr) != (a->vNew == nullptr) ||
      a->cacheSeqStride < 0 ||
      (!a->kCachePtrs && a->batch > 1 &&
       a->cacheSeqStride < (int64_t)a->cacheRows * a->kvHeads * a->headDim) ||
      decode_rope_args_error(*a) != nullptr)
    return static_fail(RT_INVALID_ARGUMENT,
                       "rt_attn_decode_noalloc: a size or option is out of range (same rules as "
                       "rt_attn_decode)");

  StaticDecodeArea* area;
  int smCount;
  cudaError_t e;
  if (int s = static_area(&area, &smCount)) return s;

  DecodeParams p{};
  decode_params_from_args(*a, p);
  std::string err;
  if (!plan_decode(p, a->dtype, smCount, &err)) return static_fail(RT_INVALID_ARGUMENT, err);
  const size_t zBlocks = (size_t)(p.kvHeads + p.kvPerCta - 1) / p.kvPerCta;
  const size_t sets = p.hasSecond ? 2 : 1;
  const size_t perSplit = sets * p.batch * p.qHeads * (2 + p.hd);
  const size_t fit = kStaticScratchFloats / perSplit;
  if (a->splits == 0 && (size_t)p.splits > fit && fit >= 2) {
    p.splits = (int)fit;   // the plan's own choice: as many as the area holds
    if (!plan_decode(p, a->dtype, smCount, &err)) return static_fail(RT_INVALID_ARGUMENT, err);
  }
  if (a->splits == 0 && p.mma && fit < 2) {
    // No room for two splits: what runs is what the FP32 kernel would run unsplit, whichever kernel
    // it then is.  (By their own plan the tensor cores would split, and so refuse, 275 sequences of
    // 2048 keys with 64 heads of 36 on 32.)
    DecodeParams simt = p;
    simt.splits = 0;
    if (!plan_decode(simt, a->dtype, smCount, &err, false)) return static_fail(RT_INVALID_ARGUMENT, err);
    p.splits = simt.splits;
    if (!plan_decode(p, a->dtype, smCount, &err)) return static_fail(RT_INVALID_ARGUMENT, err);
  }
  const size_t needFloats = p.splits > 1 ? p.splits * perSplit : 0;
  const size_t needCounters = p.splits > 1 ? sets * p.batch * zBlocks : 0;
  if (needFloats > kStaticScratchFloats || needCounters > kStaticCounters)
    return static_fail(
        RT_INVALID_ARGUMENT,
        "rt_attn_decode_noalloc: batch*splits*qHeads*(2+headDim) = " + std::to_string(needFloats) +
            " floats (limit " + std::to_string(kStaticScratchFloats) + ") or batch*headBlocks = " +
            std::to_string(needCounters) + " counters (limit " + std::to_string(kStaticCounters) +
            ") exceeds the fixed scratch; pass fewer splits or a smaller batch");
  cudaStream_t stream = static_cast<cudaStream_t>(cuda_stream);
  // The area keeps the last call's contents.  Partials are fully rewritten
  // before they are read; the arrival counters must start at zero.
  if (needCounters) {
    e = cudaMemsetAsync(area->counters, 0, needCounters * sizeof(unsigned), stream);
    if (e != cudaSuccess)
      return static_fail(RT_EXECUTION_FAILED,
                         std::string("cudaMemsetAsync: ") + cudaGetErrorString(e));
  }
  p.scratch = area->partials;
  p.counters = area->counters;
  p.status = &area->status;
  e = launch_decode(p, a->dtype, stream);
  if (e != cudaSuccess)
    return static_fail(RT_EXECUTION_FAILED, std::string("decode launch: ") + cudaGetErrorString(e));
  return RT_OK;
}

}  // extern "C"
