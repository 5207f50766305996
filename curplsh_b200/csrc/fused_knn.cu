// fused_knn.cu -- the fused distance + candidate-filter pass on the 5th-gen
// tensor cores (sm_100a).
//
// Replaces, in one kernel, the reference's per-tile chain (cuRPLSH paths):
//   matrixMultiply / cublasSgemm        src/internal/matrix_ops.cu:8-60   (-2 q.x)
//   l2Select (+ ||x||^2, top-k)         src/internal/select.cu:189-224
//   adjustIndices                       src/internal/search.cu:21-42      (tile -> global row)
// The Q x N distance matrix never leaves the SM: each 128-query x 256-row
// tile is accumulated in TMEM, read back by the epilogue warps, compared with a
// per-query bound and only the survivors are appended to a per-query candidate
// pool in global memory.
//
// Roles (320 threads, one CTA per SM, persistent over a balanced schedule):
//   warp 0      TMA producer: query block (resident, or streamed per K chunk)
//               and database tiles, 128-byte-swizzled, into a stage ring.
//   warp 1      allocates 512 TMEM columns (two accumulator slots of 128 x 256,
//               or with dual blocks of two 128 x 128) and issues tcgen05.mma from
//               one elected lane of a uniform warp; commits release stages and
//               publish accumulators.
//   warps 2..9  epilogue: two warpgroups; thread = one query (TMEM lane).  With
//               dual blocks each warpgroup owns one query block, else one
//               128-column half of every tile.  A warp takes the minimum of
//               every eight columns, and only where one is under its query's
//               bound looks at the columns and appends survivors to the pool; it
//               radix-selects a pool that is about to overflow, keeping the k'
//               smallest (distance, row) keys, and publishes the tightened bound
//               to the shared per-query bound array so other CTAs working on the
//               same queries filter harder.
//
// Schedule: the (query block, database tile) space is flattened and split into
// equal contiguous ranges, one per CTA, so the work is balanced to one tile for
// any Q, N.  A range covers a few "units" = (query block, tile sub-range).
#include <cuda.h>

#include <cstdio>

#include "common.cuh"
#include <algorithm>
#include <atomic>

#include "fused_knn.h"
#include "ptx.cuh"
#include "select.cuh"

namespace curplsh_b200 {

// ------------------------------------------------------------------ forms
template <int FORM>
struct FormTraits;
template <>
struct FormTraits<kFormExact> {
  static constexpr int kAParts = 2, kBParts = 2, kProducts = 3;
  static constexpr int kChunkElems = 64, kStepElems = 16;  // bf16
  static constexpr bool kFP8 = false, kRowScales = false;
  static constexpr bool kFolded = true;  // norms ride in the augmented K columns
  // products: hi*hi, hi*lo, lo*hi  (the lo*lo term, O(2^-16) relative, is dropped)
  __device__ static constexpr int a_part(int p) { return p == 2 ? 1 : 0; }
  __device__ static constexpr int b_part(int p) { return p == 1 ? 1 : 0; }
};
template <>
struct FormTraits<kFormBF16> {
  static constexpr int kAParts = 1, kBParts = 1, kProducts = 1;
  static constexpr int kChunkElems = 64, kStepElems = 16;
  static constexpr bool kFP8 = false, kRowScales = false;
  static constexpr bool kFolded = true;
  __device__ static constexpr int a_part(int) { return 0; }
  __device__ static constexpr int b_part(int) { return 0; }
};
// The FP8 form's kernels for databases with per-row scales: no norm tails, the
// norms and scales are applied in the epilogue.  A form of its own at compile
// time: as a run-time branch it cost the tiles with tails a sixth of their pass
// (FP8 sphere 17.5 -> 14.8 ms).
constexpr int kFormFP8Rows = 3;
struct FP8Traits {
  static constexpr int kAParts = 1, kBParts = 1, kProducts = 1;
  static constexpr int kChunkElems = 128, kStepElems = 32;  // e4m3
  static constexpr bool kFP8 = true;
  static constexpr bool kFolded = false;  // the accumulator is d / (2 s_q s), or needs norms and scales
  __device__ static constexpr int a_part(int) { return 0; }
  __device__ static constexpr int b_part(int) { return 0; }
};
template <>
struct FormTraits<kFormFP8> : FP8Traits {
  static constexpr bool kRowScales = false;
};
template <>
struct FormTraits<kFormFP8Rows> : FP8Traits {
  static constexpr bool kRowScales = true;
};

// FILL: eights of a warp's 16 with survivors from which 32 columns are taken at a
// time (one query, 100,000 rows, k' = 1,024: pass 43 -> 25 us; 6 and 9 alike).
constexpr int kDenseEights = 6;
// FILL: keys that a pool may end its unit with.
__host__ __device__ constexpr int end_limit(int kprime) { return kprime + kprime / 4; }

constexpr uint32_t kAChunkBytes = kBM * kChunkBytes;  // 16 KB
constexpr uint32_t kBChunkBytes = kBN * kChunkBytes;  // 32 KB
// A narrow tail chunk holds the last <= 16 BF16 columns (the augmented norm
// columns when d is a multiple of 64): 32-byte rows, 32-byte swizzle.
constexpr uint32_t kTailRowBytes = 32;
constexpr uint32_t kATailBytes = kBM * kTailRowBytes;  // 4 KB
constexpr uint32_t kBTailBytes = kBN * kTailRowBytes;  // 8 KB

// ------------------------------------------------------------------ smem layout
struct SmemLayout {
  int kdim;            // K extent of the MMA (d, plus kAugCols for the folded forms)
  int nkc;             // K chunks (128 bytes of K each, except a narrow tail)
  int tail_narrow;     // 1: the last chunk is a 16-column, 32-byte-swizzled tail
  int a_stream;        // 1: query chunks travel with each stage
  uint32_t a_bytes;    // resident query block bytes (0 when streamed)
  uint32_t stage_bytes;
  int stages;
  uint32_t bar_off;    // offset of the barrier block
  uint32_t hist_off;   // warp-private radix histograms
  uint32_t pool_off;   // per-row candidate pool counts and bounds
  uint32_t total;      // dynamic smem bytes requested (includes 1 KB alignment slack)
  uint32_t b_chunk;    // bytes of one B part of a K chunk (this CTA's database rows)
  uint32_t a_block;    // bytes between the two resident query blocks (dual)
  uint32_t b_tail;     // bytes of the B tail chunk
};

// pair = 1: this CTA holds half of each 256-row database tile (CTA pairs);
// epi_warps: epilogue warps (each has a 1 KB histogram / staging area);
// dual = 1: two resident query blocks (a_block bytes apart) and 128-row tiles.
__host__ __device__ inline SmemLayout make_layout(int form, int d, int pair = 0, int epi_warps = kEpiWarps,
                                                  int dual = 0) {
  SmemLayout L{};
  L.b_chunk = (pair || dual) ? kBChunkBytes / 2 : kBChunkBytes;
  L.b_tail = (pair || dual) ? kBTailBytes / 2 : kBTailBytes;
  const bool folded = form != kFormFP8 && form != kFormFP8Rows;
  const int chunk_elems = folded ? 64 : 128;
  const int a_parts = (form == kFormExact) ? 2 : 1;
  const int b_parts = (form == kFormExact) ? 2 : 1;
  L.kdim = folded ? d + kAugCols : d;
  L.nkc = (L.kdim + chunk_elems - 1) / chunk_elems;
  // narrow tail only when it holds nothing but the norm columns (d % 64 == 0):
  // the tail runs the hi x hi product alone, which is exact only for those.
  // FP8 rows: the norm tail, when the 32-byte steps of the codes fill the chunks
  // (without a tail such dimensions loaded norms in the epilogue: 4,096 queries,
  // 10^6 rows, d = 256 2.81 -> 1.46 ms, d = 512 2.98 -> 1.87).
  L.tail_narrow = folded ? d % 64 == 0 : form == kFormFP8 && (d + 31) / 32 % 4 == 0;
  if (!folded && L.tail_narrow) ++L.nkc;
  // everything below the barrier block must fit the 227 KB opt-in limit
  const uint32_t pool_bytes = dual ? 0u : 1024u;  // counts and bounds of 128 shared pools
  const uint32_t warp_bytes = (uint32_t)epi_warps * 1024u;  // radix histograms
  const uint32_t budget = 227u * 1024u - 256u - warp_bytes - pool_bytes - 1024u;
  const int nreg = L.nkc - (L.tail_narrow ? 1 : 0);
  const uint32_t a_one = (uint32_t)nreg * a_parts * kAChunkBytes + (L.tail_narrow ? kATailBytes : 0u);
  L.a_block = (a_one + 1023u) & ~1023u;
  const uint32_t a_res = dual ? 2u * L.a_block : a_one;
  // a stage = one regular K chunk of the tile; the last one also carries the tail
  const uint32_t b_stage = (uint32_t)b_parts * L.b_chunk + (L.tail_narrow ? L.b_tail : 0u);
  if (((a_res + 1023u) & ~1023u) + 2 * b_stage <= budget) {
    L.a_stream = 0;
    L.a_bytes = (a_res + 1023u) & ~1023u;
    L.stage_bytes = b_stage;
  } else {
    L.a_stream = 1;
    L.a_bytes = 0;
    L.stage_bytes = b_stage + (uint32_t)a_parts * kAChunkBytes + (L.tail_narrow ? kATailBytes : 0u);
  }
  L.stage_bytes = (L.stage_bytes + 1023u) & ~1023u;
  int s = (int)((budget - L.a_bytes) / L.stage_bytes);
  L.stages = s < 2 ? 2 : (s > 8 ? 8 : s);
  L.bar_off = L.a_bytes + (uint32_t)L.stages * L.stage_bytes;
  L.hist_off = L.bar_off + 256;  // barriers: 2*8 + 6 mbarriers + tmem slot + flags < 256 B
  L.pool_off = L.hist_off + warp_bytes;
  L.total = L.pool_off + pool_bytes + 1024;
  return L;
}

// Offset of resident query chunk `kc`, part `part` (0 hi, 1 lo); the narrow
// tail (kc = nkc-1) has a part 0 only.
__device__ __forceinline__ uint32_t a_res_off(const SmemLayout& L, int kc, int part, int a_parts) {
  return (uint32_t)(kc * a_parts + part) * kAChunkBytes;
}

// Offsets inside a stage: B parts, then streamed A parts, then the tail (B, A).
template <int kAP, int kBP>
__device__ __forceinline__ uint32_t stage_a_off(const SmemLayout& L, int part) {
  return (uint32_t)kBP * L.b_chunk + (uint32_t)part * kAChunkBytes;
}
template <int kAP, int kBP>
__device__ __forceinline__ uint32_t stage_tail_off(const SmemLayout& L) {
  return (uint32_t)kBP * L.b_chunk + (L.a_stream ? (uint32_t)kAP * kAChunkBytes : 0u);
}

// ------------------------------------------------------------------ schedule
// Launch arguments: the batch header, then per-item scalars and tensor maps.
template <int MAXI>
struct FusedArgs {
  FusedBatch B;
  FusedItem items[MAXI];
  CUtensorMap maps[MAXI * kMapsPerItem];
};

// Walks the contiguous range [cta*W, min(total,(cta+1)*W)) of the flattened
// (item, query block, tile position) space as units (item, query block,
// [t0, t1)); positions map to database tiles through a per-block rotation.  A
// unit also ends at every multiple of the item's split length L, so no unit
// gathers candidates from more than L tiles (a split-N knob: longer units
// mean fewer pool lists for the merge but more in-pool selections).
// u_ord numbers the units of one query block: the number of cuts (CTA range
// starts and multiples of L) in (0, t0].  A position that is both kinds of
// cut leaves one ordinal unused (`gap`): that unit writes zero counts for it.
// With CTA pairs the space counts query groups of two blocks and a range
// belongs to a pair; each CTA of the pair gets its own block of the group
// (block = 2 * group + rank) and the same tiles.
struct UnitWalk {
  long long pos, end, W;
  int ii, shift, rank;
  __device__ UnitWalk(int cta, const FusedBatch& B, uint32_t cta_rank)
      : W(B.work_per_cta), ii(0), shift(B.pair | B.dual), rank((int)cta_rank) {
    pos = (long long)(cta >> B.pair) * W;
    end = pos + W < B.total_work ? pos + W : B.total_work;
  }
  template <int MAXI>
  __device__ bool next(const FusedArgs<MAXI>& A, int& item, int& qb, int& t0, int& t1, int& u_ord, bool& gap,
                       int& rot) {
    if (pos >= end) return false;
    while (ii < A.B.num_items && A.items[ii].work_end <= pos) ++ii;
    if (ii >= A.B.num_items) return false;
    const FusedItem& it = A.items[ii];
    const long long wb = it.work_begin;
    const int T = it.num_tiles;
    const int Ls = it.split_tiles;
    const long long lp = pos - wb;
    qb = (int)(lp / T);
    t0 = (int)(lp - (long long)qb * T);
    long long len = (end - pos) < (long long)(T - t0) ? (end - pos) : (long long)(T - t0);
    if (len > (long long)(Ls - t0 % Ls)) len = Ls - t0 % Ls;
    t1 = t0 + (int)len;
    const long long base = wb + (long long)qb * T;
    u_ord = (int)(pos / W - base / W) + t0 / Ls;
    gap = t0 > 0 && t0 % Ls == 0 && pos % W == 0;
    // Position j of the block is database tile (j - rot) mod T, where rot is
    // where the first CTA range starting inside this block begins: every such
    // CTA then reads tiles 0, 1, 2, ... from the start, in step with the
    // others, so concurrent CTAs share the database tiles in L2 (a contiguous
    // assignment alone would have them at spread-out offsets).
    {
      const long long first = (base + W - 1) / W * W - base;
      rot = first < T ? (int)first : 0;
    }
    item = ii;
    qb = (qb << shift) + rank;
    pos += len;
    return true;
  }
};

// Bounded wait that also gives up as soon as another role has aborted.
// `cl`: the arrivals come from the other CTA of a pair (acquire at cluster scope).
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                              bool cl = false) {
  auto poll = [&]() { return cl ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity); };
  // the timer is read only once a wait has already gone on for a while
  for (int i = 0; i < 16; ++i)
    if (poll()) return true;
  const uint64_t t0 = globaltimer_ns();
  for (uint32_t i = 0; i < kWaitPollLimit; ++i) {
    if (poll()) return true;
    if ((i & 255u) == 255u) {
      if (*abort_flag) return false;
      if (globaltimer_ns() - t0 > kWaitTimeoutNs) return false;
    }
  }
  return false;
}

__device__ __forceinline__ void raise_abort(volatile int* abort_flag, uint32_t* status, uint32_t code) {
  *abort_flag = 1;
  atomicOr(status, code);
}

// Filter bound on d' = ||x||^2 - 2 q.x for a pool whose k'-th key distance is
// dstar: keys store fl(d' + ||q||^2), so admit d' <= dstar - ||q||^2 with a
// few-ulp slack; admitting slightly more never changes the selected set, which
// is decided by exact key order.
__device__ __forceinline__ float bound_to_thr(float dstar, float qn) {
  return (dstar - qn) + (fabsf(dstar) + fabsf(qn)) * 4.76837158203125e-7f;  // 2^-21
}

// Filter threshold for a bound `dstar` on the key distance.  The folded forms
// compare the accumulator, which is the key distance itself, so the bound is
// used as is; the FP8 form compares ||x||^2 - 2 q.x and needs bound_to_thr.
template <bool kFolded>
__device__ __forceinline__ float thr_from(float dstar, float qn) {
  return kFolded ? dstar : bound_to_thr(dstar, qn);
}

// Instrumentation (compiled in only with -DCURPLSH_FUSED_STATS): per-role
// cycle counters accumulated in registers and added to B.stats at exit.
#ifdef CURPLSH_FUSED_STATS
#define STAT_DECL(name) unsigned long long name = 0
#define STAT_BEGIN(t) const long long t = clock64()
#define STAT_END(t, acc) acc += (unsigned long long)(clock64() - t)
#define STAT_INC(acc, v) acc += (unsigned long long)(v)
#define STAT_FLUSH(slot, acc) \
  if (B.stats) atomicAdd(&B.stats[slot], acc)
#else
#define STAT_DECL(name)
#define STAT_BEGIN(t)
#define STAT_END(t, acc)
#define STAT_INC(acc, v)
#define STAT_FLUSH(slot, acc)
#endif

// The filter admits a column iff its distance is <= thr.  With u = the float just
// above thr that is d < u, and for the scaled FP8 form (d = km x, km > 0) the sign
// of fma(km, x, -u): one rounding never changes the sign of a nonzero
// difference, km x == u gives +0, and a NaN never passes, as with a compare.
__device__ __forceinline__ float next_above(float x) {
  const uint32_t u = __float_as_uint(x);
  if (u == 0x80000000u) return __uint_as_float(1u);  // -0: the smallest positive subnormal
  return __uint_as_float((int32_t)u >= 0 ? u + 1u : u - 1u);
}
template <bool kScaled>
__device__ __forceinline__ bool passes(float x, float km, float u) {
  return kScaled ? fmaf(km, x, -u) < 0.f : x < u;
}
// (acc << 1) | (t >> 31)
__device__ __forceinline__ uint32_t shl1_sign(uint32_t acc, uint32_t t) {
  uint32_t r;
  asm("shf.l.wrap.b32 %0, %1, %2, 1;" : "=r"(r) : "r"(t), "r"(acc));
  return r;
}
// bit j set iff km x[j] < u, j < N: a packed FMA per two columns, the sign bits
// gathered by one chain of funnel shifts
template <int N>
__device__ __forceinline__ uint32_t survive_mask(const float* x, float km, float u) {
  float t[N];
#pragma unroll
  for (int i = 0; i < N / 2; ++i) fma2_f32(t[2 * i], t[2 * i + 1], x[2 * i], x[2 * i + 1], km, km, -u, -u);
  uint32_t a = __float_as_uint(t[N - 1]) >> 31;
#pragma unroll
  for (int i = N - 2; i >= 0; --i) a = shl1_sign(a, __float_as_uint(t[i]));
  return a;
}
// smallest of 8 (NaN ignored): four instructions
__device__ __forceinline__ float min8(const float* x) {
  return fminf(fmin3(fmin3(fmin3(x[0], x[1], x[2]), x[3], x[4]), x[5], x[6]), x[7]);
}
// x[j] for a runtime j in [0, 8) without local memory: a 3-level select tree
__device__ __forceinline__ float select8(const float* x, int j) {
  const float a0 = (j & 4) ? x[4] : x[0], a1 = (j & 4) ? x[5] : x[1];
  const float a2 = (j & 4) ? x[6] : x[2], a3 = (j & 4) ? x[7] : x[3];
  const float b0 = (j & 2) ? a2 : a0, b1 = (j & 2) ? a3 : a1;
  return (j & 1) ? b1 : b0;
}

// x[j] for a runtime j in [0, 32)
__device__ __forceinline__ float select32(const float* x, int j) {
  const float a = (j & 8) ? select8(x + 8, j & 7) : select8(x, j & 7);
  const float b = (j & 8) ? select8(x + 24, j & 7) : select8(x + 16, j & 7);
  return (j & 16) ? b : a;
}

// ------------------------------------------------------------------ kernel
// MINIMA selects the block-minimum mode (FusedItem::minima, the sample pass of
// the bound estimate) at compile time, so the candidate-pool kernel carries
// none of its code.
// PAIR selects the CTA-pair kernel: a kernel that contains cta_group::2
// instructions can only be launched as clusters of two, so the single-CTA
// kernel is a separate instance without them.
// DUAL: two query blocks resident per CTA; each 128-row database tile feeds two
// 128 x 128 MMAs (one per block), so a tile crosses L2 -> SM once per 256
// queries without coupling CTAs; warp g of a lane group filters block g.
// FILL: pools that start without a bound (few rows, the estimate off, the
// allocation-free call).  Most eights of a tile then hold survivors until the
// pools' own bounds are tight, so the survivor code takes 32 columns at a time,
// and a bound that another CTA found is worth asking for at every tile.  An
// instance of its own: within the bounded kernel this code cost the FP8 sphere's
// pass 1.3 %.
template <int FORM, int MAXI, bool MINIMA = false, bool PAIR = false, bool DUAL = false, bool FILL = false>
__global__ void __launch_bounds__(kNumThreads, 1) fused_knn_kernel(const __grid_constant__ FusedArgs<MAXI> A) {
  static_assert(!(PAIR && DUAL) && !(DUAL && MINIMA), "dual blocks: single CTAs, candidate pools");
  static_assert(!(FILL && MINIMA), "block minima have no pools");
  using Tr = FormTraits<FORM>;
  const FusedBatch& B = A.B;
  // a conditional pass (a re-search after a failed check): every thread of
  // every CTA reads the same flag, written by an earlier launch on the stream,
  // and leaves before any barrier or TMEM allocation when it is zero
  if (B.run_if) {
    griddep_wait();
    if (*B.run_if == 0) return;
  }
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  constexpr int EW = kEpiWarps;
  const SmemLayout L = make_layout(FORM, B.d, PAIR ? 1 : 0, EW, DUAL ? 1 : 0);
  constexpr int kTileRows = DUAL ? kBN / 2 : kBN;  // database rows per tile
  constexpr int kQB = DUAL ? 2 : 1;                // resident query blocks
  const int S = L.stages;
  // CTA pairs: rank 0 issues the MMAs and owns the barriers the pair's loads
  // complete on; each CTA loads and filters its own query block
  constexpr bool pair = PAIR;
  uint32_t rank = 0u;
  if constexpr (PAIR) rank = cluster_ctarank();
  const bool issuer = rank == 0;

  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L.bar_off);
  uint64_t* full = bars;            // [8]
  uint64_t* empty = bars + 8;       // [8]
  uint64_t* a_full = bars + 16;
  uint64_t* a_empty = bars + 17;
  uint64_t* acc_full = bars + 18;   // [2]
  uint64_t* acc_empty = bars + 20;  // [2]
  uint64_t* drain = bars + 22;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 23);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 24);
  uint32_t* hist_all = reinterpret_cast<uint32_t*>(smem + L.hist_off);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  STAT_BEGIN(t_kernel);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(a_full, 1);
    mbar_init(a_empty, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], pair ? 2 * EW : EW);  // both CTAs' epilogue warps
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_barrier_init();
    fence_proxy_async_smem();
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      tmem_alloc_pair(tmem_slot, 512);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, 512);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  // a pair's barriers must be initialised before the other CTA's loads and
  // arrivals can reach them
  if constexpr (PAIR)
    cluster_sync();
  else
    __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // The prologue above touches nothing an earlier kernel writes.  This kernel does
  // not let its own successor in early: merge CTAs resident beside the epilogue
  // slowed it (284 queries, FP8, k' = 480: search 200 -> 260 us).
  griddep_wait();

  const int KC = Tr::kChunkElems;
  auto maps_of = [&](int ii) { return &A.maps[(MAXI == 1 ? 0 : ii) * kMapsPerItem]; };

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      fence_proxy_async();  // query operands written by the preparation kernel
      const uint64_t pol_db = l2_policy_evict_first();
      const uint64_t pol_q = l2_policy_evict_last();
      // a pair's loads complete on rank 0's barriers, which expect both CTAs' bytes
      auto load = [&](void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, uint64_t pol) {
        if constexpr (PAIR)
          tma_load_2d_pair(dst, m, bar, c0, c1, pol);
        else
          tma_load_2d(dst, m, bar, c0, c1, pol);
      };
      const uint32_t tx_mul = pair ? 2u : 1u;
      const int half_row = pair ? (int)rank * (kBN / 2) : 0;  // this CTA's rows of a tile
      UnitWalk walk(blockIdx.x, B, rank);
      int ii, qb, t0, t1, u_ord, rot, unit = 0;
      bool gap;
      uint32_t it = 0, q_loads = 0;  // stages and query blocks loaded
      bool ok = true;
      STAT_DECL(st_wait);
      while (ok && walk.next(A, ii, qb, t0, t1, u_ord, gap, rot)) {
        const CUtensorMap* mp = maps_of(ii);
        const CUtensorMap& tm_q_hi = mp[kMapQHi];
        const CUtensorMap& tm_q_lo = mp[kMapQLo];
        const CUtensorMap& tm_x_hi = mp[kMapXHi];
        const CUtensorMap& tm_x_lo = mp[kMapXLo];
        const CUtensorMap& tm_q_tail = mp[kMapQTail];
        const CUtensorMap& tm_x_tail = mp[kMapXTail];
        if (!L.a_stream) {
          if (unit > 0 && !wait_or_abort(a_empty, (unit - 1) & 1, abort_flag)) {
            raise_abort(abort_flag, B.status, kErrWaitTimeout);
            ok = false;
            break;
          }
          const int nreg = L.nkc - (L.tail_narrow ? 1 : 0);
          ++q_loads;
          if (issuer)
            mbar_arrive_expect_tx(a_full, tx_mul * (uint32_t)kQB *
                                              ((uint32_t)nreg * Tr::kAParts * kAChunkBytes +
                                               (L.tail_narrow ? kATailBytes : 0u)));
          for (int j = 0; j < kQB; ++j) {
            uint8_t* ab = smem + (uint32_t)j * L.a_block;
            const int qrow = (qb + j) * kBM;
            for (int kc = 0; kc < nreg; ++kc)
              for (int part = 0; part < Tr::kAParts; ++part)
                load(ab + a_res_off(L, kc, part, Tr::kAParts), part ? &tm_q_lo : &tm_q_hi, a_full, kc * KC, qrow,
                     pol_q);
            if (L.tail_narrow)
              load(ab + a_res_off(L, nreg, 0, Tr::kAParts), &tm_q_tail, a_full, nreg * KC, qrow, pol_q);
          }
        }
        const int nreg = L.nkc - (L.tail_narrow ? 1 : 0);
        for (int t = t0; t < t1 && ok; ++t) {
          const int T_i = A.items[MAXI == 1 ? 0 : ii].num_tiles;
          const int tile = (t - rot + T_i) % T_i;  // database tile of position t
          const int tx_row = tile * kTileRows + half_row;
          const FusedItem& p = A.items[MAXI == 1 ? 0 : ii];
          // column of a phased sample's row in its map (make_map)
          const int col0 = MINIMA && p.db_phased ? sample_phase(tile, p.db_step) * p.db_phased : 0;
          for (int kc = 0; kc < nreg; ++kc, ++it) {
            const int s = (int)(it % (uint32_t)S);
            STAT_BEGIN(tw);
            if (!wait_or_abort(&empty[s], ((it / S) & 1u) ^ 1u, abort_flag)) {
              raise_abort(abort_flag, B.status, kErrWaitTimeout);
              ok = false;
              break;
            }
            STAT_END(tw, st_wait);
            uint8_t* st = smem + L.a_bytes + (uint32_t)s * L.stage_bytes;
            const bool with_tail = L.tail_narrow && kc == nreg - 1;
            uint32_t tx = (uint32_t)Tr::kBParts * L.b_chunk + (L.a_stream ? (uint32_t)Tr::kAParts * kAChunkBytes : 0u);
            if (with_tail) tx += L.b_tail + (L.a_stream ? kATailBytes : 0u);
            if (issuer) mbar_arrive_expect_tx(&full[s], tx_mul * tx);
            for (int part = 0; part < Tr::kBParts; ++part)
              load(st + part * L.b_chunk, part ? &tm_x_lo : &tm_x_hi, &full[s], col0 + kc * KC, tx_row, pol_db);
            if (L.a_stream)
              for (int part = 0; part < Tr::kAParts; ++part)
                load(st + stage_a_off<Tr::kAParts, Tr::kBParts>(L, part), part ? &tm_q_lo : &tm_q_hi, &full[s],
                     kc * KC, qb * kBM, pol_q);
            if (with_tail) {
              uint8_t* tl = st + stage_tail_off<Tr::kAParts, Tr::kBParts>(L);
              load(tl, &tm_x_tail, &full[s], col0 + nreg * KC, tx_row, pol_db);
              if (L.a_stream) load(tl + L.b_tail, &tm_q_tail, &full[s], nreg * KC, qb * kBM, pol_q);
            }
          }
        }
        ++unit;
      }
      // After an abort nobody consumes the last loads, so this role waits for
      // their bytes itself (a pair's complete on rank 0's barriers): the shared
      // memory must not change hands under a copy.  Otherwise it has nothing
      // else to do until the MMAs are through.
      if (issuer) {
        bool landed = q_loads == 0 || mbar_wait(a_full, (q_loads - 1) & 1u);
        for (uint32_t i = it > (uint32_t)S ? it - (uint32_t)S : 0u; landed && i < it; ++i)
          landed = mbar_wait(&full[i % (uint32_t)S], (i / (uint32_t)S) & 1u);
      }
      STAT_FLUSH(kStatProducerWaitEmpty, st_wait);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    // The whole warp runs this role, so that addresses, descriptors and loop
    // counters are warp-uniform values (the tensor-core instructions take them
    // from uniform registers); one elected lane issues.  From a single diverged
    // lane an MMA took 230-280 cycles of issue, two to four times its
    // execution, and the issue bound the pass (full pass, diverged -> uniform:
    // FP8 sphere 28.1 -> 26.8 ms, BF16 integer mixture 3.39 -> 3.22, FP32-exact
    // 5.89 -> 5.58, d = 960 0.71 -> 0.61).
    if (issuer) {
      const bool leader = elect_one();
      constexpr uint32_t fmt = Tr::kFP8 ? 0u : 1u;  // e4m3 : bf16
      // a pair's MMA is 256 rows: this CTA's query block, then the partner's
      constexpr uint32_t kM = PAIR ? 2 * kBM : kBM, kN = DUAL ? kBN / 2 : kBN;
      constexpr uint32_t idesc = make_idesc(fmt, fmt, kM, kN);
      // the norm columns' step: the same shape, BF16 operands
      constexpr uint32_t idesc16 = make_idesc(1u, 1u, kM, kN);
      constexpr int kSteps = Tr::kChunkElems / Tr::kStepElems;
      static_assert(kSteps == 4, "K steps of a chunk");
      auto steps = [&](int n, uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t acc) {
        if (n >= 4)
          mma_steps<Tr::kFP8, PAIR, 4>(d, a_lo, b_lo, kDescHiSw128, idesc, acc);
        else if (n == 3)
          mma_steps<Tr::kFP8, PAIR, 3>(d, a_lo, b_lo, kDescHiSw128, idesc, acc);
        else if (n == 2)
          mma_steps<Tr::kFP8, PAIR, 2>(d, a_lo, b_lo, kDescHiSw128, idesc, acc);
        else
          mma_steps<Tr::kFP8, PAIR, 1>(d, a_lo, b_lo, kDescHiSw128, idesc, acc);
      };
      // (leader only) completion goes to the barrier at the same offset in both
      // CTAs of a pair
      auto commit = [&](uint64_t* bar) {
        if constexpr (PAIR)
          mma_commit_pair(bar);
        else
          mma_commit(bar);
      };
      // Everything a tile's issue needs, in descriptor units of 16 bytes
      const uint32_t smem_base = smem_u32(smem);
      const int nreg = L.nkc - (L.tail_narrow ? 1 : 0);
      const int last_steps = (L.kdim - (nreg - 1) * KC + Tr::kStepElems - 1) / Tr::kStepElems;  // >= 4: whole
      const uint32_t b_first = desc_lo(smem_base + L.a_bytes), stage16 = L.stage_bytes >> 4;
      const uint32_t a_block16 = L.a_block >> 4;
      constexpr uint32_t kA16 = kAChunkBytes >> 4;
      const uint32_t b_chunk16 = L.b_chunk >> 4;
      // queries: resident at a_first + chunk, or in the stage at b + a_in_stage
      const uint32_t a_first = desc_lo(smem_base), a_in_stage = stage_a_off<Tr::kAParts, Tr::kBParts>(L, 0) >> 4;
      const uint32_t tail16 = stage_tail_off<Tr::kAParts, Tr::kBParts>(L) >> 4;
      UnitWalk walk(blockIdx.x, B, rank);
      int ii, qb, t0, t1, u_ord, rot, unit = 0;
      bool gap;
      int s = 0;                 // ring stage, its phase and descriptor
      uint32_t sphase = 0, tc = 0, b_lo = b_first;
      bool ok = true;
      STAT_DECL(st_full);
      STAT_DECL(st_acc);
      while (ok && walk.next(A, ii, qb, t0, t1, u_ord, gap, rot)) {
        // The lanes wait one by one and may disagree at a time-out or an abort;
        // the vote at the end of every chunk makes them leave together (a lane
        // that left alone would strand the others at their next warp barrier).
        bool got = true;
        if (!L.a_stream) {
          got = wait_or_abort(a_full, unit & 1, abort_flag);
          tc_fence_after();
        }
        // The norm columns' K step (hi x hi alone carries them: lo rows are zero
        // there): the 32-byte-swizzled narrow tail after the last chunk, or the
        // FP8 rows' 32 bytes inside it (a K step of its 128-byte swizzled rows, as
        // the FP8 steps before it), into the same FP32 accumulator.  A norm tail
        // is BF16 in every form.
        const int fp8_tail = Tr::kFP8 ? A.items[MAXI == 1 ? 0 : ii].fp8_tail : 0;
        const bool tail = Tr::kFP8 ? !Tr::kRowScales : L.tail_narrow != 0;
        const uint32_t tail_hi = L.tail_narrow ? kDescHiSw32 : kDescHiSw128;
        const uint32_t in_chunk16 = (uint32_t)(fp8_tail - (nreg - 1) * KC) >> 4;
        const uint32_t tail_b = L.tail_narrow ? tail16 : in_chunk16;
        const uint32_t tail_a = L.a_stream ? (L.tail_narrow ? tail16 + (L.b_tail >> 4) : a_in_stage + in_chunk16)
                                : L.tail_narrow ? (a_res_off(L, nreg, 0, Tr::kAParts) >> 4)
                                                : (a_res_off(L, nreg - 1, 0, Tr::kAParts) >> 4) + in_chunk16;
        for (int t = t0; t < t1 && ok; ++t, ++tc) {
          const uint32_t slot = tc & 1u, use = tc >> 1;
          STAT_BEGIN(ta);
          got = got && wait_or_abort(&acc_empty[slot], (use & 1u) ^ 1u, abort_flag, pair);
          STAT_END(ta, st_acc);
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + slot * kBN;
          uint32_t a_lo = a_first;
          for (int kc = 0; kc < nreg; ++kc) {
            STAT_BEGIN(tf);
            got = got && wait_or_abort(&full[s], sphase, abort_flag);
            STAT_END(tf, st_full);
            tc_fence_after();
            if (L.a_stream) a_lo = b_lo + a_in_stage;
            const bool last = kc == nreg - 1;
            const int n = last ? last_steps : kSteps;
            if (leader && got) {
#pragma unroll
              for (int j = 0; j < kQB; ++j) {  // dual: block j accumulates into columns j * 128 of the slot
                const uint32_t dj = d_tmem + (uint32_t)j * (kBN / 2);
#pragma unroll
                for (int pr = 0; pr < Tr::kProducts; ++pr)
                  steps(n, dj, a_lo + (uint32_t)j * a_block16 + (uint32_t)Tr::a_part(pr) * kA16,
                        b_lo + (uint32_t)Tr::b_part(pr) * b_chunk16, pr ? 1u : (uint32_t)kc);
                if (last && tail)
                  mma_steps<false, PAIR, 1>(dj, (L.a_stream ? b_lo : a_first) + tail_a + (uint32_t)j * a_block16,
                                            b_lo + tail_b, tail_hi, idesc16, 1u);
              }
              commit(&empty[s]);
              if (last) commit(&acc_full[slot]);
            }
            if (__any_sync(0xffffffffu, !got)) {
              if (!got) raise_abort(abort_flag, B.status, kErrWaitTimeout);
              ok = false;
              break;
            }
            a_lo += Tr::kAParts * kA16;
            b_lo += stage16;
            if (++s == S) {
              s = 0;
              sphase ^= 1u;
              b_lo = b_first;
            }
          }
        }
        if (ok && leader && !L.a_stream) commit(a_empty);
        __syncwarp();
        ++unit;
      }
      // Make sure every issued MMA has retired before TMEM is released (in
      // both CTAs of a pair: the commit reaches the partner's drain barrier).
      if (leader) commit(drain);
      __syncwarp();
      mbar_wait(drain, 0);
      __syncwarp();
      if (lane == 0) {
        STAT_FLUSH(kStatMmaWaitFull, st_full);
        STAT_FLUSH(kStatMmaWaitAccEmpty, st_acc);
      }
    } else if (lane == 0 && pair) {
      // the partner's MMAs also write this CTA's TMEM and read its shared
      // memory: wait for its final commit before the teardown
      mbar_wait(drain, 0);
    }
  } else {
    // ------------------------------------------------------------ epilogue
    // Warps ew and ew + 4 read the same TMEM lanes (queries); warp g takes the
    // 64-column chunks 2g and 2g + 1 of an accumulator slot.
    //   Single blocks: the two warps split each tile's columns and share ONE
    // candidate pool per (query, unit): appends reserve slots with a
    // shared-memory counter, and at every S-th tile end the pair meets at a
    // named barrier, splits the pools that need a selection between them, and
    // meets again.  A shared pool sees all of a tile's rows, so its bound
    // tightens as one pool over the whole tile would -- about half the survivors
    // and selections of a pool per half.
    //   Dual blocks (OWN): warp g filters query block qb + g alone, so a lane
    // owns its query's pool: its count and bound live in registers and the
    // warps meet nowhere.  CTA pairs do the same with two pools per query, one
    // per warp (kLists): an accumulator waits for both CTAs' warps, so what the
    // warps wait for each other is paid twice (FP32-exact integer mixture as
    // pairs: full pass 5.30 -> 4.72 ms).  Pairs whose pools start without a bound
    // share them all the same: two pools fill with twice the keys (FP32-exact, d =
    // 256, k' = 32, 3,000 rows, 1,000 queries: pass 106 us, 281 with two).  Block
    // minima need no pool at all.
    constexpr bool OWN = DUAL || (PAIR && !FILL) || MINIMA;
    constexpr int kLists = PAIR && !FILL ? 2 : 1;
    const int ew = warp - 2;       // 0..EW-1
    const int g = ew >> 2;         // this warp's index within its lane group
    const int lg = warp & 3;       // TMEM lane group this warp may access
    const int row = lg * 32 + lane;
    const int pair_bar = 1 + lg;   // named barrier of the two warps of lane group lg
    constexpr int kGroupThreads = 64;
    uint32_t* hist = hist_all + ew * 256;
    int* cnt_s = reinterpret_cast<int*>(smem + L.pool_off);             // [128] pool counts (single blocks)
    float* thr_s = reinterpret_cast<float*>(smem + L.pool_off) + kBM;   // [128] pool bounds
    const uint32_t lane_base = (uint32_t)(lg * 32) << 16;
    UnitWalk walk(blockIdx.x, B, rank);
    int ii, qb, t0, t1, u_ord, rot;
    bool gap;
    uint32_t tc = 0;
    bool ok = true;
    STAT_DECL(st_wait);
    STAT_DECL(st_filter);
    STAT_DECL(st_refresh);
    STAT_DECL(st_nref);
    STAT_DECL(st_surv);
    STAT_DECL(st_slow);
    STAT_DECL(st_iters);
    STAT_DECL(st_bar);
#ifdef CURPLSH_FUSED_STATS
    if (threadIdx.x == 64 && B.stats) g_radix_pass_counter = &B.stats[kStatRadixPasses];
#endif
    while (ok && walk.next(A, ii, qb, t0, t1, u_ord, gap, rot)) {
      const FusedItem& p = A.items[MAXI == 1 ? 0 : ii];  // one item: constants at fixed addresses
      const int P = p.pool_cap;
      const int U = p.units_per_block;
      const int S = OWN ? 1 : pool_sync_tiles(P, p.kprime);
      // At a unit's end pools above k' are selected, so that the merge reads little
      // beyond what it needs.  Short units end with some more in every pool, and
      // a selection of most of its keys frees nothing for its 10 us (k' = 224, 3,000
      // rows, 1,000 queries: pass 256 us, 44 without).
      const int end_lim = FILL ? end_limit(p.kprime) : p.kprime;
      if (u_ord < 0 || u_ord >= U) {  // identical in every epilogue warp: both of a pair leave here
        raise_abort(abort_flag, B.status, kErrBadSchedule);
        ok = false;
        break;
      }
      const int qbw = DUAL ? qb + g : qb;  // this warp's query block
      const int q = qbw * kBM + row;
      const bool valid = q < p.nq;
      const float qn = valid ? p.q_norms[q] : 0.f;
      // FP8: d = ||x||^2 + 2 s_q s_x acc (the query codes are stored negated)
      float s2 = 2.f;
      if (Tr::kFP8) s2 = valid ? 2.f * p.q_scale[q] : 0.f;
      // FP8 with one scale s for every database row and the norm tails: the
      // accumulator is d / ku, ku = 2 s_q s; the filter compares ku acc with the
      // bound and scales only the survivors (km = 1: the accumulator is d itself
      // or is made d below)
      constexpr bool fold = Tr::kFP8 && !Tr::kRowScales;
      const float ku = s2 * p.db_scale_uniform;
      const float km = fold ? ku : 1.f;
      auto key_d = [&](float x) -> float { return Tr::kFolded ? x : fmaf(km, x, qn); };
      const size_t pool_row0 = (size_t)qbw * kBM;  // pool index of lane-group row 0 is added per lane
      auto list_of = [&](int r) -> size_t {
        return ((pool_row0 + (size_t)r) * U + (size_t)u_ord) * kLists + (kLists > 1 ? g : 0);
      };
      auto pool_of = [&](int r) -> uint64_t* {
        return p.pools + list_of(r) * (size_t)P;
      };
      uint64_t* pool = pool_of(row);
      // a new unit starts with an empty pool (the previous unit's last barrier
      // ordered every use of the old state before this)
      int own_cnt = 0;
      if constexpr (!OWN) {
        if (g == 0) {
          cnt_s[row] = 0;
          thr_s[row] = 3.402823466e38f;
        }
        bar_sync_named(pair_bar, kGroupThreads);
      }
      // FLT_MAX admits every finite distance until a pool fills; a padding row
      // of the last query block admits none
      float thr = valid ? 3.402823466e38f : -__builtin_huge_valf();

      // Selections of the pools in `need` (lane bits of this lane group; of a
      // shared pool's two warps, warp g owns those of lanes l with l mod 2 = g,
      // so two warps never touch the same pool's state).  Each keeps `keep`
      // keys, records the pool's new count and bound and publishes a full
      // set's k'-th distance to q_bound.
      auto refresh = [&](uint32_t need, int keep) {
        STAT_BEGIN(tr);
        while (need) {
          const int src = __ffs(need) - 1;
          need &= need - 1;
          STAT_INC(st_nref, 1);
          const int r = lg * 32 + src;
          const int n_src = OWN ? __shfl_sync(0xffffffffu, own_cnt, src) : cnt_s[r];
          int kept = 0;
          const uint64_t kmax = warp_select_keep_any(pool_of(r), n_src < P ? n_src : P, keep, P, hist, kept);
          if (lane == src) {
            const uint32_t ord = (uint32_t)(kmax >> 32);
            const float nt = thr_from<Tr::kFolded>(ord2f(ord), qn);
            if constexpr (OWN) {
              own_cnt = kept;
              thr = fminf(thr, nt);
            } else {
              cnt_s[r] = kept;
              thr_s[r] = fminf(thr_s[r], nt);
            }
            // only a full set of k' keys bounds the global k'-th distance
            if (kept >= p.kprime) atomicMin(&p.q_bound[q], ord);
          }
        }
        STAT_END(tr, st_refresh);
      };

      // takes c slots of this lane's pool; returns the first
      auto reserve = [&](int c) -> int {
        if constexpr (OWN) {
          own_cnt += c;
          return own_cnt - c;
        } else {
          return c ? atomicAdd(&cnt_s[row], c) : 0;
        }
      };

      float* colv = reinterpret_cast<float*>(hist);  // FP8 without tails: [128] norms, then [128] scales
      // Coarse distances of `count` (a multiple of 4) accumulator columns from c
      // on of this warp's 128: the accumulator itself (BF16 and exact forms),
      // d / ku (FP8 with norm tails), else from the staged norms and scales.
      auto dist_of = [&](const uint32_t* v, int c, float* x, int count) {
#pragma unroll
        for (int j = 0; j < count; ++j) x[j] = __uint_as_float(v[j]);
        if (Tr::kRowScales) {
          const float4* xn4 = reinterpret_cast<const float4*>(colv + c);
          const float4* sx4 = reinterpret_cast<const float4*>(colv + kHalfN + c);
#pragma unroll
          for (int j = 0; j < count; j += 4) {  // fma(acc * s_x, 2 s_q, ||x||^2)
            const float4 xn = xn4[j / 4], sx = sx4[j / 4];
            x[j] = fmaf(x[j] * sx.x, s2, xn.x);
            x[j + 1] = fmaf(x[j + 1] * sx.y, s2, xn.y);
            x[j + 2] = fmaf(x[j + 2] * sx.z, s2, xn.z);
            x[j + 3] = fmaf(x[j + 3] * sx.w, s2, xn.w);
          }
        }
      };

      const int T_i = p.num_tiles;
      int tphys = t0 - rot;  // database tile of position t, kept in [0, T)
      if (tphys < 0) tphys += T_i;
      int until_sync = S;    // tiles until the pair meets
      // The shared bound is an L2 round trip and moves rarely: it is asked for
      // at one tile and used four tiles later (FILL: at the next)
      uint32_t nb_ob = kOrdInf;
      if (valid) nb_ob = ld_relaxed_u32(&p.q_bound[q]);
      for (int t = t0; t < t1; ++t, ++tc) {
        const uint32_t slot = tc & 1u, use = tc >> 1;
        if constexpr (!OWN) thr = fminf(thr, thr_s[row]);
        if (FILL || ((t - t0) & 3) == 0) {
          if (nb_ob != kOrdInf) thr = fminf(thr, thr_from<Tr::kFolded>(ord2f(nb_ob), qn));
          if (valid) nb_ob = ld_relaxed_u32(&p.q_bound[q]);
        }
        const float thr_up = next_above(thr);  // d <= thr  <=>  d < thr_up
        const int tile0 = tphys * kTileRows;   // first database row of the tile
        if (++tphys == T_i) tphys = 0;
        // FP8 without norm tails: the database norms and scales of this warp's
        // 128 columns, loaded before the accumulator wait (their latency
        // overlaps it) and staged in the warp's histogram area, which is free
        // outside a refresh
        float pxn[4], psx[4];
        if (Tr::kRowScales) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            // < nb_pad: rows are padded to whole tiles (a strided sample has no padding)
            const int c0 = tile0 + (DUAL ? 0 : g * kHalfN) + 32 * i + lane;
            size_t c = (size_t)c0;
            if (MINIMA)
              c = c * (size_t)p.db_step + (p.db_phased ? sample_phase(tile0 / kTileRows, p.db_step) : 0);
            pxn[i] = __ldg(p.db_norms + c);
            psx[i] = __ldg(p.db_scale + c);
          }
        }
        STAT_BEGIN(tw);
        // the same for the whole warp: what follows is warp-wide
        const bool got = __all_sync(0xffffffffu, wait_or_abort(&acc_full[slot], use & 1u, abort_flag));
        if (!got) raise_abort(abort_flag, B.status, kErrWaitTimeout);
        STAT_END(tw, st_wait);
        // an aborting warp skips the tile but still meets its partner below
        if (got) {
        STAT_BEGIN(tfl);
        tc_fence_after();
        if (Tr::kRowScales) {
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            colv[lane + 32 * i] = pxn[i];
            colv[kHalfN + lane + 32 * i] = psx[i];
          }
          __syncwarp();
        }
        const uint32_t t_src = tmem_base + lane_base + slot * kBN + g * kHalfN;
        const int tcol = tile0 + (DUAL ? 0 : g * kHalfN);  // database row of the warp's first column
        // Smallest distance of every 8 of the warp's 128 columns: half an
        // instruction a column (the masks of every column took 1.5) decides
        // whether anything of the tile survives, and which eights hold it.  The
        // warp's cost is latency -- about six cycles an instruction at two
        // warps per sub-partition -- so fewer instructions are the gain (full
        // pass: FP8 sphere 26.8 -> 16.9 ms, BF16 integer mixture 3.22 -> 2.84
        // and FP32-exact 5.58 -> 4.70 with dual blocks).
        float gm[16];
        {
          uint32_t v[64];
          float x[32];
          auto mins = [&](const uint32_t* v, int i) {
            dist_of(v, 32 * i, x, 32);
            if (MINIMA && tcol + 32 * i + 32 > p.nb) {  // columns past nb do not count
#pragma unroll
              for (int j = 0; j < 32; ++j) x[j] = tcol + 32 * i + j < p.nb ? x[j] : __builtin_huge_valf();
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) gm[4 * i + e] = min8(x + 8 * e);
          };
          tmem_ld_32x32b_x64(t_src, v);
          tmem_ld_wait();
          mins(v, 0);
          mins(v + 32, 1);
          tmem_ld_32x32b_x64(t_src + 64, v);
          tmem_ld_wait();
          mins(v, 2);
          mins(v + 32, 3);
        }
        const float dmin = fminf(min8(gm), min8(gm + 8));
        if (MINIMA) {
          if (valid) {
            const int br = p.minima_rows, per = kHalfN / br;  // 1 or 16 blocks of this warp's columns
            float* o = p.minima + (size_t)q * (2 * (size_t)T_i * per) + (size_t)(2 * (tile0 / kTileRows) + g) * per;
            auto key = [&](float x) { return Tr::kFolded ? x : (fold ? km * x : x) + qn; };
            if (br == kHalfN) {
              *o = key(dmin);
            } else {
#pragma unroll
              for (int e = 0; e < 16; e += 4)
                *reinterpret_cast<float4*>(o + e) =
                    make_float4(key(gm[e]), key(gm[e + 1]), key(gm[e + 2]), key(gm[e + 3]));
            }
          }
        } else if (__any_sync(0xffffffffu, passes<Tr::kFP8>(dmin, km, thr_up))) {
          STAT_INC(st_slow, 1);
          // the eights in which some lane has a survivor (uniform), one at a
          // time, fetched again from TMEM: one copy of the survivor code, which
          // holds no tile registers (unrolled over register-held columns it
          // missed the instruction caches)
          uint32_t hit = __reduce_or_sync(
              0xffffffffu, survive_mask<8>(gm, km, thr_up) | survive_mask<8>(gm + 8, km, thr_up) << 8);
          if (FILL && __popc(hit) >= kDenseEights) {
#pragma unroll 1
            for (int c32 = 0; c32 < kHalfN; c32 += 32) {
              uint32_t w[32];
              float x[32];
              tmem_ld_32x32b_x32(t_src + c32, w);
              tmem_ld_wait();
              dist_of(w, c32, x, 32);
              const int c0 = tcol + c32;
              uint32_t m = survive_mask<32>(x, km, thr_up);
              if (c0 + 32 > p.nb) m &= c0 >= p.nb ? 0u : (1u << (p.nb - c0)) - 1u;
              const int c = __popc(m);
              int n = reserve(c);
              STAT_INC(st_surv, c);
              if (m == ~0u) {  // every column (no bound yet)
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (n + j < P) pool[n + j] = make_key(key_d(x[j]), (uint32_t)(c0 + j));
                m = 0u;
              }
#pragma unroll 1
              while (__any_sync(0xffffffffu, m != 0u)) {
                STAT_INC(st_iters, 1);
                const int j = __ffs(m) - 1;  // -1: none left
                const float xs = select32(x, j);
                m &= m - 1u;
                if (j >= 0 && n < P) pool[n] = make_key(key_d(xs), (uint32_t)(c0 + j));
                ++n;
              }
            }
            hit = 0u;
          }
#pragma unroll 1
          while (hit) {
            const int e = __ffs(hit) - 1;
            hit &= hit - 1u;
            uint32_t w[8];
            float x[8];
            tmem_ld_32x32b_x8(t_src + 8 * e, w);
            tmem_ld_wait();
            dist_of(w, 8 * e, x, 8);
            const int c8 = tcol + 8 * e;
            uint32_t m = survive_mask<8>(x, km, thr_up);
            // database rows beyond nb (padding of the last tile) never survive
            if (c8 + 8 > p.nb) m &= c8 >= p.nb ? 0u : (1u << (p.nb - c8)) - 1u;
            const int c = __popc(m);
            int n = reserve(c);
            STAT_INC(st_surv, c);
            if (__any_sync(0xffffffffu, c > 2)) {
              // dense (a pool without a tight bound yet): every column in order
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const bool take = (m >> j) & 1u;
                if (take && n < P) pool[n] = make_key(key_d(x[j]), (uint32_t)(c8 + j));
                n += take ? 1 : 0;
              }
              continue;
            }
            // mostly one survivor, in one lane
#pragma unroll 1
            do {
              STAT_INC(st_iters, 1);
              const int j = __ffs(m) - 1;  // -1: none left
              const float xs = select8(x, j);
              m &= m - 1u;
              if (j >= 0 && n < P) pool[n] = make_key(key_d(xs), (uint32_t)(c8 + j));
              ++n;
            } while (__any_sync(0xffffffffu, m != 0u));
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (PAIR)
            mbar_arrive_remote(&acc_empty[slot], 0);  // the issuer's barrier counts both CTAs
          else
            mbar_arrive(&acc_empty[slot]);
        }
        STAT_END(tfl, st_filter);
        }  // got
        if constexpr (OWN) {
          if (!got) {
            ok = false;
            break;
          }
          // pools that may not have room for the next tile, or, at the unit's
          // end, every pool above the end's limit
          const int lim = t + 1 < t1 ? P - kHalfN : end_lim;
          const uint32_t need = __ballot_sync(0xffffffffu, valid && own_cnt > lim);
          if (need) {
            if (own_cnt > P) atomicOr(B.status, kErrPoolOverflow);
            __syncwarp();  // the other lanes read this lane's keys
            refresh(need, p.kprime);
          }
          continue;
        }
        // every S tiles (and at the unit's end) meet the partner warp; leave
        // together if either aborted
        if (--until_sync != 0 && t + 1 < t1) continue;
        until_sync = S;
        STAT_BEGIN(tb1);
        const bool leave = bar_red_or(pair_bar, kGroupThreads, !got || *abort_flag != 0);
        STAT_END(tb1, st_bar);
        if (leave) {
          ok = false;
          break;
        }
        // as above, for the next S tiles (both halves)
        const int lim = t + 1 < t1 ? P - S * kTileRows : end_lim;
        const bool mine = (lane & 1) == g;
        const int cn = mine ? cnt_s[row] : 0;
        if (cn > P) atomicOr(B.status, kErrPoolOverflow);
        refresh(__ballot_sync(0xffffffffu, mine && valid && cn > lim), p.kprime);
        STAT_BEGIN(tb2);
        bar_sync_named(pair_bar, kGroupThreads);
        STAT_END(tb2, st_bar);
      }
      if (!ok) break;
      // a refresh may keep a few more than k' keys (unsorted): record them all;
      // the merge pass selects exactly
      if (!MINIMA && valid && (OWN || g == 0)) {
        const int cn = OWN ? own_cnt : cnt_s[row];
        p.pool_counts[list_of(row)] = cn < P ? cn : P;
        if (gap) p.pool_counts[list_of(row) - kLists] = 0;
      }
      if constexpr (!OWN) bar_sync_named(pair_bar, kGroupThreads);  // the counts are read before the next unit resets them
    }
    // After an abort the lists of the current unit and of those not reached are
    // written as empty: the merge still runs, and the workspace's memory may have
    // held anything before.
    if constexpr (!MINIMA) {
      if (!ok) {
        do {
          const FusedItem& p = A.items[MAXI == 1 ? 0 : ii];
          const int U = p.units_per_block;
          const long long q = (long long)(DUAL ? qb + g : qb) * kBM + row;
          if (u_ord >= 0 && u_ord < U && q < p.nq && (OWN || g == 0)) {
            const size_t l = ((size_t)q * U + (size_t)u_ord) * kLists + (kLists > 1 ? g : 0);
            p.pool_counts[l] = 0;
            if (gap) p.pool_counts[l - kLists] = 0;
          }
        } while (walk.next(A, ii, qb, t0, t1, u_ord, gap, rot));
      }
    }
    if (lane == 0) {
      STAT_FLUSH(kStatEpiWaitAccFull, st_wait);
      STAT_FLUSH(kStatEpiFilter, st_filter);
      STAT_FLUSH(kStatEpiRefresh, st_refresh);
      STAT_FLUSH(kStatRefreshes, st_nref);
      STAT_FLUSH(kStatSlowChunks, st_slow);
      STAT_FLUSH(kStatLoopIters, st_iters);
      STAT_FLUSH(kStatPairBarrier, st_bar);
    }
    STAT_FLUSH(kStatSurvivors, st_surv);
  }

  tc_fence_before();
  // a pair releases its TMEM together, and neither CTA leaves while the
  // other may still signal its barriers or read its shared memory
  if constexpr (PAIR)
    cluster_sync();
  else
    __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if constexpr (PAIR)
      tmem_dealloc_pair(tmem_base, 512);
    else
      tmem_dealloc(tmem_base, 512);
  }
#ifdef CURPLSH_FUSED_STATS
  if (threadIdx.x == 0 && B.stats) atomicAdd(&B.stats[kStatCtaCycles], (unsigned long long)(clock64() - t_kernel));
#endif
}

// ------------------------------------------------------------------ host side
namespace {

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// 2-D K-major operand map: rows x ld elements, box = (128 bytes of K) x box_rows
// with the 128-byte swizzle, or (narrow) 32 bytes of K with the 32-byte
// swizzle; zero fill out of bounds.  Map row j is stored row j * row_step; with
// `phased` it is the row_step stored rows from there on, one after another: row f
// of them starts at column f * ld_elems, and a box that reaches past it holds the
// next row's first columns, which meet zeros of the query rows.
bool make_map(CUtensorMap* m, const void* base, bool fp8, long long rows, long long ld_elems, int box_rows,
              bool narrow = false, int row_step = 1, bool phased = false) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return false;
  const int esz = fp8 ? 1 : 2;
  const cuuint64_t step = (cuuint64_t)(row_step > 1 ? row_step : 1);
  cuuint64_t dims[2] = {(cuuint64_t)ld_elems * (phased ? step : 1), (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(ld_elems * esz) * step};
  cuuint32_t box[2] = {(cuuint32_t)((narrow ? kTailRowBytes : kChunkBytes) / esz), (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, fp8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
                  const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  narrow ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// Raises the kernel's dynamic shared memory limit once per device.
template <int FORM, int MAXI, bool MINIMA = false, bool PAIR = false, bool DUAL = false, bool FILL = false>
cudaError_t ensure_attributes() {
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_done[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(fused_knn_kernel<FORM, MAXI, MINIMA, PAIR, DUAL, FILL>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         227 * 1024);
    if (e != cudaSuccess) return e;
    attr_done[dev & 63] = true;
  }
  return cudaSuccess;
}

template <int FORM, int MAXI, bool MINIMA = false, bool PAIR = false, bool DUAL = false, bool FILL = false>
cudaError_t launch_form(const FusedItemSpec* specs, const FusedItemPlan* plans, int n, const FusedBatchPlan& bp,
                        uint32_t* status, unsigned long long* stats, cudaStream_t st,
                        const int* run_if) {
  cudaError_t e = ensure_attributes<FORM, MAXI, MINIMA, PAIR, DUAL, FILL>();
  if (e != cudaSuccess) return e;
  const uint32_t smem = make_layout(FORM, specs[0].d, PAIR ? 1 : 0, kEpiWarps, DUAL ? 1 : 0).total;
  if (smem > 227u * 1024u) return cudaErrorInvalidConfiguration;  // a layout bug, not a caller error
  FusedArgs<MAXI> a;
  memset(&a, 0, sizeof(a));
  a.B.num_items = n;
  a.B.form = FORM;
  a.B.d = specs[0].d;
  a.B.pair = bp.pair;
  a.B.total_work = bp.total_work;
  a.B.work_per_cta = bp.work_per_cta;
  a.B.dual = bp.dual;
  const int xrows = kBN >> (bp.pair | bp.dual);  // database rows one CTA loads per tile
  a.B.status = status;
  a.B.stats = stats;
  a.B.run_if = run_if;
  constexpr bool fp8 = FormTraits<FORM>::kFP8;
  for (int i = 0; i < n; ++i) {
    const FusedItemSpec& f = specs[i];
    const FusedItemPlan& pl = plans[i];
    FusedItem& it = a.items[i];
    it.nq = f.nq;
    it.nb = f.nb;
    it.kprime = f.kprime;
    it.pool_cap = f.pool_cap;
    it.num_qblocks = pl.num_qblocks;
    it.num_tiles = pl.num_tiles;
    it.units_per_block = pl.units_per_block;
    it.split_tiles = pl.split_tiles;
    it.work_begin = pl.work_begin;
    it.work_end = pl.work_end;
    it.db_norms = f.xn;
    it.db_scale = f.xs;
    it.q_norms = f.qn;
    it.q_scale = f.qs;
    it.pools = f.pools;
    it.pool_counts = f.pool_counts;
    it.q_bound = f.q_bound;
    it.db_step = f.db_step > 1 ? f.db_step : 1;
    it.db_phased = f.db_phased ? (int)(fp8 ? f.ld8 : f.ld16) : 0;
    it.db_scale_uniform = f.xs_uniform;
    it.fp8_tail = FORM == kFormFP8 ? (int)fp8_tail_offset(f.d, f.ld8) : 0;
    it.minima = f.minima;
    it.minima_rows = f.minima_rows;
    CUtensorMap* m = &a.maps[i * kMapsPerItem];
    const void* qh = fp8 ? (const void*)f.q8 : (const void*)f.qh;
    const void* xh = fp8 ? (const void*)f.x8 : (const void*)f.xh;
    const long long ldq = fp8 ? f.ld8 : f.ld16;
    if (!MINIMA && it.db_step > 1) return cudaErrorInvalidValue;  // samples are block-minimum passes
    const int step = it.db_step;
    const bool phased = it.db_phased != 0;
    if (!make_map(&m[kMapQHi], qh, fp8, f.nq_pad, ldq, kBM) ||
        !make_map(&m[kMapXHi], xh, fp8, f.nb_pad, ldq, xrows, false, step, phased))
      return cudaErrorInvalidValue;
    if (FORM == kFormExact) {
      if (!make_map(&m[kMapQLo], f.ql, false, f.nq_pad, f.ld16, kBM) ||
          !make_map(&m[kMapXLo], f.xl, false, f.nb_pad, f.ld16, xrows, false, step, phased))
        return cudaErrorInvalidValue;
    } else {
      m[kMapQLo] = m[kMapQHi];
      m[kMapXLo] = m[kMapXHi];
    }
    if (!make_map(&m[kMapQTail], qh, fp8, f.nq_pad, ldq, kBM, true) ||
        !make_map(&m[kMapXTail], xh, fp8, f.nb_pad, ldq, xrows, true, step, phased))
      return cudaErrorInvalidValue;
  }
  if (PAIR && bp.grid % 2) return cudaErrorInvalidValue;
  return launch_dependent(fused_knn_kernel<FORM, MAXI, MINIMA, PAIR, DUAL, FILL>, (unsigned)bp.grid, kNumThreads, smem, st,
                          bp.pdl != 0, PAIR ? 2 : 1, a);
}

// The candidate-pool instance of a plan.  Dual blocks without bounds are planned
// for FP8 alone (plan_fused_batch).
template <int FORM, int MAXI>
cudaError_t launch_pools(const FusedItemSpec* specs, const FusedItemPlan* plans, int n, const FusedBatchPlan& bp,
                         uint32_t* status, unsigned long long* stats, cudaStream_t st,
                         const int* run_if) {
  if (bp.dual) {
    if constexpr (FormTraits<FORM>::kFP8)
      if (bp.fill)
        return launch_form<FORM, MAXI, false, false, true, true>(specs, plans, n, bp, status, stats, st, run_if);
    return launch_form<FORM, MAXI, false, false, true>(specs, plans, n, bp, status, stats, st, run_if);
  }
  if (bp.pair)
    return bp.fill ? launch_form<FORM, MAXI, false, true, false, true>(specs, plans, n, bp, status, stats, st, run_if)
                   : launch_form<FORM, MAXI, false, true>(specs, plans, n, bp, status, stats, st, run_if);
  return bp.fill ? launch_form<FORM, MAXI, false, false, false, true>(specs, plans, n, bp, status, stats, st, run_if)
                 : launch_form<FORM, MAXI>(specs, plans, n, bp, status, stats, st, run_if);
}

template <int FORM>
cudaError_t launch_form_any(const FusedItemSpec* specs, const FusedItemPlan* plans, int n, const FusedBatchPlan& bp,
                            uint32_t* status, unsigned long long* stats, cudaStream_t st,
                            const int* run_if) {
  if (n == 1 && specs[0].minima)
    return bp.pair ? launch_form<FORM, 1, true, true>(specs, plans, n, bp, status, stats, st, run_if)
                   : launch_form<FORM, 1, true>(specs, plans, n, bp, status, stats, st, run_if);
  for (int i = 0; i < n; ++i)
    if (specs[i].minima) return cudaErrorInvalidValue;  // block-minimum mode is single-item
  if (n == 1) return launch_pools<FORM, 1>(specs, plans, n, bp, status, stats, st, run_if);
  return launch_pools<FORM, kFusedMaxItems>(specs, plans, n, bp, status, stats, st, run_if);
}

}  // namespace

#ifndef CURPLSH_DUAL_DEFAULT
#define CURPLSH_DUAL_DEFAULT 1
#endif
namespace {
std::atomic<int> g_cta_pairs{kPairsAuto};
std::atomic<int> g_dual{CURPLSH_DUAL_DEFAULT};
// Automatic CTA pairs: BF16 and FP32-exact from these dimensions on, where two
// query blocks no longer fit one CTA and the MMAs of a tile are heavy enough that
// halving each SM's database bytes per query pays (500,000 N(0,1) rows, 4,096
// queries, k = 10, pass with single blocks -> pairs: BF16 d = 320 1,381 -> 986 us,
// 384 2,160 -> 1,144, 512 2,641 -> 1,377; FP32-exact 192 2,047 -> 1,272, 256 2,478
// -> 1,795, 384 3,498 -> 2,650; identical results).  Below the lines dual blocks
// are the rule; between the last of them and the line (FP32-exact d = 123 to 191,
// BF16 315 to 319) pairs measure ahead too (FP32-exact 144: 2,218 -> 1,067).
constexpr int kPairMinDimBF16 = 320;
constexpr int kPairMinDimExact = 192;
}  // namespace

void set_cta_pairs(int mode) {
  g_cta_pairs.store(mode == kPairsAuto ? kPairsAuto : (mode ? 1 : 0), std::memory_order_relaxed);
}
int get_cta_pairs() { return g_cta_pairs.load(std::memory_order_relaxed); }
void set_dual_blocks(int on) { g_dual.store(on ? 1 : 0, std::memory_order_relaxed); }
int get_dual_blocks() { return g_dual.load(std::memory_order_relaxed); }

void plan_fused_batch(const FusedItemSpec* specs, int n, int max_ctas, FusedItemPlan* plans, FusedBatchPlan* out,
                      int form) {
  // Query groups of two blocks (dual blocks in one CTA for BF16/FP8, else CTA
  // pairs when on) when there are enough query blocks and few groups would be
  // half empty (an item with an odd block count leaves its last group one
  // block short)
  long long blocks = 0, odd = 0;
  for (int i = 0; i < n; ++i) {
    const long long g = specs[i].nb > 0 ? (specs[i].nq + kBM - 1) / kBM : 0;
    blocks += g;
    odd += g & 1;
  }
  const bool grouped = blocks >= 4 && odd * 8 <= blocks;
  // dual blocks need both query blocks resident in shared memory, and a ring
  // whose stages cover the load latency: three, or two of the FP32-exact form's,
  // each of which feeds three products (BF16 with two stages, d = 320: 4.26 ms
  // against 3.53 as CTA pairs)
  bool dual_fits = false;
  if (n > 0 && specs[0].d > 0 && form >= 0) {
    const SmemLayout DL = make_layout(form, specs[0].d, 0, kEpiWarps, 1);
    dual_fits = !DL.a_stream && DL.stages >= (form == kFormExact ? 2 : 3);
  }
  // Pools that start without a bound fill to k' keys in every unit, and a dual
  // unit has half the rows at the same CTA range, so there are twice as many and
  // the bounds tighten later: such passes keep single blocks (1,000 queries, single
  // -> dual: FP32-exact, k' = 32, 100,000 rows 472 -> 686 us; BF16, 10^6 rows 1,042
  // -> 1,311; FP8, k' = 480, 100,000 rows 697 -> 877).  FP8's light MMAs pay for dual
  // blocks where the half unit alone ends without a selection (k' = 480, 3,000 rows,
  // 4,000 queries: 166 -> 82; k' = 1,216, 100,000 rows, 1,000: 2,728 -> 1,719).
  bool fill = false, lean = false;
  int kp_min = 1 << 30;
  for (int i = 0; i < n; ++i) {
    fill = fill || specs[i].fill_kprime > 0;
    if (specs[i].fill_kprime > 0) kp_min = std::min(kp_min, specs[i].fill_kprime);
    lean = lean || specs[i].lean;
  }
  bool dual_pays = !fill;
  if (fill && form == kFormFP8) {
    long long work = 0;
    for (int i = 0; i < n; ++i)
      work += (long long)((specs[i].nq + kBM - 1) / kBM) * ((specs[i].nb + kBN - 1) / kBN);
    const long long w = (work + max_ctas - 1) / max_ctas;
    for (int i = 0; i < n; ++i) {
      const long long rows = kBN * (specs[i].split_tiles > 0 ? std::min<long long>(w, specs[i].split_tiles) : w);
      const int lim = end_limit(specs[i].fill_kprime);
      dual_pays = dual_pays || (specs[i].fill_kprime > 0 && rows > lim && rows <= 2LL * lim);
    }
  }
  // Two query blocks per CTA: a database tile crosses L2 -> SM once per 256
  // queries, and every query's pool belongs to one lane (full pass, single ->
  // dual blocks: BF16 integer mixture 3.50 -> 2.84 ms, FP32-exact 5.64 -> 4.70)
  const int dual = (grouped && dual_fits && dual_pays && !lean && get_dual_blocks()) ? 1 : 0;
  const int pm = get_cta_pairs();
  const int d0 = n > 0 ? specs[0].d : 0;
  // FP8 pairs where a CTA's own ring is down to two stages, which no longer cover
  // the load latency: the norm tail's chunk took the third at d = 768 (pass, single
  // -> pairs: 1,842 -> 1,425 us, 1,620 before there was a tail; 1,024 2,376 ->
  // 1,714; with three stages, d = 704, 1,385 -> 1,477).  Passes of a few tiles per
  // CTA do not pay for the pair's barriers (963 rows, 708 queries, d = 960: 35 -> 41).
  long long single_work = 0;
  for (int i = 0; i < n; ++i)
    single_work += (long long)((specs[i].nq + kBM - 1) / kBM) * ((specs[i].nb + kBN - 1) / kBN);
  const bool fp8_pair = form == kFormFP8 && d0 > 0 && single_work >= 4LL * max_ctas && make_layout(form, d0).stages < 3;
  const bool want_pair = pm == 1 || (pm == kPairsAuto && ((form == kFormBF16 && d0 >= kPairMinDimBF16) ||
                                                          (form == kFormExact && d0 >= kPairMinDimExact) ||
                                                          (form == kFormFP8 && fp8_pair)));
  const int pair = (!dual && !lean && grouped && want_pair && max_ctas >= 2) ? 1 : 0;
  const int rows = kBM << (pair | dual);
  const int tile_rows = dual ? kBN / 2 : kBN;
  long long total = 0;
  for (int i = 0; i < n; ++i) {
    FusedItemPlan& pl = plans[i];
    pl.num_qblocks = specs[i].nb > 0 ? (specs[i].nq + rows - 1) / rows : 0;
    pl.num_tiles = (specs[i].nb + tile_rows - 1) / tile_rows;
    pl.split_tiles = specs[i].split_tiles > 0 && specs[i].split_tiles < pl.num_tiles ? specs[i].split_tiles
                                                                                      : std::max(pl.num_tiles, 1);
    pl.work_begin = total;
    total += (long long)pl.num_qblocks * pl.num_tiles;
    pl.work_end = total;
    pl.pair = pair;
    pl.dual = dual;
  }
  const long long units = max_ctas >> pair;  // CTAs, or pairs of CTAs
  long long grid = units < total ? units : total;
  if (grid < 1) grid = 1;
  out->pair = pair;
  out->dual = dual;
  out->total_work = total;
  out->work_per_cta = total > 0 ? (total + grid - 1) / grid : 1;
  out->grid = total > 0 ? (int)((total + out->work_per_cta - 1) / out->work_per_cta) << pair : 0;
  const long long W = out->work_per_cta;
  // Pairs whose units are single tiles never fill pools of 128 keys and more, one
  // per warp, to k': no bound, no selection (FP32-exact, d = 512, k' = 128, 2,000
  // rows, 1,000 queries: pass 50 us, 146 with shared pools).
  out->fill = fill && !(pair && W == 1 && kp_min >= kHalfN) ? 1 : 0;
  for (int i = 0; i < n; ++i) {
    FusedItemPlan& pl = plans[i];
    pl.fill = out->fill;
    int U = 1;
    for (int qb = 0; qb < pl.num_qblocks; ++qb) {
      const long long base = pl.work_begin + (long long)qb * pl.num_tiles;
      const long long u = (base + pl.num_tiles - 1) / W - base / W + (pl.num_tiles - 1) / pl.split_tiles + 1;
      if (u > U) U = (int)u;
    }
    pl.units_per_block = U;
  }
}

void plan_fused(int nq, int nb, int num_sms, FusedPlan* out, int split_q4, int form, int d, int fill_kprime, bool lean) {
  FusedItemSpec s{};
  s.nq = nq;
  s.nb = nb;
  s.d = d;
  s.fill_kprime = fill_kprime;
  s.lean = lean;
  FusedItemPlan ip;
  FusedBatchPlan bp;
  plan_fused_batch(&s, 1, num_sms, &ip, &bp, form);
  if (split_q4 < 4 && bp.grid > 0) {
    s.split_tiles = split_tiles_for(bp.work_per_cta, split_q4);
    plan_fused_batch(&s, 1, num_sms, &ip, &bp, form);
  }
  out->num_qblocks = ip.num_qblocks;
  out->num_tiles = ip.num_tiles;
  out->work_per_cta = bp.work_per_cta;
  out->grid = bp.grid;
  out->pair = bp.pair;
  out->dual = bp.dual;
  out->fill = bp.fill;
  out->units_per_block = ip.units_per_block;
  out->split_tiles = ip.split_tiles;
}

uint32_t fused_smem_bytes(int form, int d) { return make_layout(form, d).total; }

template <int FORM, int MAXI>
static cudaError_t prepare_pools() {
  cudaError_t e = ensure_attributes<FORM, MAXI>();
  if (e == cudaSuccess) e = ensure_attributes<FORM, MAXI, false, true>();
  if (e == cudaSuccess) e = ensure_attributes<FORM, MAXI, false, false, true>();
  if (e == cudaSuccess) e = ensure_attributes<FORM, MAXI, false, false, false, true>();
  if (e == cudaSuccess) e = ensure_attributes<FORM, MAXI, false, true, false, true>();
  if constexpr (FormTraits<FORM>::kFP8)
    if (e == cudaSuccess) e = ensure_attributes<FORM, MAXI, false, false, true, true>();
  return e;
}

template <int FORM>
static cudaError_t prepare_form() {
  cudaError_t e = prepare_pools<FORM, 1>();
  if (e == cudaSuccess) e = prepare_pools<FORM, kFusedMaxItems>();
  if (e == cudaSuccess) e = ensure_attributes<FORM, 1, true>();
  if (e == cudaSuccess) e = ensure_attributes<FORM, 1, true, true>();
  return e;
}

cudaError_t prepare_fused_kernels(int form) {
  switch (form) {
    case kFormExact:
      return prepare_form<kFormExact>();
    case kFormBF16:
      return prepare_form<kFormBF16>();
    case kFormFP8: {
      const cudaError_t e = prepare_form<kFormFP8>();
      return e != cudaSuccess ? e : prepare_form<kFormFP8Rows>();
    }
    default:
      return cudaErrorInvalidValue;
  }
}

cudaError_t launch_fused_batch(int form, const FusedItemSpec* specs, const FusedItemPlan* plans, int n,
                               const FusedBatchPlan& bp, uint32_t* status, unsigned long long* stats,
                               cudaStream_t st, const int* run_if) {
  if (n < 1 || n > kFusedMaxItems) return cudaErrorInvalidValue;
  for (int i = 1; i < n; ++i)
    if (specs[i].d != specs[0].d) return cudaErrorInvalidValue;
  if (bp.grid == 0) return cudaSuccess;
  switch (form) {
    case kFormExact:
      return launch_form_any<kFormExact>(specs, plans, n, bp, status, stats, st, run_if);
    case kFormBF16:
      return launch_form_any<kFormBF16>(specs, plans, n, bp, status, stats, st, run_if);
    case kFormFP8: {
      // one scale per database for all items of the launch, or per-row scales for all
      const bool rows = !(specs[0].xs_uniform > 0.f);
      for (int i = 1; i < n; ++i)
        if (rows != !(specs[i].xs_uniform > 0.f)) return cudaErrorInvalidValue;
      return rows ? launch_form_any<kFormFP8Rows>(specs, plans, n, bp, status, stats, st, run_if)
                  : launch_form_any<kFormFP8>(specs, plans, n, bp, status, stats, st, run_if);
    }
    default:
      return cudaErrorInvalidValue;
  }
}

cudaError_t launch_fused(const FusedLaunch& f, cudaStream_t st) {
  FusedItemSpec s{};
  s.nq = f.nq;
  s.nb = f.nb;
  s.d = f.d;
  s.kprime = f.kprime;
  s.pool_cap = f.pool_cap;
  s.nq_pad = f.nq_pad;
  s.nb_pad = f.nb_pad;
  s.ld16 = f.ld16;
  s.ld8 = f.ld8;
  s.qh = f.qh;
  s.ql = f.ql;
  s.q8 = f.q8;
  s.qn = f.qn;
  s.qs = f.qs;
  s.xh = f.xh;
  s.xl = f.xl;
  s.x8 = f.x8;
  s.xn = f.xn;
  s.xs = f.xs;
  s.xs_uniform = f.xs_uniform;
  s.pools = f.pools;
  s.pool_counts = f.pool_counts;
  s.q_bound = f.q_bound;
  s.db_step = f.db_step;
  s.db_phased = f.db_phased;
  s.minima = f.minima;
  s.minima_rows = f.minima_rows;
  FusedItemPlan ip;
  ip.num_qblocks = f.plan.num_qblocks;
  ip.num_tiles = f.plan.num_tiles;
  ip.units_per_block = f.plan.units_per_block;
  ip.split_tiles = f.plan.split_tiles > 0 ? f.plan.split_tiles : std::max(f.plan.num_tiles, 1);
  ip.work_begin = 0;
  ip.work_end = (long long)f.plan.num_qblocks * f.plan.num_tiles;
  ip.pair = f.plan.pair;
  ip.dual = f.plan.dual;
  ip.fill = f.plan.fill;
  FusedBatchPlan bp;
  bp.total_work = ip.work_end;
  bp.work_per_cta = f.plan.work_per_cta;
  bp.grid = f.plan.grid;
  bp.pair = f.plan.pair;
  bp.dual = f.plan.dual;
  bp.fill = f.plan.fill;
  bp.pdl = f.pdl ? 1 : 0;
  return launch_fused_batch(f.form, &s, &ip, 1, bp, f.status, f.stats, st, f.run_if);
}

}  // namespace curplsh_b200
