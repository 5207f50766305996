// common.cuh -- definitions shared by the kernels and the host orchestration.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp8.h>

namespace curplsh_b200 {

// ------------------------------------------------------------ dependent launches
// A search is a chain of five short kernels.  Launched as programmatic
// dependents, a kernel's launch and prologue overlap its predecessor's end: each
// kernel waits (before it touches global memory) until its predecessor has
// completed, and the short ones let their successor be scheduled early.  Both are
// no-ops in an ordinary launch (one query against 10^4 rows 72 -> 59 us a search,
// 100 queries 75 -> 63, 1,284 against 60,000 rows 155 -> 147).
#ifdef __CUDACC__
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// kernel<<<grid, block, smem, st>>>(args...), as a programmatic dependent when
// `pdl`, in clusters of `cluster` CTAs when > 1.
template <class... P, class... A>
cudaError_t launch_dependent(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, bool pdl,
                             int cluster, const A&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(block, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  unsigned n = 0;
  if (pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)cluster;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
#endif

// ------------------------------------------------------------ precision forms
// Form of the coarse (tensor-core) distance pass.  Every form finishes with
// an exact FP32 rerank of its candidates, so returned distances are
// sum_i (q_i - x_i)^2 in FP32 regardless of the coarse precision.
enum Form : int {
  kFormExact = 0,  // 3 x BF16 split products (hi*hi + hi*lo + lo*hi), FP32 accumulate
  kFormBF16 = 1,   // BF16 x BF16, FP32 accumulate, k' = rerank_factor * k candidates
  kFormFP8 = 2,    // FP8-E4M3 with per-vector FP32 scales, k' = rerank_factor * k
};

// ------------------------------------------------------------ device error word
// Bit flags written (atomicOr) to a device status word by kernels that give up.
enum DeviceError : uint32_t {
  kErrNone = 0,
  kErrWaitTimeout = 1u << 0,    // an mbarrier wait exceeded its poll limit
  kErrPoolOverflow = 1u << 1,   // a candidate pool would have overflowed (never expected)
  kErrBadSchedule = 1u << 2,    // unit bookkeeping out of range (never expected)
};

// ------------------------------------------------------------ ordered keys
// Candidates are 64-bit keys: (order-preserving bits of the FP32 distance) << 32
// | database row.  Unsigned comparison of keys is (distance, index)
// lexicographic order, the engine's tie rule (lower index first).
__host__ __device__ __forceinline__ uint32_t f_bits(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t u;
  __builtin_memcpy(&u, &f, 4);
  return u;
#endif
}
__host__ __device__ __forceinline__ float bits_f(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  __builtin_memcpy(&f, &u, 4);
  return f;
#endif
}
__host__ __device__ __forceinline__ uint32_t f2ord(float f) {
  uint32_t u = f_bits(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ __forceinline__ float ord2f(uint32_t o) {
  uint32_t u = (o & 0x80000000u) ? (o & 0x7FFFFFFFu) : ~o;
  return bits_f(u);
}
__host__ __device__ __forceinline__ uint64_t make_key(float d, uint32_t idx) {
  return ((uint64_t)f2ord(d) << 32) | idx;
}
constexpr uint64_t kKeyEmpty = ~0ull;
constexpr uint32_t kOrdInf = 0xFFFFFFFFu;  // "no bound yet" for per-query thresholds

// ------------------------------------------------------------ fused pass geometry
constexpr int kBM = 128;          // queries per block: MMA M, one TMEM lane per query
constexpr int kBN = 256;          // database rows per tile: MMA N (TMEM columns per accumulator)
constexpr int kHalfN = kBN / 2;   // columns of a tile handled by one epilogue warpgroup
constexpr int kChunkBytes = 128;  // K extent of one smem chunk row (one 128-byte swizzle atom)
constexpr int kNumThreads = 320;  // warp 0 TMA producer, warp 1 MMA issuer, warps 2..9 epilogue
// BF16 forms append kAugCols columns to every row so the tensor cores add the
// norms: database rows carry [n1 n2 n3 1 1 1] (||x||^2 = n1+n2+n3, three BF16
// terms), query rows (stored as -2q) carry [1 1 1 m1 m2 m3] (||q||^2 = m1+m2+m3),
// and the accumulator is ||q||^2 + ||x||^2 - 2 q.x directly.
constexpr int kAugCols = 6;
constexpr int kEpiWarps = 8;  // two per TMEM lane group
constexpr int kPoolRoom = kBN;  // free slots a candidate pool keeps for the next tile (both halves)
// Tiles between two selection points of a shared candidate pool: two when the
// capacity leaves room for two tiles of appends above k' + 128, else one.
__host__ __device__ inline int pool_sync_tiles(int cap, int kprime) { return cap >= kprime + 2 * kBN + 128 ? 2 : 1; }

// One work item of the fused pass: a query batch against one resident
// database.  A launch serves a list of items that share the form and the
// dimension; the (item, query block, tile) space of all of them is flattened
// and split evenly across the CTAs.  Items travel in the kernel parameters.
struct FusedItem {
  int nq;                  // real number of queries
  int nb;                  // real number of database rows
  int kprime;              // candidates kept per query (before the FP32 rerank)
  int pool_cap;            // capacity of one candidate pool (entries)
  int num_qblocks;         // G_i = ceil(nq / R), R = 128 query rows, 256 with dual blocks and CTA pairs
  int num_tiles;           // T_i = ceil(nb / 256), or / 128 with dual blocks
  int units_per_block;     // U_i: max units (pool lists) of one query block of this item
  int split_tiles;         // L_i: a unit never crosses a multiple of L_i tiles within its block
  long long work_begin;    // flattened offset of this item's first (block, tile)
  long long work_end;      // work_begin + G_i * T_i
  const float* db_norms;   // [nb_pad] squared norms, +inf for padding rows (FP8 form)
  const float* db_scale;   // [nb_pad] fp8 per-vector scales (FP8 form)
  const float* q_norms;    // [nq_pad]
  const float* q_scale;    // [nq_pad] (FP8 form)
  uint64_t* pools;         // [G_i*R][U_i][pool_lists][pool_cap]
  int* pool_counts;        // [G_i*R][U_i][pool_lists]
  uint32_t* q_bound;       // [nq_pad] shared per-query bound (ordered bits), init kOrdInf or an estimate
  // Database row j of this item is stored row j * db_step (>= 1; > 1 in
  // block-minimum mode only), plus sample_phase(j / 256, db_step) when db_phased,
  // which then is the columns of a stored row.
  int db_step, db_phased;
  float db_scale_uniform;  // > 0: every database row has this FP8 scale s (db_scale is not read)
  // FP8 form with one database scale: the byte offset of the 32-byte BF16 norm
  // tail of the FP8 rows (query rows, codes negated: [a1 a1 a2 a2 a1 a3], a = -1/s_q;
  // database rows [b1 b2 b1 b2 b3 b1], b = -||x||^2 / (2 s)).  One K=16 BF16 MMA over
  // the tails adds ||x||^2 / (2 s_q s) to the FP8 accumulator, which then is
  // (||x||^2 - 2 q.x) / (2 s_q s): no database norm is loaded per tile.
  int fp8_tail;
  // Non-null: block-minimum mode (no pools): minima[q * B + b] gets the smallest
  // key distance of query q over rows [b * minima_rows, +minima_rows) of the
  // B = 256 num_tiles / minima_rows blocks.
  float* minima;
  int minima_rows;         // 128 or 8
};

// Which of the db_step rows after its first each row of a phased sample's tile is:
// the fractions t * (sqrt(5) - 1) / 2 mod 1 spread the tiles evenly over them, so
// rows stored with a period that divides the step are sampled alike.
__host__ __device__ inline int sample_phase(int tile, int step) {
  return (int)(((unsigned long long)((uint32_t)tile * 2654435769u) * (uint32_t)step) >> 32);
}

// Tensor maps of one item, in this order.
enum FusedMap : int { kMapQHi = 0, kMapQLo, kMapXHi, kMapXLo, kMapQTail, kMapXTail, kMapsPerItem };

struct FusedBatch {
  int num_items;
  int form;
  int d;                   // dimension shared by every item of the launch
  int pair;                // 1: clusters of two CTAs, one 256-row MMA over two query blocks
  int dual;                // 1: each CTA holds two query blocks against 128-row database tiles
  int pad1;
  long long total_work;    // sum of G_i * T_i (G_i: query groups of 128 << pair rows)
  long long work_per_cta;  // W, per CTA (per pair when pair = 1)
  uint32_t* status;        // device error word
  unsigned long long* stats;  // per-role cycle counters, written only by builds with CURPLSH_FUSED_STATS
  const int* run_if;       // non-null: every CTA returns at once unless *run_if != 0
};

// Counter slots of FusedBatch::stats (instrumented builds).
enum FusedStat : int {
  kStatProducerWaitEmpty = 0,  // producer lane: cycles waiting for a free stage
  kStatMmaWaitFull,            // MMA lane: cycles waiting for TMA data
  kStatMmaWaitAccEmpty,        // MMA lane: cycles waiting for the epilogue to free an accumulator
  kStatEpiWaitAccFull,         // epilogue warps (lane 0): cycles waiting for an accumulator
  kStatEpiFilter,              // epilogue warps: cycles filtering tiles
  kStatEpiRefresh,             // epilogue warps: cycles in pool refreshes
  kStatRefreshes,              // number of pool refreshes
  kStatSurvivors,              // candidates appended to pools
  kStatCtaCycles,              // sum over CTAs of kernel cycles
  kStatRadixPasses,            // histogram passes run by pool refreshes
  kStatSlowChunks,             // warp-tiles (a warp's 128 columns) that entered the survivor path
  kStatLoopIters,              // survivor-append loop iterations executed by warps
  kStatPairBarrier,            // epilogue warps (lane 0): cycles in the pair barriers
  kStatCount
};

}  // namespace curplsh_b200
