// ptx.cuh -- thin inline-PTX wrappers for the sm_100a features the engine uses:
// mbarriers, TMA tensor loads, and the 5th-generation tensor core (tcgen05:
// TMEM allocation, MMA, commit, TMEM->register loads).  Every spin-wait here is
// bounded: it gives up after a fixed number of polls and reports failure so the
// caller can record an error status and wind down instead of hanging the GPU.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace curplsh_b200 {

// Every mbarrier wait gives up after kWaitTimeoutNs of wall time (read from
// %globaltimer) or kWaitPollLimit polls, whichever comes first, and reports
// failure; callers then record an error status and wind down.
constexpr uint64_t kWaitTimeoutNs = 2000000000ull;  // 2 s
constexpr uint32_t kWaitPollLimit = 1u << 28;

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// Named barrier over `count` threads (whole warps).  Every participating
// warp must reach it; it orders their shared and global memory accesses.
__device__ __forceinline__ void bar_sync_named(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
// Named barrier that also returns the OR of `v` over the participants.
__device__ __forceinline__ bool bar_red_or(int id, int count, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred pi, po;\n\tsetp.ne.u32 pi, %1, 0;\n\tbar.red.or.pred po, %2, %3, pi;\n\tselp.u32 %0, 1, 0, po;\n\t}"
      : "=r"(r)
      : "r"((uint32_t)v), "r"(id), "r"(count)
      : "memory");
  return r != 0;
}

// A packed FP32 pair (sm_100): one instruction, two IEEE results rounded as the
// scalar fma.rn would round them.
__device__ __forceinline__ void fma2_f32(float& d0, float& d1, float a0, float a1, float b0, float b1, float c0,
                                         float c1) {
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t"
      "mov.b64 rc, {%6, %7};\n\tfma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d0), "=f"(d1)
      : "f"(a0), "f"(a1), "f"(b0), "f"(b1), "f"(c0), "f"(c1));
}

__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait for the phase with the given parity.  Returns false on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  for (uint32_t i = 0; i < kWaitPollLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 1023u) == 1023u && globaltimer_ns() - t0 > kWaitTimeoutNs) return false;
  }
  return false;
}

// ---------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}

// 2-D tiled bulk tensor load global -> shared, completion on an mbarrier.
// c0 is the innermost (contiguous) coordinate in elements; callers keep
// c0 * element size a multiple of 16 bytes (it is always 0 or a multiple of
// the 128-byte box width here).
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const void* tmap, uint64_t* bar, int c0, int c1,
                                            uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "l"(policy)
      : "memory");
}

__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

// ---------------------------------------------------------------- tcgen05
// TMEM allocation is warp-collective; the base address is written to smem.
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// D[tmem] (+)= A[smem] * B[smem]^T over N consecutive 32-byte K steps, both
// operands K-major, f32 accumulate; F8: e4m3 inputs (kind::f8f6f4), else f16 or
// bf16 (kind::f16); PAIR: the 256-row MMA of a CTA pair, issued by rank 0 with
// the offsets of each CTA's halves, the same in both CTAs.  Descriptors are given
// as their low words and the high word they share; a K step inside the swizzled
// row is + 2.  One asm block per group keeps the issue loop short (full pass, a
// block per K step -> per chunk: FP8 sphere 17.9 -> 17.5 ms, others unchanged).
#define CURPLSH_MMA_STEP(I, K, P)                                                                         \
  "add.u32 x, %1, " #I ";\n\tadd.u32 y, %2, " #I ";\n\tmov.b64 a, {x, %5};\n\tmov.b64 b, {y, %5};\n\t" \
  "tcgen05.mma." K " [%0], a, b, %3, " P ";\n\t"
#define CURPLSH_MMA_BLOCK(BODY)                                                                        \
  asm volatile("{\n\t.reg .pred p, t;\n\t.reg .b32 x, y;\n\t.reg .b64 a, b;\n\t"                       \
               "setp.ne.b32 p, %4, 0;\n\tsetp.eq.u32 t, 0, 0;\n\t" BODY "}" ::"r"(d_tmem),            \
               "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(hi)                              \
               : "memory")
#define CURPLSH_MMA_N(K)                                                                               \
  if constexpr (N == 1)                                                                                \
    CURPLSH_MMA_BLOCK(CURPLSH_MMA_STEP(0, K, "p"));                                                    \
  else if constexpr (N == 2)                                                                           \
    CURPLSH_MMA_BLOCK(CURPLSH_MMA_STEP(0, K, "p") CURPLSH_MMA_STEP(2, K, "t"));                        \
  else if constexpr (N == 3)                                                                           \
    CURPLSH_MMA_BLOCK(CURPLSH_MMA_STEP(0, K, "p") CURPLSH_MMA_STEP(2, K, "t") CURPLSH_MMA_STEP(4, K, "t")); \
  else                                                                                                 \
    CURPLSH_MMA_BLOCK(CURPLSH_MMA_STEP(0, K, "p") CURPLSH_MMA_STEP(2, K, "t") CURPLSH_MMA_STEP(4, K, "t")   \
                          CURPLSH_MMA_STEP(6, K, "t"))
template <bool F8, bool PAIR, int N>
__device__ __forceinline__ void mma_steps(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc,
                                          uint32_t accumulate) {
  static_assert(N >= 1 && N <= 4, "a 128-byte swizzled chunk has four K steps");
  if constexpr (F8 && PAIR) {
    CURPLSH_MMA_N("cta_group::2.kind::f8f6f4");
  } else if constexpr (F8) {
    CURPLSH_MMA_N("cta_group::1.kind::f8f6f4");
  } else if constexpr (PAIR) {
    CURPLSH_MMA_N("cta_group::2.kind::f16");
  } else {
    CURPLSH_MMA_N("cta_group::1.kind::f16");
  }
}
#undef CURPLSH_MMA_N
#undef CURPLSH_MMA_BLOCK
#undef CURPLSH_MMA_STEP

// Arrive (once) on an mbarrier when all previously issued tcgen05 async
// operations of this thread have completed.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// 32 lanes x 64 columns of 32-bit TMEM -> 64 registers per thread
// (thread t of the warp receives lane base+t, register j = column base+j).
// The registers may be used only after tmem_ld_wait.
__device__ __forceinline__ void tmem_ld_32x32b_x64(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, %48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]), "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
      : "r"(taddr)
      : "memory");
}
// 32 lanes x 32 columns -> 32 registers per thread.
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// 32 lanes x 8 columns -> 8 registers per thread.
__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor for a K-major operand tile stored with the
// 128-byte swizzle, as laid down by a TMA load with CU_TENSOR_MAP_SWIZZLE_128B
// and a 128-byte inner box: rows of 128 B, 8-row groups 1024 B apart.
//   bits  0-13 start address >> 4      bits 16-29 leading offset >> 4 (1: unused for SW128 K-major)
//   bits 32-45 stride offset >> 4 (1024 B between 8-row groups)
//   bits 46-47 descriptor version (1 on sm_100)   bits 61-63 layout (2 = 128-byte swizzle)
// The tile base must be 1024-byte aligned; a K step inside the 128-byte atom is
// taken by advancing the start address (32 B per 16 bf16 / 32 fp8 elements).
// The low word is desc_lo(address), the high word a constant of the layout.
constexpr uint32_t kDescHiSw128 = (1024u >> 4) | (1u << 14) | (2u << 29);
// A K-major tile with the 32-byte swizzle (TMA CU_TENSOR_MAP_SWIZZLE_32B, 32-byte
// rows, 8-row groups 256 B apart), layout code 6.  One descriptor covers one K
// step of 32 bytes.  The tile base must be 256-byte aligned.
constexpr uint32_t kDescHiSw32 = (256u >> 4) | (1u << 14) | (6u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr >> 4) & 0x3FFFu) | (1u << 16); }

// ---------------------------------------------------------------- CTA pairs
// A cluster of two CTAs on neighbouring SMs runs the MMA as one 256-row
// operation (cta_group::2): each CTA holds half of A (its own 128 query rows)
// and half of B (128 of the tile's 256 database rows) in its shared memory,
// and its own 128 accumulator lanes in its TMEM.  The even CTA (rank 0) issues
// the MMAs; every load of the pair completes on rank 0's barriers.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// All threads of both CTAs; orders shared-memory accesses across the pair.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the object at `p`'s offset in CTA `rank`
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
// Arrive on the mbarrier at `bar`'s offset in CTA `rank` (release, cluster scope).
__device__ __forceinline__ void mbar_arrive_remote(uint64_t* bar, uint32_t rank) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr(bar, rank))
               : "memory");
}
// Wait that also acquires what other CTAs of the cluster released before
// arriving.
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// 2-D tiled load into this CTA's shared memory whose completion (bytes) is
// counted on rank 0's mbarrier at `bar`'s offset.  No multicast.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const void* tmap, uint64_t* bar, int c0, int c1,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(cluster_addr(bar, 0)), "r"(c0), "r"(c1), "l"(policy)
      : "memory");
}
// TMEM allocation / release for both CTAs of the pair: the same warp of
// each CTA executes it with the same column count and slot offset.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Arrive once on the mbarrier at `bar`'s offset in both CTAs of the pair
// when the issuing thread's earlier tcgen05 operations have completed.
__device__ __forceinline__ void mma_commit_pair(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b16 m;\n\tmov.b16 m, 3;\n\t"
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}" ::"r"(
          smem_u32(bar))
      : "memory");
}

// Instruction descriptor: dense, f32 accumulate, K-major A and B.
//   bits 4-5 D format (1 = f32); 7-9 A format; 10-12 B format; 17-22 N >> 3; 24-28 M >> 4.
// Formats: kind::f16 -> 0 f16, 1 bf16; kind::f8f6f4 -> 0 e4m3, 1 e5m2.
__host__ __device__ constexpr uint32_t make_idesc(uint32_t a_fmt, uint32_t b_fmt, uint32_t m, uint32_t n) {
  return (1u << 4) | (a_fmt << 7) | (b_fmt << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// ---------------------------------------------------------------- misc
// min(a, b, c) in one instruction (three-input min, sm_100).
__device__ __forceinline__ float fmin3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// One lane of a fully active warp (the same one every time).
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
  return r != 0;
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

}  // namespace curplsh_b200
