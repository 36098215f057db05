// Thin inline-PTX wrappers for the sm_100a features the kernels use:
// mbarrier (with bounded waits), TMA bulk-tensor copies, tcgen05 MMA / TMEM.
//
// Every wait in this file is bounded: a waiter that sees no progress for
// B200AIT_WAIT_LIMIT_NS records an error code in a global status word, sets a
// CTA-wide abort flag and returns, so that a broken pipeline ends with an
// error status on the host instead of a hung GPU.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200ait {

// n / d for 0 <= n < 2^31 as a multiply-high and a shift: with p = 31 + ceil(log2 d), mul = ceil(2^p / d), shr = p - 32,
// floor(n * mul / 2^p) == floor(n / d) (the rounding error n * (mul - 2^p / d) / 2^p stays below 1 / d).
struct FastDiv {
  unsigned mul = 0, shr = 0;
  explicit FastDiv(int d) {
    if (d > 1) {
      unsigned lg = 0;
      while ((1ull << lg) < static_cast<unsigned long long>(d)) ++lg;
      const unsigned pw = 31 + lg;
      mul = static_cast<unsigned>(((1ull << pw) + static_cast<unsigned>(d) - 1) / static_cast<unsigned>(d));
      shr = pw - 32;
    }
  }
};
__device__ __forceinline__ int fast_div(int n, int d, unsigned mul, unsigned shr) {
  return d == 1 ? n : static_cast<int>(__umulhi(static_cast<unsigned>(n), mul) >> shr);
}


#ifndef B200AIT_WAIT_LIMIT_NS
#define B200AIT_WAIT_LIMIT_NS 2000000000ull  // 2 s; kernels here run for milliseconds
#endif

// error codes written to the device status word (first error wins)
enum DeviceError : int {
  kDevOk = 0,
  kDevWaitFullTimeout = 1,    // MMA warp waited for a TMA stage
  kDevWaitEmptyTimeout = 2,   // producer waited for a free smem stage
  kDevWaitAccFullTimeout = 3, // epilogue waited for an accumulator
  kDevWaitAccEmptyTimeout = 4,// MMA warp waited for a free accumulator
  kDevWaitOtherTimeout = 5,
  kDevBadSmemAlignment = 6,
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// make generic-proxy smem writes visible to the async proxy (TMA / tcgen05 operands)
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
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

// Bounded wait. `abort_flag` lives in shared memory and is CTA-wide; once it is
// set every later wait returns at once. Returns false if the wait gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          int* status, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  if (*abort_flag) return false;
  uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((++spins & 255u) == 0u) {
      if (*abort_flag) return false;
      if (globaltimer_ns() - t0 > B200AIT_WAIT_LIMIT_NS) {
        *abort_flag = 1;
        if (status) atomicCAS(status, 0, code);
        return false;
      }
    }
  }
}

// Bounded wait whose acquire covers the whole cluster: for a barrier on which threads of the PEER CTA arrive
// (mbar_arrive_cluster) after writing this CTA's shared memory through the cluster window.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                                  int* status, int code) {
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((++spins & 255u) == 0u) {
      if (*abort_flag) return false;
      if (globaltimer_ns() - t0 > B200AIT_WAIT_LIMIT_NS) {
        *abort_flag = 1;
        if (status) atomicCAS(status, 0, code);
        return false;
      }
    }
  }
}
// Four consecutive 32-bit words (16-byte aligned), same contract: 16 bytes credited.
__device__ __forceinline__ void st_async_cluster_v4(uint32_t cluster_addr, uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3,
                                                    uint32_t cluster_bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                   cluster_addr),
               "r"(v0), "r"(v1), "r"(v2), "r"(v3), "r"(cluster_bar)
               : "memory");
}
// arrive on a peer CTA's mbarrier without ordering this thread's earlier writes
__device__ __forceinline__ void mbar_arrive_cluster_relaxed(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// the cluster-wide barrier in two halves (every thread of every CTA of the cluster executes each exactly once)
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// --------------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void bulk_commit_group() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// waits until the bulk groups of this thread have finished READING their shared-memory source
__device__ __forceinline__ void bulk_wait_group_read0() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_group0() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ----------------------------------------------------------------- tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ------------------------------------------------ issue by a whole, converged warp
// The operands of a tcgen05.mma sit in uniform registers. Code under `if (lane == 0)` cannot compute there: every descriptor
// is worked out in ordinary registers and moved over, about 60 cycles per MMA whatever its size (four 128 x 64 x 16 MMAs
// and a commit: 290 cycles to issue, 459 to completion). So the whole warp runs the issuing code, every wait ends in a
// vote, and only the instruction itself is predicated on the one lane chosen by elect_one(): 67 to issue, 333 to completion
// (P from TMEM: 326 and 497 -> 60 and 245). A commit covers the MMAs of the same lane.
__device__ __forceinline__ uint32_t elect_one() {  // 1 in one lane of a converged warp, 0 in the others
  uint32_t e;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
  return e;
}
// mbar_wait by a converged warp; one answer for all lanes
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status,
                                               int code) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, status, code));
}
// Shared-memory matrix descriptor of a 128-byte-swizzled tile whose rows are 128 bytes (64 half elements) apart:
//   bits  0-13 start address >> 4      bits 16-29 leading byte offset >> 4
//   bits 32-45 stride byte offset >> 4 bits 46-47 descriptor version (1 on sm_100)
//   bits 61-63 swizzle mode (2 = 128 B)
// Passed as its low word; the high word is the same for every tile here (8-row groups 1024 bytes apart).
__device__ __forceinline__ uint32_t umma_smem_desc_sw128_lo(uint32_t smem_addr, uint32_t lbo_bytes) {
  return ((smem_addr & 0x3FFFFu) >> 4) | (((lbo_bytes >> 4) & 0x3FFFu) << 16);
}
constexpr uint32_t kUmmaDescHiSw128 = (1024u >> 4) | (1u << 14) | (2u << 29);
// `lead`: elect_one()'s answer.
// D[tmem] (+)= A[smem] * B[smem]; accumulate == 0 overwrites D
__device__ __forceinline__ void umma_f16_ss_warp(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                                 uint32_t accumulate, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %6, 0;\n\t"
      "mov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(kUmmaDescHiSw128), "r"(lead)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_f16_ts_warp(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc,
                                                 uint32_t accumulate, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %6, 0;\n\t"
      "mov.b64 b, {%2, %5};\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(kUmmaDescHiSw128), "r"(lead)
      : "memory");
}
// the mbarrier receives one arrival when every tcgen05 op issued so far by the elected lane is done
__device__ __forceinline__ void umma_commit_warp(uint64_t* bar, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %1, 0;\n\t"
      "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)),
      "r"(lead)
      : "memory");
}

// TMA copies take their operands from uniform registers as well.
__device__ __forceinline__ void mbar_arrive_expect_tx_warp(uint64_t* bar, uint32_t bytes, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %2, 0;\n\t"
      "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
      "r"(bytes), "r"(lead)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_warp(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar, int c0, int c1,
                                                 int c2, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %6, 0;\n\t"
      "@e cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}" ::
          "r"(smem_dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(lead)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_warp(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar, int c0, int c1,
                                                 int c2, int c3, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %7, 0;\n\t"
      "@e cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
      "[%2];\n\t}" ::"r"(smem_dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(lead)
      : "memory");
}

// TMA store of one box from shared memory (bulk-group completion)
__device__ __forceinline__ void tma_store_5d_warp(const CUtensorMap* m, uint32_t smem_src, int c0, int c1, int c2, int c3,
                                                  int c4, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %7, 0;\n\t"
      "@e cp.async.bulk.tensor.5d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];\n\t}" ::"l"(
          reinterpret_cast<uint64_t>(m)),
      "r"(smem_src), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(lead)
      : "memory");
}

// ------------------------------------------------ CTA pairs (cluster of two)
// Two CTAs of one cluster share one MMA: tcgen05 instructions with cta_group::2 are issued by the
// even CTA (rank 0, "leader"); each CTA keeps its own operands in its own shared memory and its own
// 128 accumulator rows in its own TMEM.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {  // every thread of every CTA of the cluster
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the same shared-memory location in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t mapa_shared(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// TMA load by either CTA of a pair; the byte count is credited to the mbarrier at `bar_cluster_addr`, which may live in the
// peer CTA. No multicast: the data lands in the issuing CTA.
__device__ __forceinline__ void tma_load_3d_pair_warp(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar_cluster_addr,
                                                      int c0, int c1, int c2, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %6, 0;\n\t"
      "@e cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];\n\t}" ::"r"(smem_dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster_addr), "r"(c0), "r"(c1), "r"(c2), "r"(lead)
      : "memory");
}
// D (256 rows: 128 in each CTA's TMEM) (+)= A (128 rows per CTA) * B (N/2 rows per CTA)
__device__ __forceinline__ void umma_f16_ss_pair_warp(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                                      uint32_t accumulate, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %6, 0;\n\t"
      "mov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
      "@e tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "n"(kUmmaDescHiSw128), "r"(lead)
      : "memory");
}
// one arrival on the mbarrier at this shared-memory offset in every CTA of `cta_mask`
__device__ __forceinline__ void umma_commit_pair_warp(uint64_t* bar, uint16_t cta_mask, uint32_t lead) {
  asm volatile(
      "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %2, 0;\n\t"
      "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(
          smem_u32(bar)),
      "h"(cta_mask), "r"(lead)
      : "memory");
}

// Instruction descriptor for kind::f16 with fp32 accumulation.
//   bits 4-5 D format (1 = f32)   bits 7-9 A format   bits 10-12 B format (0 = f16, 1 = bf16)
//   bit 15 A major, bit 16 B major (0 = K-major, 1 = MN-major)
//   bits 17-22 N >> 3             bits 24-28 M >> 4
__host__ __device__ constexpr uint32_t umma_idesc_f16(int m, int n, bool bf16, bool a_mn_major, bool b_mn_major) {
  return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((a_mn_major ? 1u : 0u) << 15) |
         ((b_mn_major ? 1u : 0u) << 16) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(m >> 4) << 24);
}

// TMEM -> registers: this warp's 32 lanes x 32 consecutive 32-bit columns (one row per thread)
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// registers -> TMEM, same shape as tmem_ld_32x32b_x16
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
      "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Packed fp32 arithmetic of sm_100 (two lanes per instruction) and the three-input max: they halve the count
// of FMA / add / mul / max instructions in the softmax threads and in the GEMM epilogue.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// Kernels launched by launch_early (common.h) may be resident before the kernel ahead of them on the stream has finished:
// everything that reads or writes global memory comes after grid_wait, which every thread of every CTA calls (a CTA that left
// without it could let the next kernel but one start too early). What it reads there may still have been written while it was
// resident, which rules out the read-only path (__ldg, `const T* __restrict__` parameters: their data must not change while the
// kernel is resident, and the compiler may move such a load above the wait) and loads whose place the compiler does not
// know to matter (__ldcs). So such kernels read through plain pointers or by ld_stream.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// a load with the streaming hint, which stays where it is written
template <typename V>
__device__ __forceinline__ V ld_stream(const V* p) {
  static_assert(sizeof(V) == 16 || sizeof(V) == 8 || sizeof(V) == 4 || sizeof(V) == 2 || sizeof(V) == 1, "a vector or an element");
  if constexpr (sizeof(V) == 16) {
    uint4 v;
    asm volatile("ld.global.cs.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
  } else if constexpr (sizeof(V) == 8) {
    uint2 v;
    asm volatile("ld.global.cs.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
  } else if constexpr (sizeof(V) == 4) {
    uint32_t v;
    asm volatile("ld.global.cs.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
  } else if constexpr (sizeof(V) == 2) {
    uint16_t v;
    asm volatile("ld.global.cs.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
  } else {
    uint16_t v;
    asm volatile("ld.global.cs.u8 %0, [%1];" : "=h"(v) : "l"(p));
    return static_cast<V>(v);
  }
}
// The next kernel's CTAs may become resident once every CTA of this grid has called this or has left. A kernel that allocates
// tensor memory calls it after its allocation: a waiting CTA of the next kernel must not hold the columns that this one needs.
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// arrives at a named barrier (and publishes what was written before) without waiting for the others
__device__ __forceinline__ void named_bar_arrive(int id, int nthreads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
// named barrier among a subset of the CTA's warps
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
}  // namespace b200ait
