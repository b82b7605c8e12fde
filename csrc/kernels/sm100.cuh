// Blackwell (sm_100a) device primitives shared by every kernel in this library:
// mbarrier with bounded waits, TMA (cp.async.bulk.tensor, always one destination CTA),
// tcgen05 MMA / TMEM allocation / TMEM loads, UMMA shared-memory and instruction
// descriptors, and the host-side tensor-map encoder.
//
// Conventions
//   * Every wait is bounded: after kSpinLimitCycles the waiter records an error code
//     in a global status word and the kernel unwinds (frees TMEM, returns).
//   * Operand tiles in shared memory are K-major, 128-byte swizzled, 1024-byte aligned:
//     a tile of R rows x 64 bf16 columns occupies R*128 bytes; 8-row groups are 1024 B
//     apart (the UMMA "stride byte offset").
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <atomic>
#include <stdint.h>

namespace b200 {

// ------------------------------------------------------------------------------------
// Error status (one word per process, written by kernels whose bounded wait ran out)
// ------------------------------------------------------------------------------------
enum KernelError : int {
  kErrNone = 0,
  kErrMbarTimeout = 1,   // an mbarrier wait inside a pipeline gave up
  kErrFlagTimeout = 2,   // a peer flag wait (fused collective) gave up
  kErrBadArg = 3,
  kErrBadAlign = 4,      // dynamic shared memory base not 1024-byte aligned
};

// 2^31 cycles is about 1.1 s at 1.9 GHz.
static constexpr long long kSpinLimitCycles = 1ll << 31;
// Waits on another GPU's progress allow for host-side jitter between ranks (about 9 s).
static constexpr long long kPeerWaitCycles = 1ll << 34;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// True in one lane of the (whole) calling warp, the same one at every call: elect.sync names the same leader for the same mask. Commits rely
// on it, as each covers what its own thread has issued.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(pred));
  return pred != 0;
}

// ------------------------------------------------------------------------------------
// mbarrier
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
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
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Pure poll (never suspends the thread), for issuers that watch several barriers at once.
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait. Returns false (and records the error) when the limit is reached.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status) {
  if (mbar_try_wait(bar, parity)) return true;
  long long t0 = clock64();
  uint32_t it = 0;
  while (!mbar_try_wait(bar, parity)) {
    if (((++it) & 0x3ff) == 0) {
      if (clock64() - t0 > kSpinLimitCycles) {
        if (status) atomicExch(status, (int)kErrMbarTimeout);
        return false;
      }
    }
  }
  return true;
}

// The whole warp waits, with one answer for all lanes. An issuing warp walks its loop as one and lets elect_one() pick the lane
// that issues: stage addresses and descriptors then stay in uniform registers, where tcgen05.mma and TMA take them from. In code
// of one lane each of them is moved there first, which bounded every product whose instructions are short.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, int* status) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, status));
}
// Index of the calling warp, known to the compiler as the same for all its lanes.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// Same, for single-thread producer / issuer warps that share their SM sub-partition with warps
// doing real work: sleeps between polls so that the polling does not compete for issue slots.
__device__ __forceinline__ bool mbar_wait_backoff(uint64_t* bar, uint32_t parity, int* status) {
  if (mbar_try_wait(bar, parity)) return true;
  long long t0 = clock64();
  uint32_t it = 0;
  while (!mbar_try_wait(bar, parity)) {
    __nanosleep(48);
    if (((++it) & 0x3ff) == 0) {
      if (clock64() - t0 > kSpinLimitCycles) {
        if (status) atomicExch(status, (int)kErrMbarTimeout);
        return false;
      }
    }
  }
  return true;
}

// Make generic-proxy shared-memory writes visible to the async proxy (TMA / tcgen05).
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ------------------------------------------------------------------------------------
// TMA loads / stores (tiled). Each copy lands in the issuing CTA only.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* m, uint64_t* bar,
                                            int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0),
      "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* m, uint64_t* bar,
                                            int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0),
      "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* m, const void* src, int c0,
                                             int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
      ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(src)), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_store_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}

// ------------------------------------------------------------------------------------
// tcgen05: TMEM allocation, MMA issue, commit, TMEM -> register loads
// ------------------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  // One full warp executes this; ncols is a power of two in [32, 512].
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// D[tmem] (+)= A[smem desc] * B[smem desc]; bf16/f16 inputs, f32 accumulate.
__device__ __forceinline__ void umma_bf16_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Same with the A operand read from TMEM (used by attention: P stays in TMEM).
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc,
                                             uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Eight e2m1 nibbles (low nibble first) -> four f16x2.
__device__ __forceinline__ void cvt_e2m1x8(uint32_t w, uint32_t (&h)[4]) {
  asm volatile(
      "{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
      "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
      "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
      "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
      "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
      "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}\n"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
      : "r"(w));
}
// fp8 (e4m3/e5m2) and other narrow formats, f32 accumulate, K = 32 per instruction.
__device__ __forceinline__ void umma_f8f6f4_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                               uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// NVFP4 block-scaled: E2M1 x E2M1 with UE4M3 scale factors (one per 16 elements) read
// from TMEM; K = 64 per instruction.
__device__ __forceinline__ void umma_nvfp4_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                              uint32_t idesc, uint32_t tmem_sfa,
                                              uint32_t tmem_sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X "
      "[%0], %1, %2, %3, [%4], [%5], p;\n\t}\n"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(tmem_sfa), "r"(tmem_sfb),
      "r"(accumulate)
      : "memory");
}
// smem -> TMEM copy of scale factors: 32 lanes x 128 bits, replicated to the 4 lane quarters.
__device__ __forceinline__ void tmem_cp_32x128b_warpx4(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc)
               : "memory");
}

// All previously issued MMAs of this thread arrive on `bar` when they complete.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}

// ------------------------------------------------------------------------------------
// CTA pairs (cta_group::2): two CTAs of a cluster share one MMA. The even CTA issues it; A rows
// and B rows of each half come from that CTA's own shared memory, each CTA's TMEM receives its
// 128 rows of D. Loads carry no cluster multicast: each CTA fetches its own halves.
// ------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared::cluster address of the same shared-memory offset in CTA `rank` of this cluster.
__device__ __forceinline__ uint32_t mapa_u32(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
// Sum of four columns over S CTAs of the cluster from rank `first` on, in their order.
template <int S>
__device__ __forceinline__ float4 sum_of(uint32_t addr, int first) {
  float4 v[S];
#pragma unroll
  for (int s = 0; s < S; ++s) v[s] = ld_cluster_f4(mapa_u32(addr, first + s));
#pragma unroll
  for (int s = 1; s < S; ++s) { v[0].x += v[s].x; v[0].y += v[s].y; v[0].z += v[s].z; v[0].w += v[s].w; }
  return v[0];
}
// Arrive on an mbarrier of another CTA of the cluster (address from mapa_u32).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load of this CTA's tile whose bytes are counted on the pair leader's mbarrier.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* m, uint32_t leader_bar,
                                                 int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(leader_bar), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* dst, const CUtensorMap* m, uint32_t leader_bar,
                                                 int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(leader_bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void umma_bf16_ss_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                                  uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_f8f6f4_ss_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                                    uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The pair's MMAs issued so far arrive on the mbarrier at this offset in every CTA of `mask`.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(smem_u32(bar)), "h"(mask)
      : "memory");
}

// TMEM -> registers: this warp's 32 lanes x 32 consecutive fp32 columns.
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// registers -> TMEM: this warp's 32 lanes x 32 consecutive 32-bit columns.
__device__ __forceinline__ void tmem_st_32x32b_x32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
      "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
      "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
      "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
      "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// ------------------------------------------------------------------------------------
// Descriptors
// ------------------------------------------------------------------------------------
// Shared-memory matrix descriptor, K-major, 128-byte swizzle (layout type 2), descriptor
// version 1 (Blackwell). `sbo_bytes` = distance between consecutive 8-row groups.
__device__ __forceinline__ uint64_t umma_desc_k_sw128(uint32_t smem_addr, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3fff);
  d |= (uint64_t)1 << 16;                               // leading byte offset (unused here)
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3fff) << 32;     // stride byte offset
  d |= (uint64_t)1 << 46;                               // version
  d |= (uint64_t)2 << 61;                               // SWIZZLE_128B
  return d;
}
// MN-major operand (the contiguous dimension is M or N, not K), 128-byte swizzle.
// A tile is stored as [k rows][64 mn elements] = 128-byte rows; 8 k-rows form a 1024 B
// swizzle atom. `lbo_bytes` = distance between consecutive 64-element MN blocks,
// `sbo_bytes` = distance between consecutive 8-row K groups.
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smem_addr, uint32_t lbo_bytes,
                                                       uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3fff);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3fff) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3fff) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// No-swizzle K-major descriptor for 8x(16 B) core matrices (used for scale-factor copies).
__device__ __forceinline__ uint64_t umma_desc_noswizzle(uint32_t smem_addr, uint32_t lbo_bytes,
                                                        uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr >> 4) & 0x3fff);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3fff) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3fff) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// Instruction descriptor for kind::f16 with bf16 A/B and f32 accumulation.
// a_mn / b_mn: 0 = K-major operand, 1 = MN-major operand.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n, int a_mn = 0,
                                                       int b_mn = 0) {
  return (1u << 4)                      // D format: f32
         | (1u << 7)                    // A format: bf16
         | (1u << 10)                   // B format: bf16
         | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16)
         | ((uint32_t)(n >> 3) << 17)   // N / 8
         | ((uint32_t)(m >> 4) << 24);  // M / 16
}
// kind::f8f6f4 with e4m3 A/B, f32 accumulation.
__host__ __device__ constexpr uint32_t umma_idesc_e4m3(int m, int n) {
  return (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}
// kind::mxf4nvf4 block-scaled: E2M1 A/B (format 1), UE4M3 scales (scale_format 0).
__host__ __device__ constexpr uint32_t umma_idesc_nvfp4(int m, int n, int sfa_id = 0,
                                                        int sfb_id = 0) {
  return ((uint32_t)sfb_id << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         (0u << 23) | ((uint32_t)(m >> 4) << 24) | ((uint32_t)sfa_id << 29);
}

// ------------------------------------------------------------------------------------
// Small numeric helpers
// ------------------------------------------------------------------------------------
// Warp-wide float max in one instruction (sm_100a).
__device__ __forceinline__ float warp_max_f32(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t v) {
  __nv_bfloat162 b = *reinterpret_cast<__nv_bfloat162*>(&v);
  return __bfloat1622float2(b);
}

// Pairs of floats in one 64-bit register: one instruction for both (each rounded like the scalar one).
__device__ __forceinline__ uint64_t pack_b32x2(uint32_t lo, uint32_t hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
  return r;
}
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) { return pack_b32x2(__float_as_uint(lo), __float_as_uint(hi)); }
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// x sigmoid(x) as |x| n / (1 + e) with e = exp(-|x|), n = 1 or e, and the sign of x: the denominator lies between 1 and 2, where an
// approximate reciprocal and one Newton step on the quotient, with what rounding took from |x| n and 1 + e put back, take the place of a
// division and its special cases. That adds less than 2^-22 to what __expf's own error (2 + 1.173 |x| units in its last place) leaves in the
// result, x / (1 + exp(-x)) no less; zeros keep their sign, infinities and NaN do as in that form. It is the time of the gated epilogues: a
// thread computes 128 of them a tile (8192 x 28672 x 4096 in fp8: 897 us with the division, 670 with this, 667 without an activation).
__device__ __forceinline__ float silu_of(float x) {
  const float a = fabsf(x), e = __expf(-a), d = 1.f + e, d_low = e - (d - 1.f), n = x >= 0.f ? 1.f : e;
  const float m = a * n, m_low = fmaf(a, n, -m);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = m * r;
  const float s = fmaf(fmaf(-q, d_low, fmaf(-q, d, m)) + m_low, r, q);
  return x > 30.f ? x : copysignf(s, x);               // (exact there, and infinity stays)
}
// Activation of a gated block, act(gate) * up. One formula for every kernel that applies it, in an epilogue or on its own: their
// results are the same bits.
enum ActKind : int { kSilu = 0, kGeluTanh = 1, kGeluErf = 2 };
__device__ __forceinline__ float act_of(float g, int kind) {
  if (kind == kSilu) return silu_of(g);
  if (kind == kGeluTanh) return 0.5f * g * (1.f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g)));
  return 0.5f * g * (1.f + erff(g * 0.7071067811865476f));
}

}  // namespace b200

// ------------------------------------------------------------------------------------
// Host side: tensor-map encoding through the driver entry point (no link against libcuda)
// ------------------------------------------------------------------------------------
namespace b200 {
// Encodes a row-major 2-D bf16/byte tensor [rows, cols] with leading dimension `ld`
// (elements) as a TMA map with box [box_rows, box_cols] and the given swizzle.
// Returns false if the driver rejects it.
bool encode_tmap_2d(CUtensorMap* out, const void* base, CUtensorMapDataType dtype,
                    size_t elem_bytes, uint64_t rows, uint64_t cols, uint64_t ld_elems,
                    uint32_t box_rows, uint32_t box_cols, CUtensorMapSwizzle swizzle);
// 3-D variant: dims (d0 fastest). strides in bytes for d1 and d2.
bool encode_tmap_3d(CUtensorMap* out, const void* base, CUtensorMapDataType dtype,
                    size_t elem_bytes, uint64_t d0, uint64_t d1, uint64_t d2,
                    uint64_t stride1_bytes, uint64_t stride2_bytes, uint32_t b0, uint32_t b1,
                    uint32_t b2, CUtensorMapSwizzle swizzle);
// bf16 matrix with 128-byte swizzled boxes; the maps of a process are kept (gemm_bf16.cu).
bool get_tmap_bf16(CUtensorMap* out, const void* p, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t br, uint32_t bc);

// What a QKV product does with its result before it stores it: per-head RMSNorm of q and k, full NeoX rotation of 128-dim heads, k and v into
// the paged cache [num_blocks, 2, block_size, Hkv, 128] too (b200_rope_kv, in the epilogue).
struct RopeOut {
  int Hq, Hkv;               // columns of the product: q heads | k heads | v heads
  const int64_t* positions;
  const float* cos_sin;      // [max_pos, 128]
  const __nv_bfloat16 *q_norm, *k_norm;
  float eps;
  int gemma;
  const int64_t* slot_mapping;
  __nv_bfloat16* kv_cache;
  int block_size;
};

// Product of at most 128 rows with K split over a cluster (gemm_cluster.cu).
struct GemmCluster {
  const void *A, *W;
  void* out;
  const void *bias, *residual;
  int lda, ldw, ldr, M, N, K;
  long long ldo;
  int out_f32, act;          // act: act_epilogue
  int gated;                 // 1 + kind: W in blocks of [128 gate | 128 up] rows, out[M, N / 2] = act(gate) * up
  int w_early;               // W is constant: fetched before the predecessor kernel has finished
  int splits;                // CTAs that share a row tile (0: chosen)
  int batch;                 // products side by side (gridDim.z)
  int batch_a_cols;
  long long batch_out;
  // e4m3 A and W (set a_scale): the sums times a_scale (per tensor or row) and w_scale (per tensor or column)
  const float *a_scale, *w_scale;
  int a_per_row, w_per_col;
  const RopeOut* rope;       // (not gated, not batched, N = (Hq + 2 Hkv) 128)
};
int launch_gemm_cluster(const GemmCluster& g, cudaStream_t stream);
bool fp8_rows_cluster(int M, int N, int K);      // whether an e4m3 product is faster so (gemm_quant.cu)

// One or two rows, on the CUDA cores; optionally with the residual addition and RMSNorm of the rows in front (gemv.cu).
struct GemvNorm {
  const void *weight, *res_in;      // res_in: [M, K] or null
  void* res_out;                    // [M, K], another buffer than res_in
  float eps;
  int gemma;
};
bool gemv_takes(int M, int N, int K);
int launch_gemv(const GemmCluster& g, const GemvNorm* norm, cudaStream_t stream);

// The same for the rows of a sorted batch, each chunk of them with its expert's weights (gemm_cluster.cu).
struct ExpertsCluster {
  const void *xs, *W;        // [max_rows + 256, K], [E, N, K]
  void* out;
  const int32_t *chunk_expert, *chunk_row0, *chunk_n, *num_chunks;
  int max_rows, max_chunks, E, N, K, gated, act;
};
int launch_experts_cluster(const ExpertsCluster& g, cudaStream_t stream);

// Process-wide device status word (lazily allocated per device).
int* device_status_word();
void clear_tile_counters();      // of the products whose tiles several CTAs share (gemm_bf16.cu), with the device idle
long long peer_wait_cycles();   // current limit of waits on other GPUs (b200_set_peer_wait_cycles)

// ------------------------------------------------------------------------------------
// Programmatic dependent launch. A kernel launched through launch_pdl() may become resident
// while its predecessor in the stream is still running: everything it does before pdl_wait()
// (barrier init, TMEM allocation, descriptor prefetch) overlaps the predecessor's tail, and
// pdl_wait() returns only when the predecessor grid has completed and its writes are visible.
// Rule for kernels launched this way: no global read of produced data and no global write before
// pdl_wait(). pdl_launch_dependents() only affects when the successor may become resident; both
// instructions are no-ops in a kernel launched the ordinary way. It is called right after pdl_wait(): ahead of it the
// successors' successors come in as well, and a step of one row of the 8B shape took 4.3 instead of 3.7 ms.
// B200_PDL=0 in the environment makes launch_pdl() an ordinary launch.
// ------------------------------------------------------------------------------------
bool pdl_enabled();
// Per-device once flag for settings that belong to a (function, device) pair, such as
// cudaFuncSetAttribute: first() is true exactly once for every device that is current when it
// is called (up to 64 devices per process).
struct PerDeviceOnce {
  std::atomic<unsigned long long> done{0};
  bool first() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return true;
    const unsigned long long bit = 1ull << dev;
    return (done.fetch_or(bit) & bit) == 0;
  }
};
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(static_cast<Args&&>(args))...);
}
// The same for a grid of clusters of `ranks` CTAs (1: none).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_cluster_pdl(void (*kernel)(KArgs...), dim3 grid, int ranks, int threads, size_t smem, cudaStream_t stream,
                                      Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  if (ranks > 1) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    attr[cfg.numAttrs].val.clusterDim.x = (unsigned)ranks;
    attr[cfg.numAttrs].val.clusterDim.y = 1;
    attr[cfg.numAttrs++].val.clusterDim.z = 1;
  }
  if (pdl_enabled()) {
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(static_cast<Args&&>(args))...);
}
#endif
// Dynamic shared memory for a kernel whose CTAs allocate `cols` of an SM's 512 columns of tensor memory and meet in clusters: `smem`, or,
// where more of them fit an SM (`fit` CTAs, as far as registers, threads and `smem` bytes each go) than find columns, enough to keep the
// others out. One CTA too many would wait in tcgen05.alloc, without limit, for columns of CTAs that may themselves be waiting, in a
// cluster barrier, for a CTA that waits in the same way on another SM.
constexpr size_t kSmBytes = 228 * 1024;        // shared memory of an SM
// CTAs that the registers of an SM let in at most: four parts of 16384, of which a warp takes its own from one, in pieces of 256.
constexpr int ctas_by_registers(int regs, int threads) {
  const int warp = ((regs < 1 ? 1 : regs) + 7) / 8 * 256;
  return 4 * (16384 / warp) / ((threads + 31) / 32);
}
constexpr size_t tmem_bound_smem(size_t smem, int fit, int cols) {
  const int most = 512 / cols;
  const size_t least = kSmBytes / (most + 1) + 1;
  return fit <= most || smem >= least ? smem : least;
}
// CTAs of two to an SM that share the K of each of `tiles` row tiles: as many as one wave holds, `most` at most (gemm_cluster.cu).
int cluster_splits(int tiles, int most);
// Activations in the epilogue of a product: 0 none, 1 SiLU, 2 GELU-tanh, 3 GELU-erf, 4 squared ReLU. FAST (results that are
// rounded to bf16): 0.5 (1 + tanh u) = 1 / (1 + e^(-2 u)) with the approximate exponential and quotient.
template <bool FAST>
__device__ __forceinline__ float act_epilogue(float x, int act) {
  if (act == 4) { x = fmaxf(x, 0.f); return x * x; }
  if (act == 2) {
    const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    return FAST ? __fdividef(x, 1.f + __expf(-2.f * u)) : 0.5f * x * (1.f + tanhf(u));
  }
  if (act == 1) return FAST ? __fdividef(x, 1.f + __expf(-x)) : x / (1.f + expf(-x));
  if (act == 3) return 0.5f * x * (1.f + erff(x * 0.7071067811865476f));
  return x;
}
template <bool FAST, int N>
__device__ __forceinline__ void act_epilogue(float (&v)[N], int act) {
  if (act == 2) {                                // (one loop per activation, so that none tests which it is)
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = act_epilogue<FAST>(v[i], 2);
  } else if (act == 4) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = act_epilogue<FAST>(v[i], 4);
  } else if (act == 1) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = act_epilogue<FAST>(v[i], 1);
  } else if (act == 3) {
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = act_epilogue<FAST>(v[i], 3);
  }
}

}  // namespace b200
