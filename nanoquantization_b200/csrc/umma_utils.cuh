// tcgen05 / tensor-memory helpers (sm_100a): allocation, register<->TMEM moves,
// the MMA itself, commit, the fences that order them against mbarriers, and the bounded waits of the kernels' roles.
#pragma once
#include <stdint.h>
#include "nqb200.h"
#include "tma_utils.cuh"

namespace nqb200 {

// 32-bit instruction descriptor of tcgen05.mma kind::f16: fp32 accumulate, A and B both
// K-major, `fmt` 0 = f16, 1 = bf16, shape M x N (M = 128 here).
__host__ __device__ constexpr uint32_t umma_idesc(int fmt, int M, int N) {
  return (1u << 4) | ((uint32_t)fmt << 7) | ((uint32_t)fmt << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Shared-memory operand descriptor, K-major tile written by TMA with the 128-byte swizzle:
// rows of 128 bytes, groups of 8 rows 1024 bytes apart.  `addr` is a shared-space address.
__device__ __forceinline__ uint64_t umma_smem_desc_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);   // start address
  d |= (uint64_t)1 << 16;                    // leading byte offset: unused for swizzled K-major
  d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                    // descriptor version for sm_100
  d |= (uint64_t)2 << 61;                    // SWIZZLE_128B
  return d;
}

__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// The mbarrier receives one arrival when every MMA issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// True in one lane of a converged warp.  What issues tensor-core and TMA instructions runs as a whole warp through control flow
// that is the same for all lanes (warp_index(), votes on the waits) and puts only the instruction itself under this: its operands
// then live in uniform registers, where under "if (lane == 0)" every operand has to be moved there for every instruction.  Two-SM
// prefill kernel, 777 tokens of 12288 -> 4096 79 -> 68 us; experts' grouped GEMM 497 -> 447; prompt attention 647 -> 575.
__device__ __forceinline__ bool elect_one() {
  uint32_t r;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(r));
  return r != 0;
}
// The warp's index, known to be the same in all its lanes.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// A wait suspends in hardware for up to kSuspendNs at a time (woken at once when the phase completes), so that warps which
// wait most of the time hardly issue; the clock is read only after a suspension that ran out.
constexpr uint32_t kSuspendNs = 20000;
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status) {
  const uint32_t b = smem_u32(bar);
  if (mbar_test_wait(b, parity)) return true;
  unsigned long long t0 = 0;
  while (!mbar_try_wait_suspend(b, parity, kSuspendNs)) {
    if (*abort_flag) return false;
    const unsigned long long t = global_timer_ns();
    if (!t0) t0 = t;
    if (t - t0 > kWaitLimitNs) {
      *abort_flag = 1;
      if (status) atomicExch(status, NQB200_ERR_WAIT_TIMEOUT);
      return false;
    }
  }
  return true;
}
// The same for a whole warp, whose lanes go on together (the vote keeps its control flow uniform, see elect_one).
__device__ __forceinline__ bool wait_bar_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status) {
  return __all_sync(0xffffffffu, wait_bar(bar, parity, abort_flag, status));
}

// 16 lanes x 128 bits, twice: thread (g = lane/4, t = lane%4) supplies
//   r0 -> (lane g, column t)   r1 -> (lane g+8, column t)   r2 -> (lane g, column t+4)   r3 -> (lane g+8, column t+4)
__device__ __forceinline__ void tmem_st_16x128b_x2(uint32_t taddr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x2.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r0), "r"(r1), "r"(r2), "r"(r3) : "memory");
}

// The same, four times: columns t, t+4, t+8, t+12.
__device__ __forceinline__ void tmem_st_16x128b_x4(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// ---- CTA pairs (cta_group::2): one MMA spans the tensor memory of the two CTAs of a cluster ----
__device__ __forceinline__ uint32_t cluster_ctarank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the shared::cluster address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank)); return r;
}
// Arrival on a barrier of a CTA of this cluster (an address from map_to_cta).  What the arrival reports here is
// tensor-memory traffic that tcgen05.wait and tcgen05.fence have already ordered, and shared memory that TMA wrote
// and an mbarrier announced, so the default semantics (release at CTA scope) are used: ".release.cluster" puts a
// fence of several hundred ns in front of every arrival (measured: 8 % of the two-CTA GEMM's time).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// `bar` is a shared::cluster address: the barrier may live in either CTA of the pair.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// D[tmem] (+)= A[tmem] * B[smem descriptor], issued by one thread for the CTA, or for a pair: M = 256, 128 rows of A and D in each
// CTA's tensor memory, B is N x K with N/2 rows in each CTA's shared memory.  The 64-bit shared-memory descriptor comes as its two halves
// (the high half is constant for a kernel, the low half is a base plus an offset: one 32-bit add per MMA for the issuing thread).
__device__ __forceinline__ void umma_ts_lohi(uint32_t d_tmem, uint32_t a_tmem, uint32_t desc_lo, uint32_t desc_hi, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile("{\n .reg .pred p;\n .reg .b64 d;\n setp.ne.b32 p, %5, 0;\n mov.b64 d, {%2, %3};\n"
               " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d, %4, p;\n}"
               ::"r"(d_tmem), "r"(a_tmem), "r"(desc_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_ts_pair_lohi(uint32_t d_tmem, uint32_t a_tmem, uint32_t desc_lo, uint32_t desc_hi, uint32_t idesc,
                                                  uint32_t accumulate) {
  asm volatile("{\n .reg .pred p;\n .reg .b64 d;\n setp.ne.b32 p, %5, 0;\n mov.b64 d, {%2, %3};\n"
               " tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], d, %4, p;\n}"
               ::"r"(d_tmem), "r"(a_tmem), "r"(desc_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate) : "memory");
}

// Two 8x8 matrices of 16-bit elements, transposed: lanes 0-7 give the row addresses of matrix 0, lanes 8-15
// of matrix 1; register i of thread (g = lane / 4, t = lane % 4) holds elements [2t][g] (low half) and
// [2t+1][g] (high half) of matrix i.
__device__ __forceinline__ void ldmatrix_x2_trans(uint32_t& r0, uint32_t& r1, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0, %1}, [%2];" : "=r"(r0), "=r"(r1) : "r"(addr) : "memory");
}

// Four of them: lanes 8j..8j+7 give the row addresses of matrix j.
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}

// Four, not transposed: register i of thread (g, t) holds elements [g][2t] and [g][2t+1] of matrix i.
__device__ __forceinline__ void ldmatrix_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr) : "memory");
}

// 32 lanes x 32 bits: thread i of the warp reads lane (base + i), N consecutive columns.
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_32x32b_x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr) : "memory");
}
}  // namespace nqb200
