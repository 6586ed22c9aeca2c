// PTX of the kernels whose CTA pairs (clusters of two) work on one tcgen05 cta_group::2 tile.  No load is multicast.
#pragma once

#include "gv_common.cuh"

namespace gv {

// Tensor memory of both CTAs at once, `columns` in each and at the same address: PTX wants one value of .cta_group for all tcgen05
// instructions of a kernel.  A warp of either CTA takes part, both after a cluster barrier (both CTAs run) and the release before either
// exits.  No CTA of the pair can hold its half while the other waits for a neighbour's: every kernel here that allocates
// tensor memory asks for more than half of an SM's shared memory, so that no two of them share one.  (Allocated by either CTA
// for itself, as before: two feed-forward layers of 2048 tokens 390.2 us at their fastest, together 392.3; the dense MLP alone takes the same.)
__device__ __forceinline__ void pair_tmem_alloc(uint32_t* smem_result, uint32_t columns) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)), "r"(columns)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void pair_tmem_dealloc(uint32_t address, uint32_t columns) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(address), "r"(columns) : "memory");
}

__device__ __forceinline__ void pair_arrive_remote(uint64_t* local_bar, uint32_t target_cta) {
  const uint32_t remote = cluster_map_shared(smem_u32(local_bar), target_cta);
  // Relaxed: the arrive announces that tensor-memory reads have completed (tcgen05.wait::ld came
  // before it); no memory written by this thread has to be visible to the leader, and a release
  // here would first wait for the thread's earlier global stores.
  asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}

// Arrives on the barrier at the same shared-memory offset in both CTAs of the pair once every
// tcgen05 operation issued so far by this thread has completed.
__device__ __forceinline__ void pair_commit_both(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}

// Tensor-map load into this CTA's shared memory that completes on a barrier of either CTA of the
// pair (`barrier` is a shared::cluster address).  No multicast: every CTA loads its own bytes.
__device__ __forceinline__ void pair_load(void* smem_dst, const void* tensor_map, uint32_t barrier, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(smem_dst)),
      "l"(tensor_map), "r"(x), "r"(y), "r"(barrier)
      : "memory");
}

__device__ __forceinline__ void pair_load_3d(void* smem_dst, const void* tensor_map, uint32_t barrier, int x, int y,
                                           int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(smem_dst)),
      "l"(tensor_map), "r"(x), "r"(y), "r"(z), "r"(barrier)
      : "memory");
}

// 32 weight rows in the column order of grouped_gemm_down.cu (map_down_pieces): half `half` of 64-column group `group`.
__device__ __forceinline__ void pair_load_piece(void* smem_dst, const void* tensor_map, uint32_t barrier, int x, int half,
                                                int group) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2"
      " [%0], [%1, {%2, %3, %3, %4, %5}], [%6];" ::"r"(smem_u32(smem_dst)),
      "l"(tensor_map), "r"(x), "r"(0), "r"(half * 4), "r"(group), "r"(barrier)
      : "memory");
}

__device__ __forceinline__ void pair_copy_sf(uint32_t tmem_address, uint32_t hi, uint32_t lo) {
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(tmem_address),
               "l"((static_cast<uint64_t>(hi) << 32) | lo)
               : "memory");
}

__device__ __forceinline__ void pair_mma(uint32_t tmem_d, uint32_t hi, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                       uint32_t tmem_sfa, uint32_t tmem_sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X"
      " [%0], %1, %2, %3, [%5], [%6], p;\n\t"
      "}" ::"r"(tmem_d),
      "l"((static_cast<uint64_t>(hi) << 32) | a_lo), "l"((static_cast<uint64_t>(hi) << 32) | b_lo), "r"(idesc),
      "r"(accumulate), "r"(tmem_sfa), "r"(tmem_sfb)
      : "memory");
}

}  // namespace gv
