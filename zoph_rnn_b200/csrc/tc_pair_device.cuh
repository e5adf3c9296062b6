// tcgen05 on pairs of CTAs (cta_group::2): the two CTAs of a cluster share one MMA of 256 rows, each holds 128 rows of the first
// operand and half of the second one's rows, and each keeps the accumulators of its own 128 rows.  The CTA of rank 0 leads: it
// issues the MMAs, and the full barriers of the operand ring are its own.
#pragma once
#include "tc_chain_device.cuh"

namespace zrnn {
namespace {

// as make_idesc, with M = 256 over both CTAs
__host__ __device__ constexpr uint32_t make_idesc_pair(uint32_t fmt, uint32_t n) {
  return (1u << 4) | (fmt << 7) | (fmt << 10) | ((n >> 3) << 17) | ((256u >> 4) << 24);
}
template <int KIND_TF32>
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  if (KIND_TF32) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        :
        : "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        :
        : "r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
  }
}
// the MMAs issued so far, when complete, arrive on the barrier at this place in both CTAs
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
               "h"((uint16_t)3)
               : "memory");
}
// as tma_load_4d / tma_load_5d: into this CTA's shared memory, the bytes counted on a barrier of either CTA (a shared::cluster address)
__device__ __forceinline__ void tma_load_4d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar, int y, int kb) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %3, %5}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(map), "r"(bar), "r"(0), "r"(y), "r"(kb)
      : "memory");
}
__device__ __forceinline__ void tma_load_5d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar, int y, int part, int kb) {
  asm volatile(
      "cp.async.bulk.tensor.5d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %3, %5, %6}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(map), "r"(bar), "r"(0), "r"(y), "r"(part), "r"(kb)
      : "memory");
}
// arrival on the leader's barrier at this place.  What it hands over is tensor memory, ordered by tcgen05.fence: a release at cluster
// scope would wait for the thread's earlier global stores as well
__device__ __forceinline__ void mbar_arrive_leader(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_map(smem_u32(bar), 0)) : "memory");
}
// both CTAs allocate and free, one warp each (the same warp number)
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* base, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(base)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free_pair(uint32_t base, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}

}  // namespace
}  // namespace zrnn
