// tcgen05 with `cta_group::2`: the instructions a CTA pair (a cluster of two
// CTAs on neighbouring SMs) uses to run ONE MMA over both CTAs' shared memory
// and tensor memory.  Inline PTX, sm_100a only.
//
//  * TMEM is allocated and freed by one warp of EACH CTA with the pair forms.
//  * Each CTA loads its own operand tiles with an ordinary TMA load whose
//    completion bytes are counted on a barrier of the LEADER CTA (rank 0 of
//    the cluster), addressed through `mapa`.  No load carries a
//    cluster-multicast qualifier.
//  * The leader's MMA thread issues the MMA and commits it with a multicast
//    arrive (`tcgen05.commit ... multicast::cluster`, mask 0b11) so that the
//    same barrier offset in both CTAs learns that the operands are free / the
//    accumulator is complete.
#pragma once
#include <cuda.h>
#include <stdint.h>

#include "mbarrier.cuh"

namespace smr {

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `smem_addr` (a shared::cta address) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 2-D tile load whose completion bytes land on a barrier that may sit in the
// peer CTA of the pair (address in the shared::cluster window).
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map,
                                                 uint32_t bar_cluster_addr, int32_t x, int32_t y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr),
        "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
               ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// `kCollect`: what becomes of A in the tensor core's operand buffer.  Two MMAs with the same A and different B read A from
// shared memory once if the first fills the buffer and the second is its last use.
enum class CollectA { kDiscard, kFill, kLastUse };
#define SMR_UMMA_PAIR(KIND, COLLECT)                                                              \
  asm volatile(                                                                                   \
      "{\n\t"                                                                                     \
      ".reg .pred p;\n\t"                                                                         \
      "setp.ne.b32 p, %4, 0;\n\t"                                                                 \
      "tcgen05.mma.cta_group::2.kind::" KIND COLLECT " [%0], %1, %2, %3, p;\n\t"                  \
      "}"                                                                                         \
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)                        \
      : "memory")
// kFp8: e4m3 operands.  kind::f8f6f4 multiplies 32 elements of K per
// instruction, i.e. the same 32 bytes of every shared-memory row as kind::f16.
template <bool kFp8, CollectA kCollect = CollectA::kDiscard>
__device__ __forceinline__ void umma_ss_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                             uint32_t accumulate) {
  static_assert(!kFp8 || kCollect == CollectA::kDiscard, "two tiles at a time are bf16");
  if constexpr (kFp8) SMR_UMMA_PAIR("f8f6f4", "");
  else if constexpr (kCollect == CollectA::kFill) SMR_UMMA_PAIR("f16", ".collector::a::fill");
  else if constexpr (kCollect == CollectA::kLastUse) SMR_UMMA_PAIR("f16", ".collector::a::lastuse");
  else SMR_UMMA_PAIR("f16", "");
}
#undef SMR_UMMA_PAIR
// One arrival on the barrier at this offset in BOTH CTAs of the pair once all
// MMAs issued so far have completed.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
      ::"r"(smem_u32(bar)), "h"(mask) : "memory");
}

}  // namespace smr
