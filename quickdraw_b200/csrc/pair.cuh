// Pairs of blocks on two SMs that share tcgen05 products (cta_group::2): places in the first block, copies that count there, commits to both.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace qd {

QD_DEVINL uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
QD_DEVINL uint32_t of_first_block(const void* p) {                    // the same place in the first block of the pair
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
    return r;
}
QD_DEVINL void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
QD_DEVINL void pair_tma_tile(void* dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_u32(dst)), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
QD_DEVINL void pair_commit(uint64_t* bar) {                           // arrives at this place in both blocks
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
QD_DEVINL void pair_commit_here(uint64_t* bar) {                      // arrives in this block alone
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
QD_DEVINL void arrive_at(uint32_t bar) {                              // `bar` as of of_first_block
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// The end of a loading warp: the last `issued` copies (of a ring of barriers on which the MMAs release stages) have been used.  A wait
// that runs out ends it as well: by then 0.2 s have passed since the last copy was asked for.
QD_DEVINL void pair_loads_taken(uint64_t* empty, int ring, int issued, unsigned int* status) {
    for (int i = issued > ring ? issued - ring : 0; i < issued; ++i)
        if (!__all_sync(0xffffffffu, mbar_wait(empty + i % ring, (i / ring) & 1, status))) return;
}
QD_DEVINL void pair_tmem_alloc(uint32_t* slot, uint32_t cols) {       // a warp of each block
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
QD_DEVINL void pair_tmem_dealloc(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}

}  // namespace qd
