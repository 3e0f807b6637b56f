// What products by pairs of blocks use: ranks and addresses in a cluster, its barrier, loads and arrivals on the
// other block's mbarriers.
#pragma once
#include "tcgen05_gemm.cuh"

__device__ __forceinline__ unsigned tp_cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
// The address, in the cluster's shared window, of `addr` in the block of rank `rank`.
__device__ __forceinline__ unsigned tp_map_to_rank(unsigned addr, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void tp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// A tiled load into this block's shared memory whose bytes are counted on an mbarrier
// that may live in the other block of the pair (`bar`: an address in the cluster's window).
__device__ __forceinline__ void tp_tma_load_2d(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
// One arrival, when the products issued so far have completed, on the mbarrier at this
// offset in the blocks of the cluster that `mask` names (a pair: both).
__device__ __forceinline__ void tp_commit_mask(unsigned bar, unsigned short mask) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
                 ::"r"(bar), "h"(mask) : "memory");
}
__device__ __forceinline__ void tp_arrive_remote(unsigned bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
