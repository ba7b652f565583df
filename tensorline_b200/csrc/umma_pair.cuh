// Device helpers of the kernels in which two thread blocks of a cluster work on one tile (tcgen05 cta_group::2).
//
// MMAs, commits and copies are issued by a whole warp, the instruction itself predicated on one elected lane (`one`): their operands are
// then uniform registers from the start.  Issued from a branch that only one thread takes, every MMA took that thread 61 cycles; so 27.
// Barriers are waited for and arrived at with the default order (this block's): a release at the cluster's scope waits for memory,
// more than 1,000 cycles a time, and what the pair hands over (tensor memory, shared memory read by an MMA) is ordered by tcgen05's own fences and commits.
#pragma once
#include "umma.cuh"

namespace {

__device__ __forceinline__ uint32_t pair_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
// the shared::cluster address of the same shared-memory location in block `rank` of this cluster
__device__ __forceinline__ uint32_t pair_peer(uint32_t local, uint32_t rank) {
    uint32_t out;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(local), "r"(rank));
    return out;
}
__device__ __forceinline__ uint32_t pair_elect() {
    uint32_t one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
    return one;
}
__device__ __forceinline__ void pair_arrive(uint32_t cluster_address) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_address) : "memory");
}
// a box by TMA (no multicast) into this block's shared memory; its bytes count on `bar`, which may be the peer's barrier
__device__ __forceinline__ void pair_load(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, uint32_t one) {
    asm volatile("{\n\t.reg .pred q;\n\t"
                 "setp.ne.b32 q, %5, 0;\n\t"
                 "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(one) : "memory");
}
__device__ __forceinline__ void pair_expect(uint64_t* bar, uint32_t bytes, uint32_t one) {
    asm volatile("{\n\t.reg .pred q;\n\t"
                 "setp.ne.b32 q, %2, 0;\n\t"
                 "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}"
                 ::"r"(smem_addr(bar)), "r"(bytes), "r"(one) : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, uint32_t one) {
    asm volatile("{\n\t.reg .pred p, q;\n\t"
                 "setp.ne.b32 p, %4, 0;\n\t"
                 "setp.ne.b32 q, %5, 0;\n\t"
                 "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(one) : "memory");
}
// arrive on the barrier at this address in both blocks when the MMAs issued so far are done
__device__ __forceinline__ void pair_commit(uint64_t* bar, uint32_t one) {
    const uint16_t mask = 3;
    asm volatile("{\n\t.reg .pred q;\n\t"
                 "setp.ne.b32 q, %2, 0;\n\t"
                 "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
                 ::"r"(smem_addr(bar)), "h"(mask), "r"(one) : "memory");
}
__device__ __forceinline__ void pair_cluster_sync() { asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory"); }
// 512 columns of tensor memory for the pair: a warp of each block
__device__ __forceinline__ void pair_tmem_alloc(uint32_t* slot) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_tmem_free(uint32_t base) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(512u) : "memory");
}

// rows of K bfloat16 values, boxes of 64 values by `box_rows` rows with the 128-byte swizzle
inline int pair_map(CUtensorMap* map, const void* base, long long rows, int K, int box_rows) {
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows}, elem[2] = {1, 1};
    const CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 101;
}

}  // namespace
