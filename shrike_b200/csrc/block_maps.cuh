// Tensor maps of the packed expert blocks of a pool and of the shared expert's block, shared by the kernels that
// stream whole weight tiles (fused_layer.cu, expert_stream.cu). Entries 0..7 are the pool's chunks, entry 8 the
// shared expert's block.
#pragma once

#include <cuda.h>

#include "internal.h"

namespace shrike {

// The one-row kernel's.
struct BlockMaps {
    CUtensorMap w1[SHRIKE_MAX_POOL_CHUNKS + 1];   // gate + up rows: (group bytes, rows, groups, 2, cells)
    CUtensorMap m1[SHRIKE_MAX_POOL_CHUNKS + 1];   // their scales and biases: (8 rows' worth, rows / 8, scale|bias, 2, cells)
    CUtensorMap w2[SHRIKE_MAX_POOL_CHUNKS + 1];   // down rows: (group bytes, rows, groups, cells)
    CUtensorMap m2[SHRIKE_MAX_POOL_CHUNKS + 1];   // their scales and biases: (8 rows' worth, rows / 8, scale|bias, cells)
};
// The streaming kernel's: the same weights in 128-byte pieces of a row (128-byte swizzle), (128 bytes, rows[, 2], pieces, cells),
// and the same scales and biases.
struct PieceMaps {
    CUtensorMap l1[SHRIKE_MAX_POOL_CHUNKS + 1], m1[SHRIKE_MAX_POOL_CHUNKS + 1];
    CUtensorMap l2[SHRIKE_MAX_POOL_CHUNKS + 1], m2[SHRIKE_MAX_POOL_CHUNKS + 1];
};

// The maps of a call's pool and shared block, cached on the handle; NULL when the layout is not one that they can
// describe (fused_layer.cu). Either may be there without the other.
const BlockMaps* block_maps_for(const shrike_moe* m, const ExpertArgs& ea);
const PieceMaps* piece_maps_for(const shrike_moe* m, const ExpertArgs& ea);

// Tiled TMA loads (no multicast): the box lands densely, innermost dimension first.
__device__ __forceinline__ void tma_4d(uint32_t dst, const CUtensorMap* map, int32_t c0, int32_t c1, int32_t c2, int32_t c3,
                                       uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_5d(uint32_t dst, const CUtensorMap* map, int32_t c0, int32_t c1, int32_t c2, int32_t c3,
                                       int32_t c4, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(smem_u32(bar)) : "memory");
}

// Weights that a call reads once: the first lines that L2 gives up, so that the activations, the router's rows and the
// code stay in it while hundreds of megabytes of experts pass through.
__device__ __forceinline__ uint64_t evict_first_policy() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void tma_4d_once(uint32_t dst, const CUtensorMap* map, int32_t c0, int32_t c1, int32_t c2, int32_t c3,
                                            uint64_t* bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4, %5}], [%6], %7;"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar)), "l"(policy) : "memory");
}
__device__ __forceinline__ void tma_5d_once(uint32_t dst, const CUtensorMap* map, int32_t c0, int32_t c1, int32_t c2, int32_t c3,
                                            int32_t c4, uint64_t* bar, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4, %5, %6}], [%7], %8;"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(smem_u32(bar)), "l"(policy) : "memory");
}

}  // namespace shrike
