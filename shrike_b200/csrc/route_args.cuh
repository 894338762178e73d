// Arguments of the router kernels, shared with the layer kernel that routes its own rows.
#pragma once

#include "internal.h"

namespace shrike {

struct RouterArgs {
    const void* w;                 // fp32 rows, or packed affine rows
    const uint16_t* scales;        // affine only
    const uint16_t* biases;        // affine only
    uint32_t bits;                 // 0 = fp32
    const float* gate_row;         // shared expert scalar gate row or NULL
    const uint16_t* eff_scale;
    const uint16_t* logit_bias;
    const uint16_t* per_expert_scale;
    const void* hidden;
    uint32_t T, stride, dt, ne, d, top_k;
    uint32_t sigmoid_scores;
    float scaling;
    uint32_t round_f16;
    float* logits;
    uint32_t* ids;
    float* weights;
    float* gate_out;
    uint32_t tokens_per_block;
    // fused decode tail (route_fused_kernel only)
    const uint64_t* table;
    uint32_t pool_cells;
    const uint32_t* io_status;
    uint32_t with_shared, int4, group;
    uint32_t* slots;
    uint32_t* counts;
    Instance* inst;
    uint32_t* n_inst;
    uint32_t* sorted;
    uint16_t* xh;
    float* xsum;
    uint32_t* done_counter;
    uint32_t* pair_cell;
    uint32_t* status;
    uint32_t max_inst;
};

RouterArgs make_router_args(const shrike_moe* m, const shrike_router_operands& ops, const void* hidden, uint32_t T,
                            uint32_t stride, uint32_t* ids, float* weights, float* shared_gate);
// router_tile.cu: the logits (and gate values) of a call of many rows; whether it takes these operands
bool router_tiles_take(const RouterArgs& a);
cudaError_t launch_router_tiles(const shrike_moe* m, cudaStream_t st, const RouterArgs& a);

}  // namespace shrike
