// Prefill path for ragged batches: rows are permuted by expert on the device
// (plan.cu), every expert's rows run through the expert-grouped GEMM (or, for
// shapes it does not take, the dequant-fused tiles in instances of 8), the
// down projection's epilogue multiplies each row by its route weight and adds
// it into one fp32 accumulator row per token (the weighted reduce of
// prefill_moe_reduce_token_major, prefill.metal:624-645, without the
// per-(row, rank) partial rows), and a last pass converts and does the two
// residual adds of RealForwardRunner.swift:4658-4665.
#include "internal.h"

namespace shrike {

// One thread per expert: ceil(count/8) instances each, in expert order.
__global__ void __launch_bounds__(256)
prefill_instances_kernel(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ counts,
                         const uint32_t* __restrict__ slot_of_expert, uint32_t ne, uint32_t T,
                         uint32_t with_shared, const uint32_t* __restrict__ sorted, Instance* __restrict__ inst,
                         uint32_t* __restrict__ n_inst) {
    __shared__ uint32_t warp_sums[8];
    const uint32_t e = threadIdx.x;
    uint32_t n = 0, slot = SHRIKE_SLOT_MISS, c = 0;
    if (e < ne && counts[e] > 0) {   // (of pairs with a cell)
        c = counts[e];
        slot = slot_of_expert[e];
        n = (c + 7) / 8;
    }
    // exclusive scan over 256 threads
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += v;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    uint32_t base = 0, total = 0;
    for (uint32_t w = 0; w < 8; ++w) {
        if (w < warp) base += warp_sums[w];
        total += warp_sums[w];
    }
    base += inc - n;
    for (uint32_t j = 0; j < n; ++j) {
        Instance in;
        in.kind = 0; in.slot = slot; in.first = offsets[e] + 8 * j; in.count = min(8u, c - 8 * j);
        for (uint32_t q = 0; q < 8; ++q) in.pair[q] = sorted[in.first + (q < in.count ? q : 0)];
        inst[base + j] = in;
    }
    const uint32_t n_shared = with_shared ? (T + 7) / 8 : 0;
    for (uint32_t j = threadIdx.x; j < n_shared; j += blockDim.x) {
        Instance in;
        in.kind = 1; in.slot = 0; in.first = 8 * j; in.count = min(8u, T - 8 * j);
        for (uint32_t q = 0; q < 8; ++q) in.pair[q] = 8 * j + (q < in.count ? q : 0);
        inst[total + j] = in;
    }
    if (threadIdx.x == 0) *n_inst = total + n_shared;
}

// x -> fp16 operand layout and per-group sums, all rows; the pairs in expert-sorted order; given `xs`, the rows in that order too, which
// the grouped GEMM copies its tiles from. (Bound by the sorted rows' bytes, top_k times x's: as a kernel of its own that read
// them back, the gather took 28 us of a 4096-row call beside 11 here.)
__global__ void __launch_bounds__(256)
prefill_xprep_kernel(const void* __restrict__ x, uint32_t T, uint32_t d, uint32_t group, uint32_t act_dtype,
                     uint32_t int4, uint16_t* __restrict__ xh, float* __restrict__ xsum, uint32_t* status,
                     const uint32_t* __restrict__ row_map, const uint32_t* __restrict__ n_rows_dev,
                     const uint32_t* __restrict__ ids, const uint32_t* __restrict__ rank_of_pair,
                     const uint32_t* __restrict__ block_base, uint32_t ne, uint32_t top_k, uint32_t* __restrict__ sorted,
                     uint16_t* __restrict__ xs, float* __restrict__ zero) {
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t items = T * (d / 8);
    const size_t row_bytes = (size_t)d * (act_dtype == SHRIKE_DTYPE_FP32 ? 4 : 2);
    const uint32_t n_rows = n_rows_dev ? *n_rows_dev : T;
    for (uint32_t i0 = blockIdx.x * blockDim.x; i0 < items; i0 += gridDim.x * blockDim.x) {
        const uint32_t i = i0 + threadIdx.x, row = i / (d / 8), col = (i - row * (d / 8)) * 8;
        const bool there = i < items;
        // the pairs' places: the first of their expert's rows in this block of rows, and those before them in the block (asked for
        // ahead of the row itself: two trips to L2)
        uint32_t pos[SHRIKE_MAX_TOP_K];
#pragma unroll
        for (uint32_t r = 0; r < SHRIKE_MAX_TOP_K; ++r) pos[r] = 0xffffffffu;
        if (there && row < n_rows && (xs || col == 0)) {
            uint32_t rank[SHRIKE_MAX_TOP_K], e[SHRIKE_MAX_TOP_K];
#pragma unroll
            for (uint32_t r = 0; r < SHRIKE_MAX_TOP_K; ++r) {
                rank[r] = r < top_k ? rank_of_pair[row * top_k + r] : 0xffffffffu;
                e[r] = r < top_k ? ids[row * top_k + r] : 0u;
            }
#pragma unroll
            for (uint32_t r = 0; r < SHRIKE_MAX_TOP_K; ++r)
                if (rank[r] != 0xffffffffu) pos[r] = block_base[(size_t)(row / kGroupTokens) * ne + e[r]] + rank[r];
        }
        xprep_item(x, row_bytes, d, group, act_dtype, int4 != 0, i, there, xh, xsum, status, row_map, n_rows);
        if (there) {   // the rows that the down projection adds into
            float* const z = zero + (size_t)i * 8;
            if (((uintptr_t)zero & 15u) == 0) {
                ((float4*)z)[0] = ((float4*)z)[1] = make_float4(0.f, 0.f, 0.f, 0.f);
            } else {   // (the caller's own rows)
#pragma unroll
                for (int k = 0; k < 8; ++k) z[k] = 0.f;
            }
        }
        if (!there || row >= n_rows) continue;
        if (col == 0) {
#pragma unroll
            for (uint32_t r = 0; r < SHRIKE_MAX_TOP_K; ++r)
                if (pos[r] != 0xffffffffu) sorted[pos[r]] = row * top_k + r;
        }
        if (!xs) continue;
        const uint4 v = *(const uint4*)(xh + (size_t)i * 8);   // this thread's own
#pragma unroll
        for (uint32_t r = 0; r < SHRIKE_MAX_TOP_K; ++r)
            if (pos[r] != 0xffffffffu) *(uint4*)(xs + (size_t)pos[r] * d + col) = v;
    }
}

// y[t] = the accumulated row (shared term and weighted expert rows, fp32); hidden += y.
__global__ void __launch_bounds__(256)
prefill_combine_kernel(const float* __restrict__ yacc, uint32_t n, uint32_t act_dtype, uint32_t y_dtype,
                       void* __restrict__ y, void* __restrict__ hidden) {
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float acc = yacc[i];
    store_act(y, i, y_dtype, acc);
    if (hidden) {
        const float h = load_act(hidden, i, act_dtype) + round_act(y_dtype, acc);
        store_act(hidden, i, act_dtype, h);
    }
}

cudaError_t launch_prefill_plan(const shrike_moe* m, cudaStream_t st, const uint32_t* ids,
                                const uint32_t* slots, const void* x, uint32_t T, bool with_shared,
                                uint32_t pool_cells, bool warp_mma_instances, const uint32_t* io_status,
                                const uint32_t* row_map, const uint32_t* n_rows, float* accumulator) {
    const shrike_moe_config& c = m->cfg;
    const Workspace& ws = m->ws;
    cudaError_t e = launch_group_plan(m, st, ids, T, slots, io_status, with_shared, pool_cells);
    if (e != cudaSuccess) return e;
    const uint32_t items = T * (c.d / 8);
    e = launch_after(m, st, prefill_xprep_kernel, dim3(min(2048u, (items + 255) / 256)), 256, 0, x, T, c.d, c.group_size, c.act_dtype,
                     c.weight_bits == 4 ? 1u : 0u, ws.xh, ws.xsum, ws.status, row_map, n_rows, ids, ws.rank_of_pair, ws.block_hist,
                     c.num_experts, c.top_k, ws.sorted, warp_mma_instances ? nullptr : ws.xs,
                     accumulator ? accumulator : ws.yacc);   // the rows the down epilogue adds into: the workspace's, or the caller's fp32 output itself
    if (e == cudaSuccess && warp_mma_instances) {   // the tensor-core path has its 256-row instances from the plan
        prefill_instances_kernel<<<1, 256, 0, st>>>(ws.expert_offsets, ws.expert_counts, ws.slot_of_expert,
                                                    c.num_experts, T, with_shared ? 1u : 0u, ws.sorted,
                                                    ws.inst, ws.n_inst);
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t launch_prefill_combine(const shrike_moe* m, cudaStream_t st, uint32_t T, void* y, void* hidden) {
    const shrike_moe_config& c = m->cfg;
    const uint32_t n = T * c.d;
    return launch_after(m, st, prefill_combine_kernel, dim3((n + 255) / 256), 256, 0, m->ws.yacc, n, c.act_dtype, c.y_dtype, y, hidden);
}

}  // namespace shrike
