// Device-side routing plans: which rows go to which expert block.
//
// Decode (few rows): the (row, rank) pairs are ordered by pool slot with a
// rank sort inside one block, cut into instances of at most 8 rows that share
// a block, and the activation rows are copied to the fp16 operand layout.
//
// Prefill: PrefillMoEGrouping.groupTokenExpertPairs
// (PrefillMoEGrouping.swift:269-370) as a counting sort by expert id that
// keeps (token, rank) order inside an expert, in place of the host sort the
// reference runs between two GPU syncs (RealForwardRunner.swift:4305): three
// launches for the grouping as a call of its own, one for a prefill call,
// whose rows are placed where they are converted (prefill.cu).
#include "plan.cuh"

namespace shrike {

constexpr uint32_t kPlanThreads = 512;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t n = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += n;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    uint32_t base = 0, tot = 0;
    const uint32_t nw = blockDim.x >> 5;
    for (uint32_t w = 0; w < nw; ++w) {
        const uint32_t s = warp_sums[w];
        if (w < warp) base += s;
        tot += s;
    }
    __syncthreads();
    total = tot;
    return base + inc - v;
}

__global__ void __launch_bounds__(kPlanThreads)
decode_plan_kernel(const uint32_t* __restrict__ slots, uint32_t T, uint32_t top_k,
                   const uint32_t* __restrict__ io_status, uint32_t with_shared, uint32_t pool_cells,
                   Instance* __restrict__ inst, uint32_t* __restrict__ n_inst,
                   uint32_t* __restrict__ sorted, const void* __restrict__ x, uint32_t act_dtype,
                   uint32_t d, uint32_t int4, uint32_t group, uint16_t* __restrict__ xh,
                   float* __restrict__ xsum, uint32_t* status, uint32_t max_inst, uint32_t* __restrict__ pair_cell) {
    __shared__ PlanSmem sm;
    const uint32_t tid = threadIdx.x;
    const uint32_t n_pairs = T * top_k;

    // moe_io_ready (moe.metal:36-39): a pending or failed batch leaves only the
    // shared term.
    bool ready = true;
    if (io_status) {
        const uint32_t s = *io_status;
        ready = s == 1u || s == 3u;
    }
    for (uint32_t p = tid; p < n_pairs; p += kPlanThreads) {
        uint32_t s = ready ? slots[p] : SHRIKE_SLOT_MISS;
        if (s != SHRIKE_SLOT_MISS && s >= pool_cells) {
            report_status(status, kStatusBadIndex);
            s = SHRIKE_SLOT_MISS;
        }
        sm.key[p] = s;
        pair_cell[p] = s;
    }
    __syncthreads();
    plan_body(sm, n_pairs, T, with_shared, inst, n_inst, sorted, max_inst, status);

    // fp16 operand copy of the activation rows and their per-group sums
    const uint32_t items = T * (d / 8);
    const size_t row_bytes = (size_t)d * (act_dtype == SHRIKE_DTYPE_FP32 ? 4 : 2);
    for (uint32_t i0 = 0; i0 < items; i0 += kPlanThreads)
        xprep_item(x, row_bytes, d, group, act_dtype, int4 != 0, i0 + tid, i0 + tid < items, xh, xsum, status);
}

cudaError_t launch_decode_plan(const shrike_moe* m, cudaStream_t st, const uint32_t* slots,
                               const void* x, uint32_t T, const uint32_t* io_status, bool with_shared,
                               uint32_t pool_cells) {
    decode_plan_kernel<<<1, kPlanThreads, 0, st>>>(
        slots, T, m->cfg.top_k, io_status, with_shared ? 1u : 0u, pool_cells,
        m->ws.inst, m->ws.n_inst, m->ws.sorted, x, m->cfg.act_dtype, m->cfg.d,
        m->cfg.weight_bits == 4 ? 1u : 0u, m->cfg.group_size, m->ws.xh, m->ws.xsum, m->ws.status, max_instances(m->cfg, T),
        m->ws.pair_cell);
    return cudaGetLastError();
}

// ---- prefill grouping -------------------------------------------------------

using GroupBits = uint32_t[SHRIKE_MAX_EXPERTS][kGroupTokens / 32];

// Row tl of the block names expert e. False: there is no such expert.
__device__ __forceinline__ bool name_expert(GroupBits& named, uint32_t e, uint32_t ne, uint32_t tl, uint32_t* status) {
    if (e >= ne) {
        // out of range: the pair is dropped and reported (0xffffffff is the expert-parallel layer's
        // "this pick lives on another rank" and is dropped silently)
        if (e != 0xffffffffu) report_status(status, kStatusBadIndex);
        return false;
    }
    // a row that names one expert twice (no top-k router does) is counted once and reported
    const uint32_t bit = 1u << (tl & 31);
    if (atomicOr(&named[e][tl >> 5], bit) & bit) report_status(status, kStatusBadIndex);
    return true;
}

// The block's rows of each expert (block_hist: [block][expert]).
__device__ __forceinline__ void count_rows(const GroupBits& bits, uint32_t ne, uint32_t* block_hist) {
    for (uint32_t e = threadIdx.x; e < ne; e += blockDim.x) {
        uint32_t c = 0;
#pragma unroll
        for (uint32_t w = 0; w < kGroupTokens / 32; ++w) c += __popc(bits[e][w]);
        block_hist[(size_t)blockIdx.x * ne + e] = c;
    }
}

// Step 1: per block, a bitmap of the rows that chose each expert; writes the per-(block, expert) counts.
__global__ void __launch_bounds__(256)
group_hist_kernel(const uint32_t* __restrict__ ids, uint32_t T, uint32_t top_k, uint32_t ne,
                  uint32_t* __restrict__ block_hist, uint32_t* status) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ GroupBits bits;
    const uint32_t t0 = blockIdx.x * kGroupTokens;
    for (uint32_t i = threadIdx.x; i < SHRIKE_MAX_EXPERTS * (kGroupTokens / 32); i += blockDim.x)
        (&bits[0][0])[i] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kGroupTokens * top_k; i += blockDim.x) {
        const uint32_t tl = i / top_k, t = t0 + tl;
        if (t < T) name_expert(bits, ids[(size_t)t * top_k + (i - tl * top_k)], ne, tl, status);
    }
    __syncthreads();
    count_rows(bits, ne, block_hist);
}

// Rows before row tl of the block that chose expert e.
__device__ __forceinline__ uint32_t rows_before(const GroupBits& bits, uint32_t e, uint32_t tl) {
    uint32_t before = 0;
    const uint32_t word = tl >> 5;
    for (uint32_t w = 0; w < word; ++w) before += __popc(bits[e][w]);
    return before + __popc(bits[e][word] & ((1u << (tl & 31)) - 1u));
}

// Step 2 (one block): per-expert totals, exclusive scan over experts, and the
// running base of every (block, expert) cell.
__device__ __forceinline__ void group_scan(uint32_t* warp_sums, uint32_t* block_hist, uint32_t n_blocks, uint32_t ne,
                                           uint32_t* __restrict__ offsets, uint32_t* __restrict__ counts, uint32_t& total, uint32_t& base) {
    const uint32_t e = threadIdx.x;
    constexpr uint32_t kKept = 8;   // blocks' counts that a second look does not ask L2 for again
    uint32_t kept[kKept];
    total = 0;
#pragma unroll
    for (uint32_t b = 0; b < kKept; ++b) kept[b] = b < n_blocks && e < ne ? __ldcg(block_hist + (size_t)b * ne + e) : 0u;
#pragma unroll
    for (uint32_t b = 0; b < kKept; ++b) total += kept[b];
    if (e < ne) {
#pragma unroll 8
        for (uint32_t b = kKept; b < n_blocks; ++b) total += __ldcg(block_hist + (size_t)b * ne + e);
    }
    uint32_t all;
    base = block_exclusive_scan(total, warp_sums, all);
    if (e < ne) {
        counts[e] = total;
        offsets[e] = total ? base : 0xffffffffu;
        uint32_t run = base;
#pragma unroll
        for (uint32_t b = 0; b < kKept; ++b) {
            if (b < n_blocks) block_hist[(size_t)b * ne + e] = run;
            run += kept[b];
        }
#pragma unroll 8
        for (uint32_t b = kKept; b < n_blocks; ++b) {
            const uint32_t c = __ldcg(block_hist + (size_t)b * ne + e);
            block_hist[(size_t)b * ne + e] = run;
            run += c;
        }
    }
}
__global__ void __launch_bounds__(256)
group_scan_kernel(uint32_t* block_hist, uint32_t n_blocks, uint32_t ne,
                  uint32_t* __restrict__ offsets, uint32_t* __restrict__ counts) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ uint32_t warp_sums[8];
    uint32_t total, base;
    group_scan(warp_sums, block_hist, n_blocks, ne, offsets, counts, total, base);
}

// Step 3: place every pair at base(block, expert) + number of earlier rows of
// the block that chose the same expert.
__global__ void __launch_bounds__(256)
group_place_kernel(const uint32_t* __restrict__ ids, const float* __restrict__ weights, uint32_t T,
                   uint32_t top_k, uint32_t ne, const uint32_t* __restrict__ block_base,
                   uint32_t* __restrict__ sorted_pairs) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ uint32_t bits[SHRIKE_MAX_EXPERTS][kGroupTokens / 32];
    const uint32_t t0 = blockIdx.x * kGroupTokens;
    for (uint32_t i = threadIdx.x; i < SHRIKE_MAX_EXPERTS * (kGroupTokens / 32); i += blockDim.x)
        (&bits[0][0])[i] = 0;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kGroupTokens * top_k; i += blockDim.x) {
        const uint32_t tl = i / top_k, t = t0 + tl;
        if (t < T) {
            const uint32_t e = ids[(size_t)t * top_k + (i - tl * top_k)];
            if (e < ne) atomicOr(&bits[e][tl >> 5], 1u << (tl & 31));
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kGroupTokens * top_k; i += blockDim.x) {
        const uint32_t tl = i / top_k, t = t0 + tl, r = i - tl * top_k;
        if (t >= T) continue;
        const uint32_t e = ids[(size_t)t * top_k + r];
        if (e >= ne) continue;
        const uint32_t pos = block_base[(size_t)blockIdx.x * ne + e] + rows_before(bits, e, tl);
        uint4 p;
        p.x = t; p.y = e; p.z = r;
        // weight bits as the reference stores them: fp16 in the low half
        p.w = weights ? (uint32_t)__half_as_ushort(__float2half_rn(weights[(size_t)t * top_k + r])) : 0u;
        ((uint4*)sorted_pairs)[pos] = p;
    }
}

// The list of instances: all full ones (256 rows; the shared expert's first), then every expert's rest, most rows first. A tile of
// 256 rows takes twice the time of one of 16, and a list that ends on long ones leaves SMs idle. All tiles of more than 128 rows come before the
// others, so a block changes the layout of its shared memory once at most. Thread e has expert e's `c` rows, which begin at `first`
// in the sorted order; n_inst[0] = instances, [1], [2]: tiles handed out in phase 0, 1.
__device__ __forceinline__ void chunk_instances(uint32_t* warp_sums, uint32_t (&key)[256], uint32_t c, uint32_t first, uint32_t slot, uint32_t T,
                                                uint32_t with_shared, ChunkInstance* __restrict__ inst, uint32_t* __restrict__ n_inst) {
    const uint32_t e = threadIdx.x, n = c / kChunkRows, rest = c % kChunkRows, mine = rest << 8 | (255u - e);
    const uint32_t shared_rest = with_shared ? T % kChunkRows : 0u, n_shared = with_shared ? T / kChunkRows : 0u;
    key[e] = mine;
    uint32_t total;
    uint32_t base = block_exclusive_scan(n, warp_sums, total);
    const uint32_t before_shared = (uint32_t)__syncthreads_count(rest > shared_rest);   // rests that come before the shared expert's
    const uint32_t n_rest = (uint32_t)__syncthreads_count(rest != 0) + (shared_rest != 0);
    base += n_shared;
    total += n_shared;
    auto put = [&](uint32_t at, uint32_t kind, uint32_t cell, uint32_t from, uint32_t count) {
        *(uint4*)(inst + at) = make_uint4(kind, cell, from, count);
    };
    for (uint32_t j = 0; j < n; ++j) put(base + j, 0, slot, first + kChunkRows * j, kChunkRows);
    if (rest) {
        uint32_t rank = rest <= shared_rest ? 1u : 0u;
        for (uint32_t j = 0; j < 256; j += 4) {
            const uint4 v = *(const uint4*)&key[j];
            rank += (v.x > mine) + (v.y > mine) + (v.z > mine) + (v.w > mine);
        }
        put(total + rank, 0, slot, first + kChunkRows * n, rest);
    }
    for (uint32_t j = e; j < n_shared; j += blockDim.x) put(j, 1, 0, kChunkRows * j, kChunkRows);
    if (e == 0) {
        if (shared_rest) put(total + before_shared, 1, 0, kChunkRows * n_shared, shared_rest);
        n_inst[0] = total + n_rest;
        n_inst[1] = n_inst[2] = 0;   // tiles handed out, per phase
    }
}

// The prefill plan in one launch: step 1, and every pair's rows before it in its block of rows; the block that finishes last
// takes step 2 and lists the instances. Only pairs with a cell are counted and placed, so that every place an instance covers is
// written, whatever the slots say: an expert that becomes resident while they are looked up has pairs of both kinds. The pairs' places follow from the two where the rows are converted. Bound by a chain of trips
// to L2 (ids, counts, ticket, counts again, list). Counting, scan, places and list as launches of their own, and this: a call of 70 rows
// 155.9 -> 150.1 us, 333 rows 181.5 -> 177.6, 1134 rows 247.9 -> 243.2.
__global__ void __launch_bounds__(256)
group_plan_kernel(const uint32_t* __restrict__ ids, uint32_t T, uint32_t top_k, uint32_t ne, uint32_t* block_hist, uint32_t* status,
                  const uint32_t* __restrict__ slots, const uint32_t* __restrict__ io_status, uint32_t* slot_of_expert,
                  uint32_t* __restrict__ rank_of_pair, uint32_t* __restrict__ offsets, uint32_t* __restrict__ counts, uint32_t* ticket,
                  uint32_t with_shared, uint32_t pool_cells, ChunkInstance* __restrict__ inst, uint32_t* __restrict__ n_inst) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ GroupBits named, bits;   // the rows that name each expert; those that have a cell for it
    __shared__ uint32_t warp_sums[8], s_last;
    __shared__ __align__(16) uint32_t key[256];
    // a thread's pairs, asked for at once and kept
    constexpr uint32_t N = kGroupTokens * SHRIKE_MAX_TOP_K / 256;
    const uint32_t t0 = blockIdx.x * kGroupTokens, n = min(T - t0, kGroupTokens) * top_k, io = io_status ? *io_status : 1u;
    const bool ready = io == 1u || io == 3u;
    uint32_t e[N], cell[N];
#pragma unroll
    for (uint32_t j = 0; j < N; ++j) {
        const uint32_t i = j * 256 + threadIdx.x;
        e[j] = i < n ? ids[(size_t)t0 * top_k + i] : 0xffffffffu;
        cell[j] = i < n ? slots[(size_t)t0 * top_k + i] : SHRIKE_SLOT_MISS;
    }
#pragma unroll
    for (uint32_t j = 0; j < sizeof(GroupBits) / 4 / 256; ++j) (&named[0][0])[j * 256 + threadIdx.x] = (&bits[0][0])[j * 256 + threadIdx.x] = 0;
    __syncthreads();
#pragma unroll
    for (uint32_t j = 0; j < N; ++j) {
        const uint32_t tl = (j * 256 + threadIdx.x) / top_k;
        if (!name_expert(named, e[j], ne, tl, status) || !ready) cell[j] = SHRIKE_SLOT_MISS;
        if (cell[j] != SHRIKE_SLOT_MISS && cell[j] >= pool_cells) {
            report_status(status, kStatusBadIndex);
            cell[j] = SHRIKE_SLOT_MISS;
        }
        if (cell[j] != SHRIKE_SLOT_MISS) {
            atomicOr(&bits[e[j]][tl >> 5], 1u << (tl & 31));
            slot_of_expert[e[j]] = cell[j];   // (of an expert with two cells either)
        }
    }
    __syncthreads();
    count_rows(bits, ne, block_hist);
#pragma unroll
    for (uint32_t j = 0; j < N; ++j) {
        const uint32_t i = j * 256 + threadIdx.x;
        if (i < n) rank_of_pair[(size_t)t0 * top_k + i] = cell[j] == SHRIKE_SLOT_MISS ? 0xffffffffu : rows_before(bits, e[j], i / top_k);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1 ? 1u : 0u;
        if (s_last) *ticket = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    uint32_t total, base;
    group_scan(warp_sums, block_hist, gridDim.x, ne, offsets, counts, total, base);
    const uint32_t slot = threadIdx.x < ne && total ? __ldcg(slot_of_expert + threadIdx.x) : SHRIKE_SLOT_MISS;
    chunk_instances(warp_sums, key, total, base, slot, T, with_shared, inst, n_inst);
}

cudaError_t launch_group_pairs(const shrike_moe* m, cudaStream_t st, const uint32_t* ids,
                               const float* weights, uint32_t T, uint32_t* sorted_pairs,
                               uint32_t* offsets, uint32_t* counts) {
    const uint32_t nb = (T + kGroupTokens - 1) / kGroupTokens;
    const uint32_t ne = m->cfg.num_experts, k = m->cfg.top_k;
    if (nb == 0) {
        cudaError_t e = cudaMemsetAsync(counts, 0, ne * 4, st);
        if (e != cudaSuccess) return e;
        return cudaMemsetAsync(offsets, 0xff, ne * 4, st);
    }
    cudaError_t e = launch_after(m, st, group_hist_kernel, dim3(nb), 256, 0, ids, T, k, ne, m->ws.block_hist, m->ws.status);
    if (e != cudaSuccess) return e;
    e = launch_after(m, st, group_scan_kernel, dim3(1), 256, 0, m->ws.block_hist, nb, ne, offsets, counts);
    if (e != cudaSuccess) return e;
    return launch_after(m, st, group_place_kernel, dim3(nb), 256, 0, ids, weights, T, k, ne, m->ws.block_hist, sorted_pairs);
}

cudaError_t launch_group_plan(const shrike_moe* m, cudaStream_t st, const uint32_t* ids, uint32_t T, const uint32_t* slots,
                              const uint32_t* io_status, bool with_shared, uint32_t pool_cells) {
    const Workspace& ws = m->ws;
    return launch_after(m, st, group_plan_kernel, dim3((T + kGroupTokens - 1) / kGroupTokens), 256, 0, ids, T, m->cfg.top_k, m->cfg.num_experts,
                        ws.block_hist, ws.status, slots, io_status, ws.slot_of_expert, ws.rank_of_pair, ws.expert_offsets, ws.expert_counts,
                        ws.plan_ticket, with_shared ? 1u : 0u, pool_cells, (ChunkInstance*)ws.chunk_inst, ws.n_chunk_inst);
}

}  // namespace shrike
