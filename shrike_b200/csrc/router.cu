// Router: logits, top-k selection with renormalisation, residency lookup.
//
//   router_gemv_body            moe.metal:324-364   (affine rows)
//   router_topk_select_body     moe.metal:419-491
//   prefill_router_tiled_body   prefill.metal:446-563 (same arithmetic per row)
//   moe_classify_residency_body moe.metal:121-151
//
// Selection must agree with the CPU restatement bit for bit, so the logits are
// summed in one fixed order: a warp owns an expert row, lane l accumulates its
// elements sequentially with fused multiply-adds, and the 32 lane sums are
// combined by a butterfly (xor 16, 8, 4, 2, 1). fp32 rows: lane l takes the
// float4 chunks l, l+32, ... ; affine rows: lane l takes elements 64g+2l,
// 64g+2l+1 of every group g, as the shader does. exp() is a fixed sequence of
// fp32 operations (exp_det) instead of the library routine for the same reason.
#include "plan.cuh"
#include "route_args.cuh"
#include "router_math.cuh"
#include "select.cuh"

namespace shrike {

constexpr int kRouterWarps = 8;       // expert rows per block (router_gemv_r4 has four); the block that finishes last
                                      // selects with as many warps

// Logits (and the shared expert's scalar gate as row `ne`) of this warp's row
// for the block's tokens. `pre` runs between the weight-row prefetch and the
// first read of the activations.
template <int N, bool PRED, typename Pre>
__device__ __forceinline__ void logits_rows(const RouterArgs& a, Pre pre) {
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t e = blockIdx.x * kRouterWarps + warp;
    const bool is_gate = a.gate_row != nullptr && e == a.ne;
    const bool active = e < a.ne || is_gate;
    const bool f32row = a.bits == 0 || is_gate;
    const uint32_t chunks = a.d / 4, groups = a.d / 64;
    float4 wr[N];
    if (active && f32row)
        load_row_f32<N, PRED>(is_gate ? a.gate_row : (const float*)a.w + (size_t)e * a.d, chunks, lane, wr);
    pre();
    if (!active) return;
    const uint32_t t0 = blockIdx.y * a.tokens_per_block;
    const uint32_t t1 = min(a.T, t0 + a.tokens_per_block);
    const size_t esz = a.dt == SHRIKE_DTYPE_FP32 ? 4 : 2;
    for (uint32_t tk = t0; tk < t1; ++tk) {
        const void* xrow = (const uint8_t*)a.hidden + (size_t)tk * a.stride * esz;
        float acc;
        if (f32row) {
            acc = lane_dot_f32<N, PRED>(wr, chunks, lane, xrow, a.dt, is_gate ? nullptr : a.eff_scale);
        } else {
            const uint8_t* const row = (const uint8_t*)a.w + (size_t)e * (a.d * a.bits / 8);
            const uint16_t *const s_row = a.scales + (size_t)e * groups, *const b_row = a.biases + (size_t)e * groups;
            if (a.dt == SHRIKE_DTYPE_FP32) acc = lane_dot_affine_f32(row, s_row, b_row, a.bits, groups, lane, (const float*)xrow, a.eff_scale);
            else acc = lane_dot_affine(row, s_row, b_row, a.bits, groups, lane, xrow, a.dt, a.eff_scale);
        }
        acc = butterfly_sum(acc);
        if (lane == 0) {
            if (is_gate) a.gate_out[tk] = sigmoid_det(acc);
            else a.logits[(size_t)tk * a.ne + e] = acc;
        }
    }
}

// The common hidden sizes get straight-line code without bounds checks.
template <typename Pre>
__device__ __forceinline__ void logits_body(const RouterArgs& a, Pre pre) {
    if (a.d == 2048) logits_rows<16, false>(a, pre);
    else if (a.d == 2304) logits_rows<18, false>(a, pre);
    else logits_rows<kRouterMaxChunks, true>(a, pre);
}

// grid (ceil((ne + has_gate)/4), token blocks)
__global__ void __launch_bounds__(kRouterWarps * 32) router_logits_kernel(const RouterArgs a) {
    pdl_wait();
    pdl_launch_dependents();
    logits_body(a, [] {});
}

__global__ void __launch_bounds__(128) router_select_kernel(const RouterArgs a) {
    __shared__ RowScratch rs[4];
    pdl_wait();
    pdl_launch_dependents();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t row = blockIdx.x * 4 + warp;
    if (row >= a.T) return;
    uint32_t id;
    float w;
    select_row_ranked<false>(a.logits + (size_t)row * a.ne, a, lane, rs[warp], id, w);
    if (lane < a.top_k) {
        a.ids[(size_t)row * a.top_k + lane] = id;
        a.weights[(size_t)row * a.top_k + lane] = w;
    }
}

// Decode (T <= 64) in one launch: logits by all blocks; the block that
// finishes last then selects, looks the experts up in the residency table and
// builds the work lists -- no wait on another block anywhere. Every block also
// converts its slice of the activation rows to the fp16 operand layout.
// grid (ceil((ne + has_gate)/4), 1..4 token groups).
__global__ void __launch_bounds__(kRouterWarps * 32) route_fused_kernel(const RouterArgs a) {
    __shared__ PlanSmem sm;
    __shared__ uint32_t ids_sm[kPlanMaxPairs];
    __shared__ SelectSmem sel;
    __shared__ uint32_t s_last, s_miss;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // the weight rows do not depend on the previous kernel: fetch them first
    logits_body(a, [&] {
        pdl_wait();
        pdl_launch_dependents();
    });

    // every block converts its share of the activation rows (blocks of 8 elements)
    {
        const uint32_t items = a.T * (a.d / 8);
        const size_t esz = a.dt == SHRIKE_DTYPE_FP32 ? 4 : 2;
        const uint32_t n_blocks = gridDim.x * gridDim.y, block = blockIdx.y * gridDim.x + blockIdx.x;
        for (uint32_t i0 = block * blockDim.x; i0 < items; i0 += n_blocks * blockDim.x)
            xprep_item(a.hidden, (size_t)a.stride * esz, a.d, a.group, a.dt, a.int4 != 0, i0 + tid, i0 + tid < items,
                       a.xh, a.xsum, a.status);
    }

    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const uint32_t ticket = atomicAdd(a.done_counter, 1u);
        s_last = ticket == gridDim.x * gridDim.y - 1 ? 1u : 0u;
        if (s_last) *a.done_counter = 0;
        s_miss = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();

    if (a.T == 1) {
        // one row: the whole block ranks it (no serial rounds)
        uint32_t id;
        float w;
        select_row_block(a.logits, a, sel, id, w);
        if (warp == 0 && lane < a.top_k) {
            a.ids[lane] = id;
            a.weights[lane] = w;
            ids_sm[lane] = id;
        }
    } else {
        // several rows: a warp per row, the rows side by side (the same picks and weights: both forms build the
        // list of the reference's insertion scan). By rounds: ranked by comparison, as in the streaming kernel, this launch
        // takes 14.8 us instead of 15.8 for 16 rows of 256 experts, but 11.1 instead of 10.4 for 4 rows of 32.
        for (uint32_t row = warp; row < a.T; row += kRouterWarps) {
            uint32_t id;
            float w;
            select_row<true>(a.logits + (size_t)row * a.ne, a, lane, id, w);
            if (lane < a.top_k) {
                a.ids[(size_t)row * a.top_k + lane] = id;
                a.weights[(size_t)row * a.top_k + lane] = w;
                ids_sm[row * a.top_k + lane] = id;
            }
        }
    }
    __syncthreads();
    bool ready = true;
    if (a.io_status) {
        const uint32_t s = *a.io_status;
        ready = s == 1u || s == 3u;
    }
    const uint32_t n_pairs = a.T * a.top_k;
    uint32_t misses = 0;
    for (uint32_t p = tid; p < n_pairs; p += blockDim.x) {
        const uint32_t e = min(ids_sm[p], a.ne - 1u);
        const uint64_t word = a.table[e];
        uint32_t slot = (uint32_t)(word & 0xffffffffu);
        const bool hit = (uint32_t)(word >> 32) == 2u && slot != SHRIKE_SLOT_MISS;
        if (!hit) { slot = SHRIKE_SLOT_MISS; ++misses; }
        if (a.slots) a.slots[p] = slot;
        if (slot != SHRIKE_SLOT_MISS && slot >= a.pool_cells) {
            report_status(a.status, kStatusBadIndex);
            slot = SHRIKE_SLOT_MISS;
        }
        sm.key[p] = ready ? slot : SHRIKE_SLOT_MISS;
        a.pair_cell[p] = sm.key[p];
    }
    if (misses) atomicAdd(&s_miss, misses);
    __syncthreads();
    if (tid == 0 && a.counts) {
        a.counts[0] = n_pairs - s_miss;
        a.counts[1] = s_miss;
    }
    // One row: every pair is its own instance; order them by cell as plan_body
    // would, with eight shuffles instead of the block-wide sort.
    bool fast = false;
    if (a.T == 1) {
        const uint32_t my = lane < n_pairs ? sm.key[lane] : SHRIKE_SLOT_MISS;
        uint32_t rank = 0;
        bool dup = false;
        for (uint32_t j = 0; j < n_pairs; ++j) {
            const uint32_t o = __shfl_sync(0xffffffffu, my, j);
            if (my != SHRIKE_SLOT_MISS && o != SHRIKE_SLOT_MISS) {
                rank += (o < my || (o == my && j < lane)) ? 1u : 0u;
                dup |= (o == my && j != lane);
            }
        }
        fast = !__any_sync(0xffffffffu, dup);  // same answer in every warp
        if (fast && warp == 0) {
            const uint32_t n_routed = __popc(__ballot_sync(0xffffffffu, my != SHRIKE_SLOT_MISS));
            if (my != SHRIKE_SLOT_MISS) {
                Instance in;
                in.kind = 0; in.slot = my; in.first = rank; in.count = 1;
                for (int q = 0; q < 8; ++q) in.pair[q] = lane;
                a.inst[rank + (a.with_shared ? 1u : 0u)] = in;
                a.sorted[rank] = lane;
            }
            if (lane == 0) {
                if (a.with_shared) {
                    Instance in;
                    in.kind = 1; in.slot = 0; in.first = 0; in.count = 1;
                    for (int q = 0; q < 8; ++q) in.pair[q] = 0;
                    a.inst[0] = in;
                }
                *a.n_inst = n_routed + (a.with_shared ? 1u : 0u);
            }
        }
    }
    if (!fast) plan_body(sm, n_pairs, a.T, a.with_shared, a.inst, a.n_inst, a.sorted, a.max_inst, a.status);
}

// moe_classify_residency_body for T rows. The miss lists keep router order: block b takes pairs
// [1024 b, 1024 b + 1024) and first counts the misses of all the pairs before them itself (independent loads,
// no hand-over between blocks), so its misses go to their final places.
__global__ void __launch_bounds__(1024) classify_kernel(const uint32_t* __restrict__ ids, const uint64_t* __restrict__ table,
                                                        uint32_t n_pairs, uint32_t ne, uint32_t* __restrict__ slots,
                                                        uint32_t* __restrict__ counts, uint32_t* __restrict__ miss_pos,
                                                        uint32_t* __restrict__ miss_exp) {
    __shared__ uint32_t s_miss[1024];
    __shared__ uint32_t s_base;
    pdl_wait();
    pdl_launch_dependents();
    auto slot_of = [](uint64_t word) {   // or SHRIKE_SLOT_MISS
        return (uint32_t)(word >> 32) == 2u ? (uint32_t)(word & 0xffffffffu) : SHRIKE_SLOT_MISS;
    };
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    uint32_t before_me = 0;
    if (counts || miss_pos || miss_exp) {   // the misses are asked for
        // Eight pairs of a thread at a time, written out: a lookup is two loads one after the other, and the compiler took the pairs
        // of a loop one by one (4096 rows of eight picks, caches cold: 17.8 us, so 9.4).
        constexpr uint32_t N = 8;
#pragma unroll 1
        for (uint32_t j = 0; j < blockIdx.x; j += N) {
            uint32_t e[N];
            uint64_t word[N];
#pragma unroll
            for (uint32_t q = 0; q < N; ++q) e[q] = j + q < blockIdx.x ? ids[(j + q) * 1024u + threadIdx.x] : 0u;
#pragma unroll
            for (uint32_t q = 0; q < N; ++q) word[q] = table[min(e[q], ne - 1u)];
#pragma unroll
            for (uint32_t q = 0; q < N; ++q) before_me += j + q < blockIdx.x && slot_of(word[q]) == SHRIKE_SLOT_MISS ? 1u : 0u;
        }
    }
    for (int o = 16; o; o >>= 1) before_me += __shfl_xor_sync(0xffffffffu, before_me, o);
    if ((threadIdx.x & 31u) == 0 && before_me) atomicAdd(&s_base, before_me);
    const uint32_t p = blockIdx.x * 1024u + threadIdx.x;
    bool miss = false;
    uint32_t e = 0;
    if (p < n_pairs) {
        e = min(ids[p], ne - 1u);
        const uint32_t slot = slot_of(table[e]);
        slots[p] = slot;
        miss = slot == SHRIKE_SLOT_MISS;
    }
    s_miss[threadIdx.x] = miss ? 1u : 0u;
    const uint32_t chunk = __syncthreads_count(miss);
    const uint32_t base = s_base;
    if (miss && (miss_pos || miss_exp)) {
        uint32_t before = 0;
        for (uint32_t j = 0; j < threadIdx.x; ++j) before += s_miss[j];
        if (miss_pos) miss_pos[base + before] = p;
        if (miss_exp) miss_exp[base + before] = e;
    }
    if (threadIdx.x == 0 && counts && blockIdx.x == gridDim.x - 1) {
        counts[0] = n_pairs - (base + chunk);
        counts[1] = base + chunk;
    }
}

RouterArgs make_router_args(const shrike_moe* m, const shrike_router_operands& ops, const void* hidden, uint32_t T,
                            uint32_t stride, uint32_t* ids, float* weights, float* shared_gate) {
    const shrike_moe_config& c = m->cfg;
    RouterArgs a = {};
    a.w = ops.weights; a.scales = ops.scales; a.biases = ops.biases; a.bits = c.router_weight_bits;
    a.gate_row = (ops.shared_gate && shared_gate) ? ops.shared_gate : nullptr;
    a.eff_scale = ops.effective_scale; a.logit_bias = ops.logit_bias; a.per_expert_scale = ops.per_expert_scale;
    a.hidden = hidden; a.T = T; a.stride = stride; a.dt = c.act_dtype; a.ne = c.num_experts; a.d = c.d;
    a.top_k = c.top_k; a.sigmoid_scores = c.router_kind == SHRIKE_ROUTER_SIGMOID; a.scaling = c.routed_scaling;
    a.round_f16 = c.round_route_weights_f16; a.logits = m->ws.logits; a.ids = ids; a.weights = weights;
    a.gate_out = shared_gate; a.tokens_per_block = T;
    return a;
}

cudaError_t launch_router(const shrike_moe* m, cudaStream_t st, const shrike_router_operands& ops,
                          const void* hidden, uint32_t T, uint32_t stride, uint32_t* ids,
                          float* weights, float* shared_gate) {
    RouterArgs a = make_router_args(m, ops, hidden, T, stride, ids, weights, shared_gate);
    const uint32_t rows = a.ne + (a.gate_row ? 1u : 0u);
    cudaError_t e;
    // A warp per row re-reads the activations for every expert row: ahead up to eight rows (the logits of 256 experts of 2048 columns, us:
    // 4 rows 2.8 against the tiles' 5.4, 8 rows 4.5 / 5.4, 16 rows 5.8 / 5.2, 64 rows 19 / 5.4; int8 rows 5.0 / 9.0, 9.0 / 9.0, 16 / 9, 60 / 9).
    // fp32 rows of 2048 and 2304 columns have straight-line code, and while its blocks run at once it keeps ahead of
    // tiles that are a few at most (4 experts of 2048 columns, 9 to 64 rows, us: bf16 6.7 / 7.1, fp32 7.2 / 8.2), of fp32 activations
    // at 2048 columns whatever the experts (16 experts 7.8 / 8.1; 128 experts, 9 rows 8.0 / 8.4, 40 rows, more than a block an SM, 12.5 / 8.5).
    const bool straight = a.bits == 0 && (a.d == 2048 || a.d == 2304) && (rows + kRouterWarps - 1) / kRouterWarps * ((T + 3) / 4) <= (uint32_t)m->sm_count &&
                          (a.ne < kRouterWarps || (a.d == 2048 && a.dt == SHRIKE_DTYPE_FP32));
    if (T > 8 && !(T <= 64 && straight) && router_tiles_take(a)) {
        e = launch_router_tiles(m, st, a);
        if (e != cudaSuccess) return e;
    } else {
        uint32_t tpb = 1;
        if (T > 64) tpb = 32;
        else if (T > 8) tpb = 4;
        a.tokens_per_block = tpb;
        const dim3 grid((rows + kRouterWarps - 1) / kRouterWarps, (T + tpb - 1) / tpb);
        e = launch_after(m, st, router_logits_kernel, grid, kRouterWarps * 32, 0, a);
        if (e != cudaSuccess) return e;
    }
    return launch_after(m, st, router_select_kernel, dim3((T + 3) / 4), 128, 0, a);
}

cudaError_t launch_route_fused(const shrike_moe* m, cudaStream_t st, const shrike_router_operands& ops,
                               const void* hidden, uint32_t T, uint32_t stride, const uint64_t* table,
                               uint32_t pool_cells, const uint32_t* io_status, uint32_t* ids, float* weights,
                               float* shared_gate, uint32_t* slots, uint32_t* counts, bool pdl) {
    RouterArgs a = make_router_args(m, ops, hidden, T, stride, ids, weights, shared_gate);
    a.table = table; a.pool_cells = pool_cells; a.io_status = io_status;
    a.with_shared = m->cfg.has_shared; a.int4 = m->cfg.weight_bits == 4; a.group = m->cfg.group_size;
    a.xsum = m->ws.xsum;
    a.slots = slots; a.counts = counts; a.inst = m->ws.inst; a.n_inst = m->ws.n_inst; a.sorted = m->ws.sorted;
    a.xh = m->ws.xh; a.done_counter = m->ws.done_counter; a.pair_cell = m->ws.pair_cell; a.status = m->ws.status; a.max_inst = max_instances(m->cfg, T);
    const uint32_t rows = a.ne + (a.gate_row ? 1u : 0u);
    cudaLaunchConfig_t cfg = {};
    // several rows: up to four blocks share an expert row's tokens (65 blocks would leave half of the SMs idle)
    const uint32_t gy = T < 4 ? (T ? T : 1u) : 4u;
    a.tokens_per_block = (T + gy - 1) / gy;
    cfg.gridDim = dim3((rows + kRouterWarps - 1) / kRouterWarps, gy);
    cfg.blockDim = dim3(kRouterWarps * 32);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = pdl ? attr : nullptr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, route_fused_kernel, a);
}

cudaError_t launch_classify(const shrike_moe* m, cudaStream_t st, const uint32_t* ids,
                            const uint64_t* table, uint32_t T, uint32_t* slots, uint32_t* counts,
                            uint32_t* miss_pos, uint32_t* miss_exp) {
    const uint32_t n_pairs = T * m->cfg.top_k;
    return launch_after(m, st, classify_kernel, dim3(n_pairs > 1024u ? (n_pairs + 1023u) / 1024u : 1u), 1024, 0, ids, table, n_pairs,
                        m->cfg.num_experts, slots, counts, miss_pos, miss_exp);
}

}  // namespace shrike

// ---- router entry point that allocates nothing --------------------------------
//
// Some hosts cannot let this library call cudaMalloc at all: a decode loop that
// has handed every free byte of HBM to the expert pool, a process whose memory
// plan is fixed before the first token, or a latency-critical thread that must
// not take cudaMalloc's device-wide synchronisation. shrike_moe_create sizes a
// workspace with cudaMalloc, so those hosts cannot own a handle. This entry
// point runs the router (logits + top-k + weights, and the shared expert's
// scalar gate) without one: its only scratch, the logits of up to
// SHRIKE_STATIC_ROUTER_MAX_ROWS rows by SHRIKE_MAX_EXPERTS experts, lives in
// the file-scope device array below (64 KiB on every GPU that loads the
// library, until the process exits).
#include <mutex>

namespace shrike {

static __device__ __align__(256) float g_static_router_logits[SHRIKE_STATIC_ROUTER_MAX_ROWS * SHRIKE_MAX_EXPERTS];

// Device address of the array, per device ordinal. The array's name is only a
// host-side stand-in in host code; the address the kernels need comes from
// cudaGetSymbolAddress, asked once per device with that device current.
static float* g_static_logits_ptr[64] = {};
static std::mutex g_static_logits_mutex;

static cudaError_t static_logits_for_current_device(float** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_static_logits_mutex);
    if (!g_static_logits_ptr[dev]) {
        float* p = nullptr;
        e = cudaGetSymbolAddress((void**)&p, g_static_router_logits);
        if (e != cudaSuccess) return e;
        g_static_logits_ptr[dev] = p;
    }
    *out = g_static_logits_ptr[dev];
    return cudaSuccess;
}

static int static_router_fail(char* text, size_t bytes, int code, const char* msg) {
    if (text && bytes) {
        size_t i = 0;
        for (; msg[i] && i + 1 < bytes; ++i) text[i] = msg[i];
        text[i] = 0;
    }
    return code;
}


// Affine rows -> fp32 (load-time utility for operands a packed file holds quantised): one thread per element.
__global__ void __launch_bounds__(256)
dequant_affine_rows_kernel(const uint8_t* __restrict__ packed, const uint16_t* __restrict__ scales,
                           const uint16_t* __restrict__ biases, uint32_t bits, uint32_t group, uint32_t meta_f16,
                           uint32_t rows, uint32_t cols, float* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)rows * cols) return;
    const uint32_t r = (uint32_t)(i / cols), c = (uint32_t)(i - (size_t)r * cols);
    const uint8_t byte = packed[(size_t)r * (cols * bits / 8) + (bits == 4 ? c / 2 : c)];
    const uint32_t q = bits == 4 ? ((c & 1u) ? (uint32_t)(byte >> 4) : (uint32_t)(byte & 15u)) : (uint32_t)byte;
    const size_t g = (size_t)r * (cols / group) + c / group;
    const float sc = meta_f16 ? f16_bits_to_f32(scales[g]) : bf16_bits_to_f32(scales[g]);
    const float bi = meta_f16 ? f16_bits_to_f32(biases[g]) : bf16_bits_to_f32(biases[g]);
    out[i] = __fmaf_rn((float)q, sc, bi);
}

cudaError_t launch_dequant_affine_rows(cudaStream_t st, const void* packed, const void* scales, const void* biases,
                                       uint32_t bits, uint32_t group, uint32_t meta_dtype, uint32_t rows, uint32_t cols,
                                       float* out) {
    const size_t n = (size_t)rows * cols;
    dequant_affine_rows_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        (const uint8_t*)packed, (const uint16_t*)scales, (const uint16_t*)biases, bits, group,
        meta_dtype == SHRIKE_DTYPE_FP16 ? 1u : 0u, rows, cols, out);
    return cudaGetLastError();
}

}  // namespace shrike

extern "C" int shrike_encode_router_static(const shrike_moe_config* config, void* stream,
                                           const shrike_router_operands* ops, const void* hidden,
                                           uint32_t query_count, uint32_t hidden_stride_elements,
                                           uint32_t* out_indices, float* out_weights, float* out_shared_gate,
                                           char* error_text, size_t error_text_bytes) {
    using namespace shrike;
    auto bad = [&](int code, const char* msg) { return static_router_fail(error_text, error_text_bytes, code, msg); };
    if (!config) return bad(SHRIKE_EINVAL, "static router: config is null");
    if (query_count == 0) return SHRIKE_OK;
    const shrike_moe_config& c = *config;
    if (query_count > SHRIKE_STATIC_ROUTER_MAX_ROWS)
        return bad(SHRIKE_ERANGE, "static router: query_count exceeds SHRIKE_STATIC_ROUTER_MAX_ROWS (64); "
                                  "the built-in scratch holds 64 rows of logits");
    if (c.num_experts == 0 || c.num_experts > SHRIKE_MAX_EXPERTS)
        return bad(SHRIKE_ERANGE, "static router: num_experts must be 1..256 (the built-in scratch is 64 x 256 floats)");
    if (c.top_k == 0 || c.top_k > SHRIKE_MAX_TOP_K || c.top_k > c.num_experts)
        return bad(SHRIKE_EINVAL, "static router: top_k must be 1..8 and at most num_experts");
    if (c.d == 0 || c.d % 64 != 0 || c.d > 2944) return bad(SHRIKE_EINVAL, "static router: d must be a multiple of 64, at most 2944");
    if (c.act_dtype > SHRIKE_DTYPE_FP32 || c.router_kind > SHRIKE_ROUTER_SIGMOID ||
        (c.router_weight_bits != 0 && c.router_weight_bits != 4 && c.router_weight_bits != 8))
        return bad(SHRIKE_EINVAL, "static router: unknown act_dtype, router_kind or router_weight_bits");
    if (!ops || !ops->weights || !hidden || !out_indices || !out_weights)
        return bad(SHRIKE_EINVAL, "static router: null operand");
    if (c.router_weight_bits != 0 && (!ops->scales || !ops->biases))
        return bad(SHRIKE_EINVAL, "static router: affine weights need scales and biases");
    if (hidden_stride_elements < c.d || hidden_stride_elements % 4 != 0)
        return bad(SHRIKE_EINVAL, "static router: hidden stride must be >= d and a multiple of 4 elements");
    if (c.shared_gated && (!ops->shared_gate || !out_shared_gate))
        return bad(SHRIKE_EINVAL, "static router: a shared_gated config needs shared_gate and out_shared_gate");
    const char* why = nullptr;
    if (!router_operands_aligned(c, *ops, hidden, &why)) return bad(SHRIKE_EINVAL, why);
    float* logits = nullptr;
    cudaError_t e = static_logits_for_current_device(&logits);
    if (e != cudaSuccess) return bad(SHRIKE_EIO, cudaGetErrorString(e));

    RouterArgs a = {};
    a.w = ops->weights; a.scales = ops->scales; a.biases = ops->biases; a.bits = c.router_weight_bits;
    a.gate_row = (ops->shared_gate && out_shared_gate) ? ops->shared_gate : nullptr;
    a.eff_scale = ops->effective_scale; a.logit_bias = ops->logit_bias; a.per_expert_scale = ops->per_expert_scale;
    a.hidden = hidden; a.T = query_count; a.stride = hidden_stride_elements; a.dt = c.act_dtype;
    a.ne = c.num_experts; a.d = c.d; a.top_k = c.top_k;
    a.sigmoid_scores = c.router_kind == SHRIKE_ROUTER_SIGMOID; a.scaling = c.routed_scaling;
    a.round_f16 = c.round_route_weights_f16; a.logits = logits; a.ids = out_indices; a.weights = out_weights;
    a.gate_out = out_shared_gate;
    const uint32_t rows = a.ne + (a.gate_row ? 1u : 0u);
    const uint32_t tpb = query_count > 8 ? 4 : 1;
    a.tokens_per_block = tpb;
    cudaStream_t st = (cudaStream_t)stream;
    router_logits_kernel<<<dim3((rows + kRouterWarps - 1) / kRouterWarps, (query_count + tpb - 1) / tpb),
                           kRouterWarps * 32, 0, st>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return bad(SHRIKE_EIO, cudaGetErrorString(e));
    router_select_kernel<<<(query_count + 3) / 4, 128, 0, st>>>(a);
    e = cudaGetLastError();
    if (e != cudaSuccess) return bad(SHRIKE_EIO, cudaGetErrorString(e));
    return SHRIKE_OK;
}

