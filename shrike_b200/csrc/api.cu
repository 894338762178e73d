// The C ABI: argument validation, handle lifetime, launch sequencing.
// No entry point below allocates after shrike_moe_create / shrike_pool_create /
// shrike_residency_create.
#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>

#include "internal.h"
#include "route_args.cuh"

using namespace shrike;

namespace {

thread_local char g_create_error[kErrorText];

int fail(shrike_moe* m, int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(m ? m->err : g_create_error, kErrorText, fmt, ap);
    va_end(ap);
    return code;
}

// A failure on one handle, reported on another.
int pass_on(shrike_moe* to, const shrike_moe* from, int code) {
    if (to != from) memcpy(to->err, from->err, kErrorText);
    return code;
}

int cuda_fail(shrike_moe* m, cudaError_t e, const char* what) {
    return fail(m, SHRIKE_EIO, "%s: %s", what, cudaGetErrorString(e));
}

#define CU(call)                                                  \
    do {                                                          \
        cudaError_t e_ = (call);                                  \
        if (e_ != cudaSuccess) return cuda_fail(m, e_, #call);    \
    } while (0)

bool valid_config(const shrike_moe_config& c, const char*& why) {
    auto bad = [&](const char* s) { why = s; return false; };
    if (c.d == 0 || c.d % 64 != 0 || c.d > 2944) return bad("d must be a multiple of 64, at most 2944");
    if (c.f == 0 || c.f % 64 != 0) return bad("f must be a multiple of 64");
    if (c.num_experts == 0 || c.num_experts > SHRIKE_MAX_EXPERTS) return bad("num_experts must be 1..256");
    if (c.top_k == 0 || c.top_k > SHRIKE_MAX_TOP_K || c.top_k > c.num_experts) return bad("top_k must be 1..8 and <= num_experts");
    if (c.weight_bits != 4 && c.weight_bits != 8) return bad("weight_bits must be 4 or 8");
    if (c.group_size != 32 && c.group_size != 64) return bad("group_size must be 32 or 64");
    if (c.meta_dtype > SHRIKE_DTYPE_FP16) return bad("meta_dtype must be BF16 or FP16");
    if (c.act_dtype > SHRIKE_DTYPE_FP32) return bad("act_dtype must be BF16, FP16 or FP32");
    if (c.activation > SHRIKE_ACT_CLAMPED_SWIGLU) return bad("unknown activation");
    if (c.router_kind > SHRIKE_ROUTER_SIGMOID) return bad("unknown router_kind");
    if (c.router_weight_bits != 0 && c.router_weight_bits != 4 && c.router_weight_bits != 8) return bad("router_weight_bits must be 0, 4 or 8");
    if (c.has_shared && (c.shared_f == 0 || c.shared_f % 64 != 0)) return bad("shared_f must be a multiple of 64");
    if (c.shared_gated && !c.has_shared) return bad("shared_gated needs has_shared");
    if (c.max_tokens == 0 || c.max_tokens > 65536) return bad("max_tokens must be 1..65536");
    if (c.y_dtype > SHRIKE_DTYPE_FP32) return bad("y_dtype must be BF16, FP16 or FP32");
    return true;
}

void make_offsets(const shrike_moe_config& c, bool shared, shrike_expert_offsets& o, uint64_t& bytes) {
    const uint32_t f = shared ? c.shared_f : c.f;
    const uint32_t rows[3] = {f, f, c.d}, cols[3] = {c.d, c.d, f};
    uint32_t w[3], s[3], b[3], ab[3];
    uint64_t cur = 0;
    for (int p = 0; p < 3; ++p) {
        const uint64_t wb = (uint64_t)rows[p] * (cols[p] * c.weight_bits / 8);
        const uint64_t mb = (uint64_t)rows[p] * (cols[p] / c.group_size) * 2;
        w[p] = (uint32_t)cur; cur += wb;
        s[p] = (uint32_t)cur; cur += mb;
        b[p] = (uint32_t)cur; cur += mb;
        if (c.expert_bias) { ab[p] = (uint32_t)cur; cur += rows[p] * 2; } else ab[p] = 0;
    }
    o.gate_w = w[0]; o.gate_s = s[0]; o.gate_b = b[0]; o.gate_ab = ab[0];
    o.up_w = w[1]; o.up_s = s[1]; o.up_b = b[1]; o.up_ab = ab[1];
    o.down_w = w[2]; o.down_s = s[2]; o.down_b = b[2]; o.down_ab = ab[2];
    bytes = cur;
}

bool offsets_aligned(const shrike_expert_offsets& o) {
    const uint32_t* p = &o.gate_w;
    for (int i = 0; i < 12; ++i)
        if (p[i] % 16 != 0) return false;
    return true;
}

// Every encode call launches on the current device against this handle's workspace and pool.
int check_device(shrike_moe* m) {
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev != m->device)
        return fail(m, SHRIKE_EINVAL, "the handle lives on device %d but device %d is current", m->device, dev);
    return SHRIKE_OK;
}

bool aligned_to(const void* p, uintptr_t a) { return ((uintptr_t)p & (a - 1)) == 0; }

// cudaMemset, finished when it returns: it runs on the legacy stream, which a caller's non-blocking stream does not wait for,
// and a call on such a stream may come next.
cudaError_t set_now(void* p, int value, size_t bytes) {
    const cudaError_t e = cudaMemset(p, value, bytes);
    return e == cudaSuccess ? cudaStreamSynchronize(cudaStreamLegacy) : e;
}

// Makes `device` current for the scope and puts the caller's device back afterwards.
struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int device) {
        cudaGetDevice(&prev);
        if (prev != device) cudaSetDevice(device);
    }
    ~DeviceGuard() { if (prev >= 0) cudaSetDevice(prev); }
};

}  // namespace

namespace shrike {
// What the router kernels' vector loads rely on; `why` receives the first violation.
bool router_operands_aligned(const shrike_moe_config& c, const shrike_router_operands& o, const void* hidden,
                             const char** why) {
    auto bad = [&](const char* s) { *why = s; return false; };
    if (!aligned_to(hidden, c.act_dtype == SHRIKE_DTYPE_FP32 ? 16 : 8))
        return bad("hidden must be 16-byte aligned (fp32) or 8-byte aligned (16-bit activations)");
    if (!aligned_to(o.weights, 16)) return bad("router weights must be 16-byte aligned");
    if (o.shared_gate && !aligned_to(o.shared_gate, 16)) return bad("shared_gate must be 16-byte aligned");
    if (o.effective_scale && !aligned_to(o.effective_scale, 8)) return bad("effective_scale must be 8-byte aligned");
    if (!aligned_to(o.scales, 2) || !aligned_to(o.biases, 2) || !aligned_to(o.logit_bias, 2) ||
        !aligned_to(o.per_expert_scale, 2))
        return bad("scales, biases, logit_bias and per_expert_scale must be 2-byte aligned");
    return true;
}
}  // namespace shrike

namespace {

void free_workspace(Workspace& w) {
    for (uint32_t i = 0; i < w.n_blocks; ++i) cudaFree(w.blocks[i]);
    free(w.tensor_maps);
    free(w.fused_geom);
    free(w.fused_maps);
    w = Workspace();
}

int fill_expert_args(shrike_moe* m, const shrike_pool* pool, const shrike_expert_offsets* ro,
                     const shrike_shared_expert* shared, const float* weights, const float* shared_gate,
                     ExpertArgs& a, bool check_gate = true) {
    const shrike_moe_config& c = m->cfg;
    if (!pool || !ro) return fail(m, SHRIKE_EINVAL, "pool and routed_offsets are required");
    if (!offsets_aligned(*ro)) return fail(m, SHRIKE_EINVAL, "routed offsets must be multiples of 16 bytes");
    if (c.has_shared) {
        if (!shared || !shared->block) return fail(m, SHRIKE_EINVAL, "this handle was created with a shared expert; pass it");
        if (!offsets_aligned(shared->offsets) || ((uintptr_t)shared->block & 15))
            return fail(m, SHRIKE_EINVAL, "shared expert block and offsets must be 16-byte aligned");
    }
    if (check_gate && shared_gate && !c.shared_gated) return fail(m, SHRIKE_EINVAL, "shared_gate given but the handle is not shared_gated");
    if (check_gate && c.shared_gated && !shared_gate) return fail(m, SHRIKE_EINVAL, "shared_gated handle needs the router's shared_gate output");
    memset(&a, 0, sizeof a);
    a.pool = pool->view;
    a.routed = to_offsets3(*ro);
    if (c.has_shared) {
        a.shared = to_offsets3(shared->offsets);
        a.shared_block = (const uint8_t*)shared->block;
    }
    a.d = c.d; a.f = c.f; a.f_shared = c.has_shared ? c.shared_f : 0; a.top_k = c.top_k;
    a.activation = c.activation; a.expert_bias = c.expert_bias; a.act_dtype = c.act_dtype; a.y_dtype = c.y_dtype;
    a.inst = m->ws.inst; a.n_inst = m->ws.n_inst; a.sorted = m->ws.sorted; a.xh = m->ws.xh;
    a.xsum = m->ws.xsum;
    a.acts = m->ws.acts; a.acts_shared = m->ws.acts_shared; a.yacc = m->ws.yacc;
    a.route_w = weights; a.shared_gate = shared_gate; a.status = m->ws.status;
#ifdef SHRIKE_TRACE
    a.trace = m->trace;
#endif
    return SHRIKE_OK;
}


// Whether the streaming kernel is the faster one for a decode call. A single row has nothing to lay out ahead of the first
// tile (us a layer, one-row or per-tile kernels and streaming; 256 experts of 2048 x 512 int4 | 32 of 2880 x 2880 int4 | 256 of
// 2304 x 1024 int8: 17.0, 22.9 | 40.4, 42.0 | 34.0, 36.3); two rows have: 29.3, 27.1 | 88, 57.5 | 46.8, 43.3. Up to 64 rows it is
// also ahead of the expert-grouped GEMM, which reads an expert once for all its rows but starts in a dozen launches, unless few
// large experts get many rows (streaming and grouped, uniform picks):
//   17 rows  65, 92 | 130, 187 | 134, 176     48 rows  110, 134 | 170, 191 | 210, 246     64 rows  121, 145 | 210, 192 | 240, 266
// With picks by Zipf(1.1), 48 rows: 67, 69 | 173, 172 | 152, 163; 64 rows: 79, 72 | 218, 179 | 179, 174. There too its rows are sums in
// a fixed order, which the grouped GEMM's are not, those of the separate calls, and of products with the packed integers as they are, where
// the grouped GEMM rounds a weight to fp16.
// The projections as calls of their own follow the same rule, so that they give a layer call's rows bit for bit. Each pays the
// kernel's set-up, with no router to share: plan and both of them, us, per-tile kernels and streaming, 30.3, 32.8 | 85, 62 | 45.9,
// 49.3 at two rows, 34.4, 37.0 | 113, 76 | 60.2, 57.5 at three, 41.1, 39.9 | 138, 82 | 72, 66 at four.
bool stream_pays(uint32_t T) { return T > 1; }

// The expert projections of a decode call's work lists (phases: 1, 2 or 3 = both, a launch each). The streaming kernel takes
// every shape whose tiles its ring and the tiled copies can hold; the per-tile kernels take the others.
cudaError_t launch_experts(const shrike_moe* m, cudaStream_t st, const ExpertArgs& a, uint32_t T, uint32_t phases, void* y,
                           void* hidden, bool pdl) {
    const uint32_t n_shared = m->cfg.has_shared ? (T + 7) / 8 : 0;
    const uint32_t mi = max_instances(m->cfg, T);
    for (uint32_t phase = 1; phase <= 2; ++phase) {
        if (!(phases & phase)) continue;
        cudaError_t e = stream_pays(T) ? launch_expert_stream(m, st, a, T, n_shared, y, hidden, pdl, phase) : cudaErrorNotSupported;
        if (e == cudaErrorNotSupported)
            e = phase == 1 ? launch_phase1(m, st, a, mi, pdl) : launch_phase2(m, st, a, T, mi, y, hidden, pdl);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// The prefill call with the status word of a streamed batch (moe.metal:36-39, 918-921): when io_status is
// given and the word is neither READY nor 3, the routed experts are skipped and y is the shared term alone.
int encode_prefill(shrike_moe* m, void* stream, const shrike_pool* pool,
                   const shrike_expert_offsets* routed_offsets, const uint32_t* topk_indices,
                   const uint32_t* resolved_slots, const float* routing_weights, const void* x,
                   uint32_t query_count, const shrike_shared_expert* shared, const float* shared_gate,
                   const uint32_t* io_status, void* y, void* hidden) {
    if (!m) return SHRIKE_EINVAL;
    if (!topk_indices || !resolved_slots || !routing_weights || !x || !y)
        return fail(m, SHRIKE_EINVAL, "prefill: null operand");
    if (query_count > m->cfg.max_tokens) return fail(m, SHRIKE_ERANGE, "query_count exceeds max_tokens");
    if (m->cfg.max_tokens <= SHRIKE_MAX_DECODE_TOKENS)
        return fail(m, SHRIKE_EINVAL, "handle was created for decode only (max_tokens <= %u)", SHRIKE_MAX_DECODE_TOKENS);
    if (query_count == 0) return SHRIKE_OK;
    ExpertArgs a;
    int rc = fill_expert_args(m, pool, routed_offsets, shared, routing_weights, shared_gate, a);
    if (rc) return rc;
    if ((rc = check_device(m))) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const uint32_t mi = max_instances(m->cfg, query_count);
    // The expert-grouped GEMM runs on the tcgen05 tensor cores. Shapes whose K is not a multiple of 64 keep
    // every expert on the 8-row warp-MMA tiles (the decode kernels); SHRIKE_PREFILL_PATH=mma in the
    // environment of shrike_moe_create forces them for a handle (a test switch).
    const bool warp_mma = m->force_warp_mma || !umma_supported(m->cfg);
    // fp32 rows out and no residual to add: the down epilogue adds straight into y and no pass over the rows follows. The
    // kernel that reads x clears y, block by block: not when y is x (they must not overlap otherwise)
    const bool direct = m->cfg.y_dtype == SHRIKE_DTYPE_FP32 && !hidden && y != x;
    if (direct) a.yacc = (float*)y;
    CU(launch_prefill_plan(m, st, topk_indices, resolved_slots, x, query_count, m->cfg.has_shared != 0,
                           pool->view.cells, warp_mma, io_status, nullptr, nullptr, direct ? (float*)y : nullptr));
    if (warp_mma) {
        CU(launch_phase1(m, st, a, mi, false));
        CU(launch_phase2_accumulate(m, st, a, mi));
    } else {
        CU(launch_umma_prefill(m, st, a, query_count));
    }
    if (!direct) CU(launch_prefill_combine(m, st, query_count, y, hidden));
    return SHRIKE_OK;
}

}  // namespace

namespace shrike {
size_t act_bytes(uint32_t dt) { return dt == SHRIKE_DTYPE_FP32 ? 4 : 2; }
}

extern "C" {

const char* shrike_last_error(const shrike_moe* moe) {
    return moe ? moe->err : g_create_error;
}

int shrike_expert_offsets_make(const shrike_moe_config* config, int shared, shrike_expert_offsets* out,
                               uint64_t* block_bytes) {
    const char* why = nullptr;
    if (!config || !out) return fail(nullptr, SHRIKE_EINVAL, "null argument");
    if (!valid_config(*config, why)) return fail(nullptr, SHRIKE_EINVAL, "%s", why);
    if (shared && !config->has_shared) return fail(nullptr, SHRIKE_EINVAL, "config has no shared expert");
    uint64_t bytes;
    make_offsets(*config, shared != 0, *out, bytes);
    if (block_bytes) *block_bytes = bytes;
    return SHRIKE_OK;
}

int shrike_moe_create(const shrike_moe_config* config, int device, shrike_moe** out) {
    if (!config || !out) return fail(nullptr, SHRIKE_EINVAL, "null argument");
    *out = nullptr;
    const char* why = nullptr;
    if (!valid_config(*config, why)) return fail(nullptr, SHRIKE_EINVAL, "%s", why);
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if (e != cudaSuccess || count == 0)
        return fail(nullptr, SHRIKE_EIO, "no CUDA device: %s (this library has no CPU path)",
                    cudaGetErrorString(e));
    if (device < 0 || device >= count) return fail(nullptr, SHRIKE_ERANGE, "device %d out of range", device);
    int caller_device = device;
    cudaGetDevice(&caller_device);
    e = cudaSetDevice(device);
    if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaSetDevice");
    // the caller's current device is put back on every way out
    struct Restore { int dev; ~Restore() { cudaSetDevice(dev); } } restore{caller_device};
    shrike_moe* m = new (std::nothrow) shrike_moe();
    if (!m) return fail(nullptr, SHRIKE_ENOMEM, "host allocation failed");
    m->cfg = *config;
    m->device = device;
    cudaDeviceGetAttribute(&m->sm_count, cudaDevAttrMultiProcessorCount, device);
    // switches for tests and diagnostics, read once here and never on the per-layer path
    m->no_pdl = getenv("SHRIKE_NO_PDL") != nullptr;
    m->single_stream = getenv("SHRIKE_SINGLE_STREAM") != nullptr;
    const char* path = getenv("SHRIKE_PREFILL_PATH");
    m->force_warp_mma = path && strcmp(path, "mma") == 0;
    const shrike_moe_config& c = m->cfg;
    Workspace& w = m->ws;
    const size_t T = c.max_tokens, K = c.top_k;
    w.max_inst = max_instances(c, c.max_tokens);
    const size_t ab = act_bytes(c.act_dtype), yb = act_bytes(c.y_dtype);
    bool ok = true;
    // The small parts share a device allocation, the others have one each: requests below a megabyte share the driver's
    // 2 MB mappings, and a mapping (0.3 ms) is what making a handle costs.
    struct Part { void** p; size_t at; } small_parts[kWorkspaceParts];
    uint32_t n_small = 0;
    size_t small_bytes = 0;
    auto A = [&](auto** p, size_t bytes) {
        if (!ok || n_small + w.n_blocks + 1 >= kWorkspaceParts) {
            ok = false;
            return;
        }
        if (bytes < (64u << 10)) {
            small_parts[n_small++] = {(void**)p, small_bytes};
            small_bytes += (bytes + 255) / 256 * 256;
            return;
        }
        void* at = nullptr;
        if (cudaMalloc(&at, bytes) != cudaSuccess) ok = false;
        else { w.blocks[w.n_blocks++] = at; *(void**)p = at; }
    };
    // words that start at zero
    A(&w.status, 4);
    A(&w.n_inst, 4);
    A(&w.done_counter, 4);
    A(&w.arrived, 8);
    A(&w.fused_epoch, 4);
    A(&w.plan_ticket, 4);
    const size_t zeroed = small_bytes;
    A(&w.logits, T * c.num_experts * 4);
    A(&w.xh, T * c.d * 2);
    A(&w.xsum, T * (c.d / c.group_size) * 4);
    A(&w.acts, T * K * c.f * 2);
    A(&w.acts_shared, c.has_shared ? T * c.shared_f * 2 : 0);
    A(&w.sorted, T * K * 4);
    A(&w.inst, (size_t)w.max_inst * sizeof(Instance));
    A(&w.inst_done, stream_done_bytes());
    A(&w.parts, stream_parts_bytes(c));
    A(&w.pair_cell, std::min(T, (size_t)SHRIKE_MAX_DECODE_TOKENS) * K * 4);
    A(&w.block_hist, ((T + 127) / 128) * c.num_experts * 4);
    A(&w.expert_offsets, c.num_experts * 4);
    A(&w.expert_counts, c.num_experts * 4);
    A(&w.slot_of_expert, c.num_experts * 4);
    A(&w.yacc, T > SHRIKE_MAX_DECODE_TOKENS ? T * c.d * 4 : 0);
    A(&w.chunk_inst, T > SHRIKE_MAX_DECODE_TOKENS ? umma_max_chunk_instances(c, c.max_tokens) * umma_chunk_instance_bytes() : 0);
    A(&w.n_chunk_inst, 16);
    if (T > SHRIKE_MAX_DECODE_TOKENS) A(&w.rank_of_pair, T * K * 4);
    if (T > SHRIKE_MAX_DECODE_TOKENS) A(&w.xs, T * K * c.d * 2);   // prefill operands
    A(&w.x_dev, T * c.d * ab);
    A(&w.y_dev, T * c.d * yb);
    A(&w.ids_dev, T * K * 4);
    A(&w.w_dev, T * K * 4);
    A(&w.gate_dev, T * 4);
    A(&w.slots_dev, T * K * 4);
    A(&w.counts_dev, 8);
    // the one-row layer kernel: sizes of its shared-memory ring, and its hand-over buffers
    int smem_optin = 0;
    cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    m->smem_optin = (uint32_t)smem_optin;
    w.fused_geom = malloc(fused_geom_bytes());
    w.fused_maps = calloc(1, fused_map_cache_bytes());
    if (!w.fused_maps) ok = false;
    if (w.fused_geom && fused_geometry(c, m->sm_count, smem_optin, *(FusedGeom*)w.fused_geom)) {
        A((uint8_t**)&w.fused_logits, fused_logits_bytes(c));
        A(&w.fused_acts, fused_acts_bytes(c));
    } else {
        free(w.fused_geom);
        w.fused_geom = nullptr;
    }
    void* small = nullptr;
    if (ok) ok = cudaMalloc(&small, small_bytes) == cudaSuccess;
    if (ok) w.blocks[w.n_blocks++] = small;
    if (!ok) {
        free_workspace(w);
        delete m;
        cudaGetLastError();
        return fail(nullptr, SHRIKE_ENOMEM, "device allocation of the workspace failed");
    }
    for (uint32_t i = 0; i < n_small; ++i) *small_parts[i].p = (uint8_t*)small + small_parts[i].at;
    cudaError_t se = cudaSuccess;
    if (w.fused_geom) {
        // no logit carries the first epoch's tag, no activation has been published
        se = cudaMemset(w.fused_logits, 0xff, fused_logits_bytes(c));
        if (se == cudaSuccess) se = cudaMemset(w.fused_acts, 0xff, fused_acts_bytes(c));
    }
    if (se == cudaSuccess) se = set_now(small, 0, zeroed);
    if (se != cudaSuccess) {
        free_workspace(w);
        delete m;
        return cuda_fail(nullptr, se, "clearing the workspace");
    }
    if (T > SHRIKE_MAX_DECODE_TOKENS) {
        w.tensor_maps = aligned_alloc(64, umma_tensor_map_bytes());
        const cudaError_t me = w.tensor_maps ? umma_prepare(m) : cudaErrorMemoryAllocation;
        if (me != cudaSuccess) {
            free_workspace(w);
            delete m;
            cudaGetLastError();
            return fail(nullptr, SHRIKE_EIO, "TMA descriptors of the prefill operands: %s", cudaGetErrorString(me));
        }
    }
    *out = m;
    return SHRIKE_OK;
}

void shrike_moe_destroy(shrike_moe* moe) {
    if (!moe) return;
    DeviceGuard guard(moe->device);
    free_workspace(moe->ws);
    if (moe->residency) cudaFree(moe->residency);
    delete moe;
}

int shrike_moe_status(shrike_moe* m, void* stream) {
    if (!m) return SHRIKE_EINVAL;
    // The word comes through the stream: a copy of its own after the synchronise is another way to the device and back (a host call of
    // two rows 120 -> 112 us). To memory that is not pinned the copy returns when it is there.
    uint32_t st = 0;
    CU(cudaMemcpyAsync(&st, m->ws.status, 4, cudaMemcpyDeviceToHost, (cudaStream_t)stream));
    CU(cudaStreamSynchronize((cudaStream_t)stream));
    if (st != kStatusOk) {
        CU(set_now(m->ws.status, 0, 4));
        if (st == kStatusWaitTimeout) return fail(m, SHRIKE_ETIMEDOUT, "a device-side wait gave up");
        if (st == kStatusOperandRange)
            return fail(m, SHRIKE_ERANGE, "an activation beyond the fp16 operand range (|x| > 65504) was clamped");
        return fail(m, SHRIKE_ERANGE, "a kernel met a slot id outside the pool");
    }
    return SHRIKE_OK;
}

#ifdef SHRIKE_TRACE
int shrike_debug_set_trace(shrike_moe* m, uint64_t* trace_device_buffer) {
    if (!m) return SHRIKE_EINVAL;
    m->trace = trace_device_buffer;
    return SHRIKE_OK;
}
#endif

// ---- pool -------------------------------------------------------------------

int shrike_pool_create(shrike_moe* m, uint32_t cells, uint64_t cell_stride, uint32_t chunks,
                       shrike_pool** out) {
    if (!m || !out) return SHRIKE_EINVAL;
    *out = nullptr;
    if (cells == 0 || chunks == 0 || chunks > SHRIKE_MAX_POOL_CHUNKS)
        return fail(m, SHRIKE_EINVAL, "cells must be > 0 and chunks 1..8");
    if (cell_stride == 0 || cell_stride % 256 != 0)
        return fail(m, SHRIKE_EINVAL, "cell_stride must be a positive multiple of 256 bytes");
    DeviceGuard guard(m->device);
    shrike_pool* p = new (std::nothrow) shrike_pool();
    if (!p) return fail(m, SHRIKE_ENOMEM, "host allocation failed");
    memset(p, 0, sizeof *p);
    p->owner = m;
    p->chunks = chunks;
    p->view.cells = cells;
    p->view.stride = cell_stride;
    p->view.cells_per_chunk = (cells + chunks - 1) / chunks;
    for (uint32_t i = 0; i < SHRIKE_MAX_POOL_CHUNKS; ++i) p->view.base[i] = nullptr;
    for (uint32_t i = 0; i < chunks; ++i) {
        const uint64_t first = (uint64_t)i * p->view.cells_per_chunk;
        if (first >= cells) { p->chunks = i; break; }
        const uint64_t n = (first + p->view.cells_per_chunk <= cells) ? p->view.cells_per_chunk : cells - first;
        cudaError_t e = cudaMalloc(&p->chunk[i], n * cell_stride);
        if (e != cudaSuccess) {
            for (uint32_t j = 0; j < i; ++j) cudaFree(p->chunk[j]);
            delete p;
            cudaGetLastError();
            return fail(m, SHRIKE_ENOMEM, "pool chunk of %llu bytes: %s", (unsigned long long)(n * cell_stride),
                        cudaGetErrorString(e));
        }
        p->view.base[i] = (const uint8_t*)p->chunk[i];
    }
    *out = p;
    return SHRIKE_OK;
}

void shrike_pool_destroy(shrike_pool* pool) {
    if (!pool) return;
    DeviceGuard guard(pool->owner->device);
    for (uint32_t i = 0; i < pool->chunks; ++i)
        if (pool->chunk[i]) cudaFree(pool->chunk[i]);
    delete pool;
}

int shrike_pool_cell_address(const shrike_pool* pool, uint32_t cell, void** out) {
    if (!pool || !out) return SHRIKE_EINVAL;
    if (cell >= pool->view.cells) return fail(pool->owner, SHRIKE_ERANGE, "cell %u out of range", cell);
    *out = (void*)pool_cell_base(pool->view, cell);
    return SHRIKE_OK;
}

int shrike_pool_upload(shrike_pool* pool, uint32_t cell, const void* block_host, uint64_t bytes, void* stream) {
    if (!pool || !block_host) return SHRIKE_EINVAL;
    shrike_moe* m = pool->owner;
    if (cell >= pool->view.cells) return fail(m, SHRIKE_ERANGE, "cell %u out of range", cell);
    if (bytes > pool->view.stride) return fail(m, SHRIKE_ERANGE, "block larger than the cell stride");
    CU(cudaMemcpyAsync((void*)pool_cell_base(pool->view, cell), block_host, bytes, cudaMemcpyHostToDevice,
                       (cudaStream_t)stream));
    return SHRIKE_OK;
}

int shrike_pool_download(shrike_pool* pool, uint32_t cell, void* block_host, uint64_t bytes, void* stream) {
    if (!pool || !block_host) return SHRIKE_EINVAL;
    shrike_moe* m = pool->owner;
    if (cell >= pool->view.cells) return fail(m, SHRIKE_ERANGE, "cell %u out of range", cell);
    if (bytes > pool->view.stride) return fail(m, SHRIKE_ERANGE, "block larger than the cell stride");
    CU(cudaMemcpyAsync(block_host, pool_cell_base(pool->view, cell), bytes, cudaMemcpyDeviceToHost,
                       (cudaStream_t)stream));
    CU(cudaStreamSynchronize((cudaStream_t)stream));
    return SHRIKE_OK;
}

int shrike_pool_fill_synthetic(shrike_moe* m, shrike_pool* pool, uint32_t first_cell, uint32_t count,
                               uint64_t seed, uint32_t layer, uint32_t first_expert, int shared, void* stream) {
    if (!m || !pool) return SHRIKE_EINVAL;
    if ((uint64_t)first_cell + count > pool->view.cells) return fail(m, SHRIKE_ERANGE, "cells out of range");
    if (shared && !m->cfg.has_shared) return fail(m, SHRIKE_EINVAL, "no shared expert in this config");
    shrike_expert_offsets o;
    uint64_t bytes;
    make_offsets(m->cfg, shared != 0, o, bytes);
    if (bytes > pool->view.stride) return fail(m, SHRIKE_ERANGE, "block larger than the cell stride");
    if (count == 0) return SHRIKE_OK;
    CU(launch_synth_fill(m, (cudaStream_t)stream, pool->view, first_cell, count, seed, layer, first_expert,
                         shared != 0, to_offsets3(o)));
    return SHRIKE_OK;
}

// ---- residency ----------------------------------------------------------------

int shrike_residency_create(shrike_moe* m, uint32_t layers, uint64_t** table_out) {
    if (!m || layers == 0) return SHRIKE_EINVAL;
    DeviceGuard guard(m->device);
    if (m->residency) { cudaFree(m->residency); m->residency = nullptr; }
    const size_t n = (size_t)layers * m->cfg.num_experts;
    cudaError_t e = cudaMalloc((void**)&m->residency, n * 8);
    if (e != cudaSuccess) { cudaGetLastError(); return fail(m, SHRIKE_ENOMEM, "residency table: %s", cudaGetErrorString(e)); }
    // every entry: state 0 (absent)
    CU(set_now(m->residency, 0, n * 8));
    m->residency_layers = layers;
    if (table_out) *table_out = m->residency;
    return SHRIKE_OK;
}

__global__ void residency_identity_kernel(uint64_t* row, uint32_t ne, uint32_t first_cell) {
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < ne) row[e] = ((uint64_t)2 << 32) | (uint64_t)(first_cell + e);
}

__global__ void residency_set_kernel(uint64_t* word, uint64_t value) {
    // one 64-bit store: the reader sees the old or the new {slot, state}, never a mix
    *(volatile uint64_t*)word = value;
}

int shrike_residency_set(shrike_moe* m, uint32_t layer, uint32_t expert, uint32_t slot, uint32_t state,
                         void* stream) {
    if (!m || !m->residency) return SHRIKE_EINVAL;
    if (layer >= m->residency_layers || expert >= m->cfg.num_experts)
        return fail(m, SHRIKE_ERANGE, "layer %u / expert %u out of range", layer, expert);
    const uint64_t v = ((uint64_t)state << 32) | slot;
    residency_set_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(
        m->residency + (size_t)layer * m->cfg.num_experts + expert, v);
    CU(cudaGetLastError());
    return SHRIKE_OK;
}

int shrike_residency_set_layer_identity(shrike_moe* m, uint32_t layer, uint32_t first_cell, void* stream) {
    if (!m || !m->residency) return SHRIKE_EINVAL;
    if (layer >= m->residency_layers) return fail(m, SHRIKE_ERANGE, "layer %u out of range", layer);
    residency_identity_kernel<<<1, 256, 0, (cudaStream_t)stream>>>(
        m->residency + (size_t)layer * m->cfg.num_experts, m->cfg.num_experts, first_cell);
    CU(cudaGetLastError());
    return SHRIKE_OK;
}

// ---- the path -------------------------------------------------------------------

// Argument checks shared by the router entry points: operands, counts, stride, alignment.
static int check_router_call(shrike_moe* m, const shrike_router_operands* ops, const void* hidden,
                             uint32_t query_count, uint32_t limit, uint32_t hidden_stride_elements,
                             bool need_gate_out, const void* out_shared_gate) {
    const shrike_moe_config& c = m->cfg;
    if (!ops || !ops->weights || !hidden) return fail(m, SHRIKE_EINVAL, "router: null operand");
    if (c.router_weight_bits != 0 && (!ops->scales || !ops->biases))
        return fail(m, SHRIKE_EINVAL, "router: affine weights need scales and biases");
    if (query_count > limit) return fail(m, SHRIKE_ERANGE, "query_count %u exceeds %u", query_count, limit);
    if (hidden_stride_elements < c.d || hidden_stride_elements % 4 != 0)
        return fail(m, SHRIKE_EINVAL, "hidden stride must be >= d and a multiple of 4 elements");
    if (c.shared_gated && (!ops->shared_gate || (need_gate_out && !out_shared_gate)))
        return fail(m, SHRIKE_EINVAL, "router: a shared_gated handle needs shared_gate and out_shared_gate");
    const char* why = nullptr;
    if (!router_operands_aligned(c, *ops, hidden, &why)) return fail(m, SHRIKE_EINVAL, "router: %s", why);
    return SHRIKE_OK;
}

int shrike_encode_router(shrike_moe* m, void* stream, const shrike_router_operands* ops, const void* hidden,
                         uint32_t query_count, uint32_t hidden_stride_elements, uint32_t* out_indices,
                         float* out_weights, float* out_shared_gate) {
    if (!m) return SHRIKE_EINVAL;
    if (query_count == 0) return SHRIKE_OK;
    if (!out_indices || !out_weights) return fail(m, SHRIKE_EINVAL, "router: null operand");
    int rc = check_router_call(m, ops, hidden, query_count, m->cfg.max_tokens, hidden_stride_elements, true,
                               out_shared_gate);
    if (rc) return rc;
    if ((rc = check_device(m))) return rc;
    CU(launch_router(m, (cudaStream_t)stream, *ops, hidden, query_count, hidden_stride_elements, out_indices,
                     out_weights, out_shared_gate));
    return SHRIKE_OK;
}

int shrike_encode_residency_classification(shrike_moe* m, void* stream, const uint32_t* topk_indices,
                                           const uint64_t* residency_table_row, uint32_t query_count,
                                           uint32_t* resolved_slots, uint32_t* counts,
                                           uint32_t* miss_positions, uint32_t* miss_experts) {
    if (!m) return SHRIKE_EINVAL;
    if (!topk_indices || !residency_table_row || !resolved_slots)
        return fail(m, SHRIKE_EINVAL, "classification: null operand");
    if (query_count > m->cfg.max_tokens) return fail(m, SHRIKE_ERANGE, "query_count exceeds max_tokens");
    if (int rc = check_device(m)) return rc;
    if (query_count == 0) {
        if (counts) CU(cudaMemsetAsync(counts, 0, 8, (cudaStream_t)stream));
        return SHRIKE_OK;
    }
    CU(launch_classify(m, (cudaStream_t)stream, topk_indices, residency_table_row, query_count, resolved_slots,
                       counts, miss_positions, miss_experts));
    return SHRIKE_OK;
}

int shrike_encode_decode_plan(shrike_moe* m, void* stream, const shrike_pool* pool,
                              const uint32_t* resolved_slots, const void* x, uint32_t query_count,
                              const uint32_t* io_status) {
    if (!m) return SHRIKE_EINVAL;
    if (!pool || !resolved_slots || !x) return fail(m, SHRIKE_EINVAL, "decode plan: null operand");
    if (query_count == 0 || query_count > SHRIKE_MAX_DECODE_TOKENS || query_count > m->cfg.max_tokens)
        return fail(m, SHRIKE_ERANGE, "decode handles 1..%u rows (max_tokens %u); use the prefill call",
                    SHRIKE_MAX_DECODE_TOKENS, m->cfg.max_tokens);
    if (int rc = check_device(m)) return rc;
    CU(launch_decode_plan(m, (cudaStream_t)stream, resolved_slots, x, query_count, io_status,
                          m->cfg.has_shared != 0, pool->view.cells));
    return SHRIKE_OK;
}

int shrike_encode_phase1(shrike_moe* m, void* stream, const shrike_pool* pool,
                         const shrike_expert_offsets* routed_offsets, const shrike_shared_expert* shared,
                         uint32_t query_count) {
    if (!m) return SHRIKE_EINVAL;
    if (query_count == 0 || query_count > SHRIKE_MAX_DECODE_TOKENS || query_count > m->cfg.max_tokens)
        return fail(m, SHRIKE_ERANGE, "phase 1: query_count out of range");
    ExpertArgs a;
    int rc = fill_expert_args(m, pool, routed_offsets, shared, nullptr, nullptr, a, false);
    if (rc) return rc;
    if ((rc = check_device(m))) return rc;
    CU(launch_experts(m, (cudaStream_t)stream, a, query_count, 1u, nullptr, nullptr, false));
    return SHRIKE_OK;
}

int shrike_encode_phase2_reduce(shrike_moe* m, void* stream, const shrike_pool* pool,
                                const shrike_expert_offsets* routed_offsets, const float* routing_weights,
                                const shrike_shared_expert* shared, const float* shared_gate,
                                uint32_t query_count, void* y, void* hidden) {
    if (!m) return SHRIKE_EINVAL;
    if (!routing_weights || !y) return fail(m, SHRIKE_EINVAL, "phase 2: null operand");
    if (query_count == 0 || query_count > SHRIKE_MAX_DECODE_TOKENS || query_count > m->cfg.max_tokens)
        return fail(m, SHRIKE_ERANGE, "phase 2: query_count out of range");
    ExpertArgs a;
    int rc = fill_expert_args(m, pool, routed_offsets, shared, routing_weights, shared_gate, a, true);
    if (rc) return rc;
    if ((rc = check_device(m))) return rc;
    CU(launch_experts(m, (cudaStream_t)stream, a, query_count, 2u, y, hidden, false));
    return SHRIKE_OK;
}

int shrike_encode_moe_decode(shrike_moe* m, void* stream, const shrike_pool* pool,
                             const shrike_expert_offsets* routed_offsets, const uint32_t* resolved_slots,
                             const float* routing_weights, const void* x, uint32_t query_count,
                             const shrike_shared_expert* shared, const float* shared_gate,
                             const uint32_t* io_status, void* y, void* hidden) {
    if (!m) return SHRIKE_EINVAL;
    if (query_count == 0) return SHRIKE_OK;
    if (!resolved_slots || !routing_weights || !x || !y) return fail(m, SHRIKE_EINVAL, "decode: null operand");
    int rc = shrike_encode_decode_plan(m, stream, pool, resolved_slots, x, query_count, io_status);
    if (rc) return rc;
    rc = shrike_encode_phase1(m, stream, pool, routed_offsets, shared, query_count);
    if (rc) return rc;
    return shrike_encode_phase2_reduce(m, stream, pool, routed_offsets, routing_weights, shared, shared_gate,
                                       query_count, y, hidden);
}

int shrike_encode_route_decode(shrike_moe* m, void* stream, const shrike_router_operands* ops,
                               const uint64_t* residency_table_row, const shrike_pool* pool,
                               const void* hidden, uint32_t query_count, uint32_t hidden_stride_elements,
                               const uint32_t* io_status, uint32_t* out_indices, float* out_weights,
                               float* out_shared_gate, uint32_t* out_resolved_slots, uint32_t* out_counts) {
    if (!m) return SHRIKE_EINVAL;
    if (query_count == 0) return SHRIKE_OK;
    if (!out_indices || !out_weights || !residency_table_row || !pool)
        return fail(m, SHRIKE_EINVAL, "route_decode: null operand");
    const uint32_t limit = m->cfg.max_tokens < SHRIKE_MAX_DECODE_TOKENS ? m->cfg.max_tokens : SHRIKE_MAX_DECODE_TOKENS;
    int rc = check_router_call(m, ops, hidden, query_count, limit, hidden_stride_elements, true, out_shared_gate);
    if (rc) return rc;
    if ((rc = check_device(m))) return rc;
    CU(launch_route_fused(m, (cudaStream_t)stream, *ops, hidden, query_count, hidden_stride_elements,
                          residency_table_row, pool->view.cells, io_status, out_indices, out_weights,
                          out_shared_gate, out_resolved_slots, out_counts, !m->no_pdl));
    return SHRIKE_OK;
}

int shrike_encode_decode_layer(shrike_moe* m, void* stream, const shrike_pool* pool,
                               const shrike_expert_offsets* routed_offsets,
                               const uint64_t* residency_table_row, const shrike_router_operands* router,
                               const shrike_shared_expert* shared, const void* x, uint32_t query_count,
                               const uint32_t* io_status, uint32_t* out_indices, float* out_weights, void* y,
                               void* hidden) {
    if (!m) return SHRIKE_EINVAL;
    if (query_count == 0) return SHRIKE_OK;
    if (!x || !y) return fail(m, SHRIKE_EINVAL, "decode_layer: null operand");
    Workspace& w = m->ws;
    uint32_t* ids = out_indices ? out_indices : w.ids_dev;
    float* wt = out_weights ? out_weights : w.w_dev;
    float* gate = m->cfg.shared_gated ? w.gate_dev : nullptr;
    if (query_count == 1 && w.fused_geom) {
        // one row: router, selection, lookup, both projections and the combine in ONE launch (fused_layer.cu)
        if (!residency_table_row || !pool) return fail(m, SHRIKE_EINVAL, "decode_layer: null operand");
        int rcf = check_router_call(m, router, x, 1, 1, m->cfg.d, false, nullptr);
        if (rcf) return rcf;
        if (!aligned_to(y, 16) || (hidden && !aligned_to(hidden, 16)))
            return fail(m, SHRIKE_EINVAL, "decode_layer: y and hidden must be 16-byte aligned");
        ExpertArgs ea;
        rcf = fill_expert_args(m, pool, routed_offsets, shared, wt, gate, ea);
        if (rcf) return rcf;
        if ((rcf = check_device(m))) return rcf;
        const cudaError_t fe = launch_fused_layer(m, (cudaStream_t)stream, ea, *router, residency_table_row,
                                                  pool->view.cells, io_status, x, ids, wt, w.slots_dev, gate, y, hidden);
        if (fe == cudaSuccess) return SHRIKE_OK;
        if (fe != cudaErrorNotSupported) return cuda_fail(m, fe, "launch_fused_layer");
        // a block layout the tiled copies cannot describe: the three launches below
    }
    if (stream_pays(query_count)) {
        // some rows: the same in one launch of the streaming kernel (expert_stream.cu). In three launches the last
        // block of the router ranked every row while the others' SMs idled (8 us of 4 rows' 43, 20 of 16 rows' 92), and
        // the next launch began 3 us later.
        if (!residency_table_row || !pool) return fail(m, SHRIKE_EINVAL, "decode_layer: null operand");
        const uint32_t limit = m->cfg.max_tokens < SHRIKE_MAX_DECODE_TOKENS ? m->cfg.max_tokens : SHRIKE_MAX_DECODE_TOKENS;
        int rcs = check_router_call(m, router, x, query_count, limit, m->cfg.d, false, nullptr);
        if (rcs) return rcs;
        ExpertArgs ea;
        rcs = fill_expert_args(m, pool, routed_offsets, shared, wt, gate, ea);
        if (rcs) return rcs;
        if ((rcs = check_device(m))) return rcs;
        RouterArgs ra = make_router_args(m, *router, x, query_count, m->cfg.d, ids, wt, gate);
        ra.table = residency_table_row; ra.pool_cells = pool->view.cells; ra.io_status = io_status;
        ra.with_shared = m->cfg.has_shared; ra.int4 = m->cfg.weight_bits == 4; ra.group = m->cfg.group_size;
        ra.slots = w.slots_dev; ra.xh = w.xh; ra.xsum = w.xsum; ra.status = w.status;
        const cudaError_t se = launch_expert_stream(m, (cudaStream_t)stream, ea, query_count, m->cfg.has_shared ? (query_count + 7) / 8 : 0,
                                                    y, hidden, !m->no_pdl, 3u, &ra);
        if (se == cudaSuccess) return SHRIKE_OK;
        if (se != cudaErrorNotSupported) return cuda_fail(m, se, "launch_expert_stream");
    }
    // Shapes that the streaming kernel does not take, with many rows, on a handle that owns the prefill operands: the
    // expert-grouped GEMM reads every expert once for all its rows, where the 8-row tiles read it once per 8. The dozen
    // launches around it pay from 17 rows on (us a layer, tiles and grouped, odd numbers of groups, picks uniform or by Zipf(1.1);
    // 256 experts of 2048 x 576 int4 | 256 of 2304 x 1088 int8 | 32 of 2880 x 2880 int4 in groups of 64):
    //   17 rows  119, 107 | 209, 198 | 227, 181     Zipf   62, 64 | 160, 155 | 165, 148
    //   32 rows  175, 139 | 286, 250 | 265, 183     Zipf   89, 69 | 205, 176 | 253, 160
    //   48 rows  228, 164 | 349, 286 | 298, 184     Zipf  122, 76 | 255, 187 | 300, 165
    //   64 rows  261, 174 | 399, 308 | 369, 185     Zipf  151, 78 | 305, 200 | 390, 172
    // The line stays: below it a row's sums have a fixed order and its weights are not rounded.
    if (query_count > 48 && w.xs && umma_supported(m->cfg) && !m->force_warp_mma) {
        int rcg = shrike_encode_router(m, stream, router, x, query_count, m->cfg.d, ids, wt, gate);
        if (rcg) return rcg;
        rcg = shrike_encode_residency_classification(m, stream, ids, residency_table_row, query_count, w.slots_dev,
                                                     nullptr, nullptr, nullptr);
        if (rcg) return rcg;
        return encode_prefill(m, stream, pool, routed_offsets, ids, w.slots_dev, wt, x, query_count, shared, gate,
                              io_status, y, hidden);
    }
    int rc = shrike_encode_route_decode(m, stream, router, residency_table_row, pool, x, query_count, m->cfg.d,
                                        io_status, ids, wt, gate, w.slots_dev, nullptr);
    if (rc) return rc;
    ExpertArgs a;
    rc = fill_expert_args(m, pool, routed_offsets, shared, wt, gate, a);
    if (rc) return rc;
    // the expert kernels may start before their predecessor has drained
    CU(launch_experts(m, (cudaStream_t)stream, a, query_count, 3u, y, hidden, !m->no_pdl));
    return SHRIKE_OK;
}

int shrike_encode_moe_prefill(shrike_moe* m, void* stream, const shrike_pool* pool,
                              const shrike_expert_offsets* routed_offsets, const uint32_t* topk_indices,
                              const uint32_t* resolved_slots, const float* routing_weights, const void* x,
                              uint32_t query_count, const shrike_shared_expert* shared,
                              const float* shared_gate, void* y, void* hidden) {
    return encode_prefill(m, stream, pool, routed_offsets, topk_indices, resolved_slots, routing_weights, x,
                          query_count, shared, shared_gate, nullptr, y, hidden);
}

int shrike_encode_group_pairs(shrike_moe* m, void* stream, const uint32_t* topk_indices,
                              const float* routing_weights, uint32_t query_count, uint32_t* sorted_pairs,
                              uint32_t* per_expert_offsets, uint32_t* per_expert_counts) {
    if (!m) return SHRIKE_EINVAL;
    if (!topk_indices || !sorted_pairs || !per_expert_offsets || !per_expert_counts)
        return fail(m, SHRIKE_EINVAL, "group_pairs: null operand");
    if (query_count > m->cfg.max_tokens) return fail(m, SHRIKE_ERANGE, "query_count exceeds max_tokens");
    CU(launch_group_pairs(m, (cudaStream_t)stream, topk_indices, routing_weights, query_count, sorted_pairs,
                          per_expert_offsets, per_expert_counts));
    return SHRIKE_OK;
}

// ---- expert parallelism ---------------------------------------------------------

int shrike_ep_encode_dispatch(shrike_moe* m, void* stream, const void* x, const uint32_t* topk_indices,
                              const float* routing_weights, uint32_t query_count, uint32_t world,
                              uint32_t experts_per_rank, uint32_t capacity_rows, void* send_x, uint32_t* send_ids,
                              float* send_weights, uint32_t* send_counts, int32_t* row_of) {
    if (!m) return SHRIKE_EINVAL;
    if (!x || !topk_indices || !routing_weights || !send_x || !send_ids || !send_weights || !send_counts || !row_of)
        return fail(m, SHRIKE_EINVAL, "ep dispatch: null operand");
    if (world == 0 || world > 64 || experts_per_rank == 0 || (uint64_t)world * experts_per_rank < m->cfg.num_experts)
        return fail(m, SHRIKE_EINVAL, "ep dispatch: world x experts_per_rank must cover num_experts");
    if (query_count > m->cfg.max_tokens) return fail(m, SHRIKE_ERANGE, "query_count exceeds max_tokens");
    if (capacity_rows < query_count)
        return fail(m, SHRIKE_ERANGE, "ep dispatch: capacity_rows must be at least query_count (a row goes to a rank at most once)");
    if (query_count == 0) {
        CU(cudaMemsetAsync(send_counts, 0, world * 4, (cudaStream_t)stream));
        return SHRIKE_OK;
    }
    CU(launch_ep_dispatch(m, (cudaStream_t)stream, x, topk_indices, routing_weights, query_count, world,
                          experts_per_rank, capacity_rows, send_x, send_ids, send_weights, send_counts, row_of));
    return SHRIKE_OK;
}

int shrike_ep_encode_local_slots(shrike_moe* m, void* stream, const uint32_t* recv_ids,
                                 const uint64_t* residency_table_row, uint32_t rows, uint32_t* resolved_slots) {
    if (!m) return SHRIKE_EINVAL;
    if (!recv_ids || !residency_table_row || !resolved_slots) return fail(m, SHRIKE_EINVAL, "ep local slots: null operand");
    if (rows == 0) return SHRIKE_OK;
    CU(launch_ep_local_slots(m, (cudaStream_t)stream, recv_ids, residency_table_row, rows, resolved_slots));
    return SHRIKE_OK;
}

int shrike_ep_encode_combine(shrike_moe* m, void* stream, const void* recv_y, const int32_t* row_of,
                             const void* y_home, uint32_t query_count, uint32_t world, uint32_t capacity_rows,
                             void* y, void* hidden) {
    if (!m) return SHRIKE_EINVAL;
    if (!recv_y || !row_of || !y) return fail(m, SHRIKE_EINVAL, "ep combine: null operand");
    if (query_count == 0) return SHRIKE_OK;
    CU(launch_ep_combine(m, (cudaStream_t)stream, recv_y, row_of, y_home, query_count, world, capacity_rows, y,
                         hidden));
    return SHRIKE_OK;
}

int shrike_moe_layer_forward_host(shrike_moe* m, void* stream, const shrike_pool* pool,
                                  const shrike_expert_offsets* routed_offsets,
                                  const uint64_t* residency_table_row, const shrike_router_operands* router,
                                  const shrike_shared_expert* shared, const void* x_host,
                                  uint32_t query_count, void* y_host, uint32_t* ids_host, float* weights_host) {
    if (!m) return SHRIKE_EINVAL;
    if (!x_host || !y_host || !router || !residency_table_row) return fail(m, SHRIKE_EINVAL, "forward_host: null operand");
    const shrike_moe_config& c = m->cfg;
    if (query_count == 0) return SHRIKE_OK;
    if (query_count > c.max_tokens) return fail(m, SHRIKE_ERANGE, "query_count exceeds max_tokens");
    cudaStream_t st = (cudaStream_t)stream;
    Workspace& w = m->ws;
    const size_t elements = (size_t)query_count * c.d;
    CU(cudaMemcpyAsync(w.x_dev, x_host, elements * act_bytes(c.act_dtype), cudaMemcpyHostToDevice, st));
    float* gate = c.shared_gated ? w.gate_dev : nullptr;
    int rc;
    if (query_count <= SHRIKE_MAX_DECODE_TOKENS) {
        rc = shrike_encode_decode_layer(m, stream, pool, routed_offsets, residency_table_row, router, shared,
                                        w.x_dev, query_count, nullptr, w.ids_dev, w.w_dev, w.y_dev, nullptr);
    } else {
        rc = shrike_encode_router(m, stream, router, w.x_dev, query_count, c.d, w.ids_dev, w.w_dev, gate);
        if (rc) return rc;
        rc = shrike_encode_residency_classification(m, stream, w.ids_dev, residency_table_row, query_count,
                                                    w.slots_dev, w.counts_dev, nullptr, nullptr);
        if (rc) return rc;
        rc = shrike_encode_moe_prefill(m, stream, pool, routed_offsets, w.ids_dev, w.slots_dev, w.w_dev, w.x_dev,
                                       query_count, shared, gate, w.y_dev, nullptr);
    }
    if (rc) return rc;
    CU(cudaMemcpyAsync(y_host, w.y_dev, elements * act_bytes(c.y_dtype), cudaMemcpyDeviceToHost, st));
    if (ids_host) CU(cudaMemcpyAsync(ids_host, w.ids_dev, (size_t)query_count * c.top_k * 4, cudaMemcpyDeviceToHost, st));
    if (weights_host) CU(cudaMemcpyAsync(weights_host, w.w_dev, (size_t)query_count * c.top_k * 4, cudaMemcpyDeviceToHost, st));
    return shrike_moe_status(m, stream);
}

int shrike_dequant_affine_rows(void* stream, const void* packed, const void* scales, const void* biases,
                               uint32_t bits, uint32_t group, uint32_t meta_dtype, uint32_t rows, uint32_t cols,
                               float* out) {
    if (!packed || !scales || !biases || !out) return SHRIKE_EINVAL;
    if ((bits != 4 && bits != 8) || (group != 32 && group != 64) || cols == 0 || cols % group != 0 ||
        (meta_dtype != SHRIKE_DTYPE_BF16 && meta_dtype != SHRIKE_DTYPE_FP16))
        return SHRIKE_EINVAL;
    if (((uintptr_t)scales & 1) || ((uintptr_t)biases & 1) || ((uintptr_t)out & 3)) return SHRIKE_EINVAL;
    if (rows == 0) return SHRIKE_OK;
    if ((uint64_t)rows * cols > 0x7fffffffull * 256) return SHRIKE_ERANGE;
    return launch_dequant_affine_rows((cudaStream_t)stream, packed, scales, biases, bits, group, meta_dtype, rows, cols,
                                      out) == cudaSuccess ? SHRIKE_OK : SHRIKE_EIO;
}

// ---- expert parallelism over peer memory ---------------------------------------------------------------

struct shrike_ep {
    shrike_moe* home;
    shrike_moe* routed;
    uint32_t rank, world, cap, epr, t_max;
    EpLayout lay;
    uint8_t* mine = nullptr;
    uint8_t* peer[SHRIKE_EP_MAX_WORLD] = {};
    bool opened[SHRIKE_EP_MAX_WORLD] = {};
    bool connected = false;
    // local scratch
    uint32_t* ids = nullptr; float* w = nullptr; float* gate = nullptr; int32_t* row_of = nullptr;
    uint32_t* send_counts = nullptr; uint32_t* miss_slots = nullptr;
    uint32_t* c_ids = nullptr; float* c_w = nullptr; uint32_t* c_slots = nullptr; uint32_t* row_map = nullptr;
    uint32_t* prefix = nullptr; uint32_t* n_rows = nullptr;
    void* y_home = nullptr;
    cudaStream_t side = nullptr;
    cudaEvent_t ev_routed = nullptr, ev_shared = nullptr;
    uint32_t epoch = 0;
    uint32_t max_polls = 1000000;   // ~1 us per poll
};

static void ep_free(shrike_ep* ep) {
    for (uint32_t g = 0; g < SHRIKE_EP_MAX_WORLD; ++g)
        if (ep->opened[g] && ep->peer[g]) cudaIpcCloseMemHandle(ep->peer[g]);
    void* ptrs[] = {ep->mine, ep->ids, ep->w, ep->gate, ep->row_of, ep->send_counts, ep->miss_slots, ep->c_ids, ep->c_w,
                    ep->c_slots, ep->row_map, ep->prefix, ep->n_rows, ep->y_home};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    if (ep->side) cudaStreamDestroy(ep->side);
    if (ep->ev_routed) cudaEventDestroy(ep->ev_routed);
    if (ep->ev_shared) cudaEventDestroy(ep->ev_shared);
    delete ep;
}

int shrike_ep_create(shrike_moe* home, shrike_moe* routed, uint32_t rank, uint32_t world, uint32_t rows_per_call,
                     shrike_ep** out) {
    if (!home || !routed || !out) return SHRIKE_EINVAL;
    shrike_moe* m = home;
    *out = nullptr;
    const shrike_moe_config& c = home->cfg;
    const shrike_moe_config& r = routed->cfg;
    if (world == 0 || world > SHRIKE_EP_MAX_WORLD || rank >= world)
        return fail(m, SHRIKE_EINVAL, "ep: world must be 1..%u and rank below it", SHRIKE_EP_MAX_WORLD);
    if (c.num_experts % world != 0 || r.num_experts != c.num_experts / world)
        return fail(m, SHRIKE_EINVAL, "ep: the routed handle must hold num_experts / world experts");
    // weight_bits, group_size and meta_dtype may differ: the home handle's describe the shared expert's block, the
    // routed handle's the routed experts' (an int8 shared expert beside int4 routed experts,
    // SharedExpertInt8.swift:55-227)
    if (r.d != c.d || r.f != c.f || r.top_k != c.top_k || r.act_dtype != c.act_dtype || r.y_dtype != c.y_dtype ||
        r.activation != c.activation || r.expert_bias != c.expert_bias || r.has_shared || home->device != routed->device)
        return fail(m, SHRIKE_EINVAL, "ep: the routed handle must share the layer's shape, dtypes and device and have no shared expert");
    if ((r.weight_bits != c.weight_bits || r.group_size != c.group_size || r.meta_dtype != c.meta_dtype) && !c.has_shared)
        return fail(m, SHRIKE_EINVAL, "ep: the handles' weight formats differ but the home handle has no shared expert to describe");
    if (rows_per_call == 0 || rows_per_call > c.max_tokens)
        return fail(m, SHRIKE_ERANGE, "ep: rows_per_call must be 1..max_tokens of the home handle");
    const uint32_t t_max = world * rows_per_call;
    if (r.max_tokens < t_max || r.max_tokens <= SHRIKE_MAX_DECODE_TOKENS)
        return fail(m, SHRIKE_ERANGE, "ep: the routed handle needs max_tokens >= max(65, world * rows_per_call)");
    DeviceGuard guard(home->device);
    shrike_ep* ep = new (std::nothrow) shrike_ep();
    if (!ep) return fail(m, SHRIKE_ENOMEM, "host allocation failed");
    ep->home = home; ep->routed = routed; ep->rank = rank; ep->world = world; ep->cap = rows_per_call;
    ep->epr = r.num_experts; ep->t_max = t_max;
    ep->lay = ep_layout(c, world, rows_per_call);
    const size_t T = rows_per_call, K = c.top_k;
    bool ok = true;
    auto A = [&](auto** p, size_t bytes) { if (ok && cudaMalloc((void**)p, bytes ? bytes : 16) != cudaSuccess) ok = false; };
    A(&ep->mine, ep->lay.bytes);
    A(&ep->ids, T * K * 4); A(&ep->w, T * K * 4); A(&ep->gate, T * 4); A(&ep->row_of, T * world * 4);
    A(&ep->send_counts, SHRIKE_EP_MAX_WORLD * 4); A(&ep->miss_slots, T * K * 4);
    A(&ep->c_ids, (size_t)t_max * K * 4); A(&ep->c_w, (size_t)t_max * K * 4); A(&ep->c_slots, (size_t)t_max * K * 4);
    A(&ep->row_map, (size_t)t_max * 4); A(&ep->prefix, (SHRIKE_EP_MAX_WORLD + 1) * 4); A(&ep->n_rows, 4);
    A((uint8_t**)&ep->y_home, c.has_shared ? T * c.d * act_bytes(c.y_dtype) : 0);
    if (ok && (cudaStreamCreateWithFlags(&ep->side, cudaStreamNonBlocking) != cudaSuccess ||
               cudaEventCreateWithFlags(&ep->ev_routed, cudaEventDisableTiming) != cudaSuccess ||
               cudaEventCreateWithFlags(&ep->ev_shared, cudaEventDisableTiming) != cudaSuccess))
        ok = false;
    if (!ok) {
        ep_free(ep);
        cudaGetLastError();
        return fail(m, SHRIKE_ENOMEM, "ep: allocation of the exchange buffers failed");
    }
    // no arrival word carries the first epoch's tag; the shared-only call of the home rows sees every pick miss
    cudaError_t se = cudaMemset(ep->mine, 0, ep->lay.bytes);
    if (se == cudaSuccess) se = set_now(ep->miss_slots, 0xff, T * K * 4);
    if (se != cudaSuccess) {
        ep_free(ep);
        return cuda_fail(m, se, "ep: clearing the exchange buffers");
    }
    ep->peer[rank] = ep->mine;
    ep->connected = world == 1;
    *out = ep;
    return SHRIKE_OK;
}

void shrike_ep_destroy(shrike_ep* ep) {
    if (!ep) return;
    DeviceGuard guard(ep->home->device);
    cudaDeviceSynchronize();
    ep_free(ep);
}

int shrike_ep_export(shrike_ep* ep, void* handle_out) {
    if (!ep || !handle_out) return SHRIKE_EINVAL;
    shrike_moe* m = ep->home;
    static_assert(sizeof(cudaIpcMemHandle_t) == SHRIKE_EP_HANDLE_BYTES, "token size");
    DeviceGuard guard(m->device);
    cudaIpcMemHandle_t h;
    CU(cudaIpcGetMemHandle(&h, ep->mine));
    memcpy(handle_out, &h, sizeof h);
    return SHRIKE_OK;
}

int shrike_ep_connect(shrike_ep* ep, const void* all_handles) {
    if (!ep || !all_handles) return SHRIKE_EINVAL;
    shrike_moe* m = ep->home;
    DeviceGuard guard(m->device);
    for (uint32_t g = 0; g < ep->world; ++g) {
        if (g == ep->rank || ep->peer[g]) continue;
        cudaIpcMemHandle_t h;
        memcpy(&h, (const uint8_t*)all_handles + (size_t)g * SHRIKE_EP_HANDLE_BYTES, sizeof h);
        void* p = nullptr;
        CU(cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess));
        ep->peer[g] = (uint8_t*)p;
        ep->opened[g] = true;
    }
    ep->connected = true;
    return SHRIKE_OK;
}

int shrike_ep_buffer(shrike_ep* ep, void** base_out, uint64_t* bytes_out) {
    if (!ep || !base_out) return SHRIKE_EINVAL;
    *base_out = ep->mine;
    if (bytes_out) *bytes_out = ep->lay.bytes;
    return SHRIKE_OK;
}

int shrike_ep_connect_pointers(shrike_ep* ep, void* const* peer_bases) {
    if (!ep || !peer_bases) return SHRIKE_EINVAL;
    for (uint32_t g = 0; g < ep->world; ++g) {
        if (g == ep->rank) continue;
        if (!peer_bases[g]) return fail(ep->home, SHRIKE_EINVAL, "ep: peer %u has no buffer", g);
        ep->peer[g] = (uint8_t*)peer_bases[g];
    }
    ep->connected = true;
    return SHRIKE_OK;
}

int shrike_ep_set_wait_polls(shrike_ep* ep, uint32_t wait_polls) {
    if (!ep) return SHRIKE_EINVAL;
    ep->max_polls = wait_polls ? wait_polls : 1000000;
    return SHRIKE_OK;
}

// Whether a forward has nobody to exchange rows with and can be the home handle's own layer call, which knows the number of its rows
// on the host, keeps them where they are and runs on one stream. What that call does not take goes the general way: formats of the
// routed experts that the home handle does not describe, one row whose y or hidden is not 16-byte aligned, y across x. Through the
// exchange buffer, in some twenty launches, and as the layer call, calls one after the other, us: 256 experts of 2048 x 512 int4, 4 rows 104 / 34; 32 of
// 2880 x 2880 int4, 3 rows 152 / 72, 144 rows 248 / 195; 256 of 2304 x 1024 int8, 39 rows 318 / 195, 2064 rows 662 / 613.
// Nor is it taken where up to 64 rows of nibbles would lose by it. The decode kernels sum (1024 + q) x, or (64 + q) x of every second nibble, and
// take the offset's share away again: behind a clamped SwiGLU, whose products are of one sign, in groups of 64 or all with 1024 (the
// per-tile kernels) they are further off than the grouped GEMM that the exchange's experts run on. Error against 64 bits, bf16 scales, GEMM and
// decode kernels: 32 experts of 2880 x 2880, odd groups of 64, 1 row 7.3e-5 and 1.0e-4 (one launch), 17 rows 6.4e-5 and 1.5e-4 (per tile); 256 of 2048 x 512, groups of
// 64, 8.5e-5 and 1.3e-4. In groups of 32 it is 6.1e-5 and 7.2e-5, 1.4e-4 and 1.1e-4 with fp16 scales; behind SiLU 2.0e-4 and 2.1e-4; of bytes 4.1e-4 and 2.1e-4. And from
// 49 rows on the per-tile kernels are the slower ones, us: 32 experts of 2880 x 2880 in groups of 64, 64 rows 235 by the exchange and 367 by
// the layer call, 256 of 2048 x 576 240 and 258.
static bool ep_alone(const shrike_ep* ep, uint32_t T, const void* x, const void* y, const void* hidden) {
    const shrike_moe_config &c = ep->home->cfg, &r = ep->routed->cfg;
    if (ep->world != 1 || T == 0 || r.weight_bits != c.weight_bits || r.group_size != c.group_size || r.meta_dtype != c.meta_dtype) return false;
    if (T == 1 && (!aligned_to(y, 16) || !aligned_to(hidden, 16))) return false;
    const bool gemm = umma_supported(c) && !ep->routed->force_warp_mma;   // what the exchange's experts run on
    const bool tiles = !(T == 1 ? ep->home->ws.fused_geom != nullptr : stream_takes_shape(ep->home));
    if (gemm && c.weight_bits == 4 && T <= SHRIKE_MAX_DECODE_TOKENS && !(tiles && T > 48 && ep->home->ws.xs) &&
        ((tiles && T > 48) || (c.activation == SHRIKE_ACT_CLAMPED_SWIGLU && (tiles || c.group_size == 64))))
        return false;
    const uintptr_t x0 = (uintptr_t)x, y0 = (uintptr_t)y, elems = (uintptr_t)T * c.d;
    return x0 == y0 || x0 + elems * act_bytes(c.act_dtype) <= y0 || y0 + elems * act_bytes(c.y_dtype) <= x0;
}

static int ep_forward_alone(shrike_ep* ep, void* stream, const shrike_pool* pool, const shrike_expert_offsets* routed_offsets,
                            const uint64_t* residency_row, const shrike_router_operands* router, const shrike_shared_expert* shared,
                            const void* x, uint32_t T, void* y, void* hidden) {
    shrike_moe* m = ep->home;
    int rc;
    if (T <= SHRIKE_MAX_DECODE_TOKENS) {
        rc = shrike_encode_decode_layer(m, stream, pool, routed_offsets, residency_row, router, shared, x, T, nullptr, ep->ids, ep->w, y, hidden);
    } else {
        float* gate = m->cfg.shared_gated ? ep->gate : nullptr;
        rc = shrike_encode_router(m, stream, router, x, T, m->cfg.d, ep->ids, ep->w, gate);
        if (!rc) rc = shrike_encode_residency_classification(m, stream, ep->ids, residency_row, T, ep->c_slots, nullptr, nullptr, nullptr);
        if (!rc) rc = encode_prefill(m, stream, pool, routed_offsets, ep->ids, ep->c_slots, ep->w, x, T, shared, gate, nullptr, y, hidden);
    }
    if (rc) return rc;
    CU(launch_ep_alone_counts(m, (cudaStream_t)stream, T, ep->send_counts, ep->prefix, ep->n_rows));
    return SHRIKE_OK;
}

int shrike_ep_forward(shrike_ep* ep, void* stream, const shrike_pool* local_pool,
                      const shrike_expert_offsets* routed_offsets, const uint64_t* local_residency_row,
                      const shrike_router_operands* router, const shrike_shared_expert* shared, const void* x,
                      uint32_t query_count, void* y, void* hidden) {
    if (!ep) return SHRIKE_EINVAL;
    shrike_moe* m = ep->home;
    shrike_moe* r = ep->routed;
    if (!ep->connected) return fail(m, SHRIKE_EINVAL, "ep: connect the ranks' buffers first");
    if (!local_pool || !routed_offsets || !local_residency_row || !router || !y || (query_count && !x))
        return fail(m, SHRIKE_EINVAL, "ep forward: null operand");
    if (query_count > ep->cap) return fail(m, SHRIKE_ERANGE, "ep forward: query_count exceeds rows_per_call");
    const shrike_moe_config& c = m->cfg;
    cudaStream_t st = (cudaStream_t)stream;
    int rc;
    if ((rc = check_device(m))) return rc;
    if (ep_alone(ep, query_count, x, y, hidden))
        return ep_forward_alone(ep, stream, local_pool, routed_offsets, local_residency_row, router, shared, x, query_count, y, hidden);
    // the call's two streams run beside each other; outside of it the handles launch as any other
    struct Beside {
        shrike_moe *a, *b;
        Beside(shrike_moe* a, shrike_moe* b) : a(a), b(b) { a->beside_others = b->beside_others = true; }
        ~Beside() { a->beside_others = b->beside_others = false; }
    } beside(m, r);
    const uint32_t epoch = ++ep->epoch;
    const uint32_t T = query_count;
    float* gate = c.shared_gated ? ep->gate : nullptr;
    if (T) {
        rc = shrike_encode_router(m, stream, router, x, T, c.d, ep->ids, ep->w, gate);
        if (rc) return rc;
    }
    // the shared expert of the home rows depends on the router's gate only: second stream, beside the exchange
    const bool with_shared = c.has_shared && T > 0;
    if (with_shared) {
        CU(cudaEventRecord(ep->ev_routed, st));
        CU(cudaStreamWaitEvent(ep->side, ep->ev_routed, 0));
        if (T <= SHRIKE_MAX_DECODE_TOKENS)
            rc = shrike_encode_moe_decode(m, ep->side, local_pool, routed_offsets, ep->miss_slots, ep->w, x, T, shared, gate,
                                          nullptr, ep->y_home, nullptr);
        else
            rc = encode_prefill(m, ep->side, local_pool, routed_offsets, ep->ids, ep->miss_slots, ep->w, x, T, shared, gate,
                                nullptr, ep->y_home, nullptr);
        if (rc) return rc;
        CU(cudaEventRecord(ep->ev_shared, ep->side));
    }
    CU(launch_ep_dispatch_peer(m, st, x, ep->ids, ep->w, T, ep->world, ep->rank, ep->epr, ep->cap, ep->peer, ep->lay, epoch,
                               ep->send_counts, ep->row_of));
    CU(launch_ep_receive(r, st, ep->mine, ep->lay, ep->world, ep->cap, epoch, local_residency_row, ep->t_max, ep->prefix,
                         ep->n_rows, ep->c_ids, ep->c_w, ep->c_slots, ep->row_map, ep->max_polls));
    {   // local experts on the received rows (read in place through the row map), accumulated per row
        ExpertArgs a;
        rc = fill_expert_args(r, local_pool, routed_offsets, nullptr, ep->c_w, nullptr, a);
        if (rc) return pass_on(m, r, rc);
        const bool warp_mma = r->force_warp_mma || !umma_supported(r->cfg);
        CU(launch_prefill_plan(r, st, ep->c_ids, ep->c_slots, ep->mine + ep->lay.off_recv_x, ep->t_max, false,
                               local_pool->view.cells, warp_mma, nullptr, ep->row_map, ep->n_rows));
        if (warp_mma) {
            const uint32_t mi = max_instances(r->cfg, ep->t_max);
            CU(launch_phase1(r, st, a, mi, false));
            CU(launch_phase2_accumulate(r, st, a, mi));
        } else {
            CU(launch_umma_prefill(r, st, a, ep->t_max));
        }
    }
    CU(launch_ep_return(r, st, ep->row_map, ep->n_rows, ep->t_max, ep->world, ep->rank, ep->cap, ep->peer, ep->lay, epoch));
    CU(launch_ep_wait_returns(m, st, ep->mine, ep->lay, ep->world, ep->cap, epoch, ep->max_polls));
    if (with_shared) CU(cudaStreamWaitEvent(st, ep->ev_shared, 0));
    if (T)
        CU(launch_ep_combine(m, st, ep->mine + ep->lay.off_ret, ep->row_of, with_shared ? ep->y_home : nullptr, T, ep->world,
                             ep->cap, y, hidden, r->ws.yacc, ep->prefix, ep->rank));
    return SHRIKE_OK;
}

int shrike_ep_status(shrike_ep* ep, void* stream) {
    if (!ep) return SHRIKE_EINVAL;
    int rc = shrike_moe_status(ep->home, stream);
    const int rc2 = shrike_moe_status(ep->routed, stream);
    if (!rc && rc2) {
        rc = pass_on(ep->home, ep->routed, rc2);
    }
    return rc;
}

int shrike_ep_last_counts(shrike_ep* ep, uint32_t* sent_per_rank, uint32_t* rows_received, uint64_t* bytes_stored) {
    if (!ep) return SHRIKE_EINVAL;
    shrike_moe* m = ep->home;
    uint32_t sent[SHRIKE_EP_MAX_WORLD] = {};
    uint32_t n = 0;
    CU(cudaMemcpy(sent, ep->send_counts, ep->world * 4, cudaMemcpyDeviceToHost));
    CU(cudaMemcpy(&n, ep->n_rows, 4, cudaMemcpyDeviceToHost));
    uint64_t rows_out = 0;
    for (uint32_t g = 0; g < ep->world; ++g) {
        if (sent_per_rank) sent_per_rank[g] = sent[g];
        if (g != ep->rank) rows_out += sent[g];
    }
    if (rows_received) *rows_received = n;
    if (bytes_stored) {
        const shrike_moe_config& c = m->cfg;
        // rows + ids + weights out, partial rows back (the rows this rank received from others), 8-byte words
        uint32_t own = 0;
        uint32_t pre[SHRIKE_EP_MAX_WORLD + 1] = {};
        CU(cudaMemcpy(pre, ep->prefix, (ep->world + 1) * 4, cudaMemcpyDeviceToHost));
        own = pre[ep->rank + 1] - pre[ep->rank];
        *bytes_stored = rows_out * ((uint64_t)c.d * act_bytes(c.act_dtype) + (uint64_t)c.top_k * 8) +
                        (uint64_t)(n - own) * c.d * act_bytes(c.y_dtype) + (uint64_t)(ep->world - 1) * 16;
    }
    return SHRIKE_OK;
}

// What a layer's launches take from its operands: a call whose operands read otherwise does not run the captured ones.
struct StackOperands {
    shrike::PoolView pool;
    shrike_expert_offsets routed;
    shrike_router_operands router;
    shrike_shared_expert shared;
    void read(const shrike_stack_layer& ly) {
        memset(this, 0, sizeof *this);   // (compared as bytes)
        pool = ly.pool->view;
        routed = *ly.routed_offsets;
        router = *ly.router;
        if (ly.shared) shared = *ly.shared;
    }
};

struct shrike_decode_stack {
    shrike_stack_layer* layers = nullptr;
    StackOperands* captured = nullptr;   // [layers], with `graph`
    cudaGraphExec_t graph = nullptr;     // the layer calls for max_rows rows, or NULL
    uint32_t layer_count = 0;
    uint32_t max_rows = 0;
    void* stream_dev = nullptr;   // [(layers + 1) x max_rows x d]
    ~shrike_decode_stack() { delete[] layers; delete[] captured; }
};

// Layer l's call for query_count rows of the stack's stream; a failure's text is on the layer's handle.
static int encode_stack_layer(const shrike_decode_stack* stack, void* stream, uint32_t l, uint32_t query_count) {
    const shrike_stack_layer& ly = stack->layers[l];
    const size_t block = (size_t)query_count * ly.moe->cfg.d * act_bytes(ly.moe->cfg.act_dtype);
    uint8_t* const x = (uint8_t*)stack->stream_dev + (size_t)l * block;
    return shrike_encode_decode_layer(ly.moe, stream, ly.pool, ly.routed_offsets, ly.residency_table_row, ly.router, ly.shared, x,
                                      query_count, nullptr, nullptr, nullptr, ly.moe->ws.y_dev, x + block);
}

// The layer calls of a full step as one graph: a cooperative launch by itself takes 2 to 3 us of a layer's 17, inside a graph nothing.
// A stack whose calls cannot be captured goes on without, and creation, which succeeds all the same, leaves no failure's text behind:
// what a layer call refuses, a forward refuses again.
static void capture_stack(shrike_decode_stack* s) {
    cudaStream_t st;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    s->captured = new (std::nothrow) StackOperands[s->layer_count];
    if (s->captured && cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
        int rc = SHRIKE_OK;
        for (uint32_t l = 0; l < s->layer_count && rc == SHRIKE_OK; ++l) {
            s->captured[l].read(s->layers[l]);
            shrike_moe* const m = s->layers[l].moe;
            char text[kErrorText];
            memcpy(text, m->err, kErrorText);
            rc = encode_stack_layer(s, st, l, s->max_rows);
            if (rc) memcpy(m->err, text, kErrorText);
        }
        cudaGraph_t g = nullptr;
        if (cudaStreamEndCapture(st, &g) == cudaSuccess && g && rc == SHRIKE_OK &&
            (cudaGraphInstantiate(&s->graph, g, 0) != cudaSuccess || cudaGraphUpload(s->graph, st) != cudaSuccess ||
             cudaStreamSynchronize(st) != cudaSuccess)) {
            if (s->graph) cudaGraphExecDestroy(s->graph);
            s->graph = nullptr;
        }
        if (g) cudaGraphDestroy(g);
    }
    cudaStreamDestroy(st);
    cudaGetLastError();
}

// Whether a step of query_count rows is the captured one: as many rows, and every layer's operands read as they did then.
static bool stack_runs_graph(const shrike_decode_stack* s, uint32_t query_count) {
    if (!s->graph || query_count != s->max_rows) return false;
    for (uint32_t l = 0; l < s->layer_count; ++l) {
        StackOperands now;
        now.read(s->layers[l]);
        if (s->layers[l].moe->beside_others || memcmp(&now, &s->captured[l], sizeof now) != 0) return false;
    }
    return true;
}

int shrike_decode_stack_create(const shrike_stack_layer* layers, uint32_t layer_count, uint32_t max_rows,
                               shrike_decode_stack** out) {
    if (!layers || layer_count == 0 || !layers[0].moe || !out) return SHRIKE_EINVAL;
    *out = nullptr;
    shrike_moe* m = layers[0].moe;
    const shrike_moe_config& c = m->cfg;
    if (max_rows == 0 || max_rows > SHRIKE_MAX_DECODE_TOKENS)
        return fail(m, SHRIKE_ERANGE, "decode_stack: max_rows must be 1..%u", SHRIKE_MAX_DECODE_TOKENS);
    for (uint32_t l = 0; l < layer_count; ++l) {
        const shrike_moe* ml = layers[l].moe;
        if (!ml || ml->device != m->device || ml->cfg.d != c.d || ml->cfg.act_dtype != c.act_dtype)
            return fail(m, SHRIKE_EINVAL, "decode_stack: layer %u does not share device, d and act_dtype with layer 0", l);
        if (max_rows > ml->cfg.max_tokens) return fail(m, SHRIKE_ERANGE, "decode_stack: max_rows exceeds layer %u's max_tokens", l);
        if (!layers[l].pool || !layers[l].routed_offsets || !layers[l].residency_table_row || !layers[l].router)
            return fail(m, SHRIKE_EINVAL, "decode_stack: layer %u has a null operand", l);
    }
    DeviceGuard guard(m->device);
    shrike_decode_stack* s = new (std::nothrow) shrike_decode_stack();
    if (!s) return fail(m, SHRIKE_ENOMEM, "host allocation failed");
    s->layers = new (std::nothrow) shrike_stack_layer[layer_count];
    if (!s->layers) {
        delete s;
        return fail(m, SHRIKE_ENOMEM, "host allocation failed");
    }
    std::copy(layers, layers + layer_count, s->layers);
    s->layer_count = layer_count;
    s->max_rows = max_rows;
    const size_t bytes = (size_t)(layer_count + 1) * max_rows * c.d * act_bytes(c.act_dtype);
    if (cudaMalloc(&s->stream_dev, bytes) != cudaSuccess) {
        delete s;
        cudaGetLastError();
        return fail(m, SHRIKE_ENOMEM, "decode_stack: residual stream of %zu bytes", bytes);
    }
    capture_stack(s);
    *out = s;
    return SHRIKE_OK;
}

void shrike_decode_stack_destroy(shrike_decode_stack* stack) {
    if (!stack) return;
    DeviceGuard guard(stack->layers[0].moe->device);
    if (stack->graph) cudaGraphExecDestroy(stack->graph);
    cudaFree(stack->stream_dev);
    delete stack;
}

int shrike_decode_stack_forward_host(shrike_decode_stack* stack, void* stream, const void* rows_host,
                                     uint32_t query_count, void* out_host) {
    if (!stack) return SHRIKE_EINVAL;
    shrike_moe* m = stack->layers[0].moe;
    if (!rows_host || !out_host) return fail(m, SHRIKE_EINVAL, "decode_stack: null operand");
    if (query_count == 0) return SHRIKE_OK;
    if (query_count > stack->max_rows) return fail(m, SHRIKE_ERANGE, "decode_stack: query_count exceeds max_rows");
    const shrike_moe_config& c = m->cfg;
    cudaStream_t st = (cudaStream_t)stream;
    const uint32_t L = stack->layer_count;
    const size_t block = (size_t)query_count * c.d * act_bytes(c.act_dtype);
    uint8_t* dev = (uint8_t*)stack->stream_dev;
    CU(cudaMemcpyAsync(dev, rows_host, (size_t)(L + 1) * block, cudaMemcpyHostToDevice, st));
    int rc;
    if (stack_runs_graph(stack, query_count)) {
        if ((rc = check_device(m))) return rc;
        CU(cudaGraphLaunch(stack->graph, st));
    } else {
        for (uint32_t l = 0; l < L; ++l)
            if ((rc = encode_stack_layer(stack, stream, l, query_count))) return pass_on(m, stack->layers[l].moe, rc);
    }
    CU(cudaMemcpyAsync(out_host, dev + (size_t)L * block, block, cudaMemcpyDeviceToHost, st));
    CU(cudaStreamSynchronize(st));
    return SHRIKE_OK;
}

int shrike_decode_stack_runs_graph(const shrike_decode_stack* stack, uint32_t query_count, int* out) {
    if (!stack || !out) return SHRIKE_EINVAL;
    *out = stack_runs_graph(stack, query_count);
    return SHRIKE_OK;
}

}  // extern "C"
