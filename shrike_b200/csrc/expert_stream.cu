// Expert projections of a few rows per expert at memory speed: gate/up + GLU and down for instances of up to 8
// rows that share an expert block (decode calls of 2 to 64 rows, and the experts with few rows of a prefill).
//
//   phase 1: acts[pair, f] = GLU(gate[f,:].x + b, up[f,:].x + b)
//            (moe_phase1_gate_up_act_spec_u16load, moe.metal:950-998; shared
//            expert: dequant_int4_shared_gate_up_gemv_simd, dequant_int4.metal:206)
//   phase 2: part[pair, d] = w * (down[d,:].acts + b)
//   phase 3: y[t, d] = sum of the row's parts; hidden[t, d] += y[t, d]
//            (moe_phase2_down_reduce_spec_k8 and moe_phase2_finish, moe.metal:889-893, 1008-1057;
//            dequant_int4_shared_down_fused, dequant_int4.metal:247-331)
//
// Every distinct expert block is read once for up to 8 rows, so HBM bounds the work; what has to keep up is the
// instruction stream that unpacks it. Hence:
//   * one persistent block per SM, sixteen multiplying warps and four finishing ones, that walks a contiguous range of
//     units (16 weight rows of one instance: 8 gate + 8 up, or 16 down), so it meets one to three instances. Their
//     activations are laid out once per block in shared memory as the tiles' B operands, with the sums that take the
//     offsets of the unpacked integers (the accumulators' initial values) and the zero points (a k8 tf32 tile over the
//     groups) out;
//   * a unit is one slot of a ring: two tiled TMA copies, the weights as 128-byte pieces of rows. A team of W warps takes a
//     unit, each its share of the pieces; none waits for the others: a warp leaves its partial sums and goes on to the
//     team's next slot. A finishing warp waits for the partial sums, adds them up in warp order, asks for the unit
//     that comes n_slots later and finishes the rows (done by the multiplying warps in turn, the activation function's
//     long chain held up every unit of the team);
//   * the parts of a row are added up in the order of its picks: results do not depend on timing. The experts of a
//     prefill add straight into fp32 rows instead.
// All phases run in one launch when the call has them: a block asks for its first phase-2 units before it waits for
// the other blocks' activations.
//
// Measured (256 experts of 2048 x 512, top 8, int4, 16 rows: 181 MB of expert blocks): both projections 56 us where the
// per-tile kernels took 82; inside the unit loops 6.5 TB/s, the rest is the start (7 us), the hand-over between the
// phases (5 us) and the last one (3 us).
#include "block_maps.cuh"
#include "tile_math.cuh"

#include <algorithm>
#include <type_traits>

namespace shrike {

namespace {

constexpr uint32_t kWarps = 16, kFinish = 4;         // multiplying and finishing warps
constexpr uint32_t kThreads = (kWarps + kFinish) * 32;
constexpr uint32_t kMaxSlots = 32, kMaxSlots2 = 64;
constexpr uint32_t kRedCol = 20;                     // floats per column of a warp's partial sums (16 + padding)
constexpr uint32_t kRedWarp = 8 * kRedCol;

}  // namespace

// Shared memory: [instance buffers][partial sums][ring]. An instance buffer holds the B operands of the instance's rows
// (columns; lanes past the count read the last one's), per four groups their sums as tf32 operands, and per group
// the accumulators' initial values. Buffers are packed: most instances of a decode call have one or two rows.
struct StreamGeom {
    uint32_t meta_off, ab_off, slot_bytes, n_slots, w1;   // phase 1: scales/biases and additive biases in a slot; warps of a team
    uint32_t ab_off2[2], w_bytes2, m_bytes2, n_slots2, w2;   // phase 2, [0] routed, [1] shared; [slot] weights, then [slot] the rest
    uint32_t off_red, off_ring, smem_bytes;
};

struct StreamArgs {
    PoolView pool;
    Offsets3 routed, shared;
    const uint8_t* shared_block;
    uint32_t d, f, f_shared, top_k, activation, expert_bias, act_dtype, y_dtype;
    const Instance* inst;
    const uint32_t* n_inst;
    uint32_t n_shared;                               // the list's first n_shared instances are the shared expert's
    const uint16_t* xh;
    uint16_t* acts;
    uint16_t* acts_shared;
    float* yacc;                                     // accumulate: fp32 rows that phase 2 adds into
    float* parts;                                    // [T x top_k routed | T shared][d] weighted rows (decode)
    const uint32_t* pair_cell;                       // cell of every pair or SHRIKE_SLOT_MISS: which parts exist
    const float* route_w;
    const float* shared_gate;
    uint32_t* status;
    uint32_t* arrived;                               // blocks done with phase 2, over all launches
    uint32_t* inst_done;                             // both phases: finished units of every instance (zeroed ahead of this launch)
    uint32_t T;
    void* y;
    void* hidden;
    uint32_t phases;                                 // bit 0, bit 1 (the last with phase 3 unless accumulate)
    uint32_t accumulate;
    uint32_t rcp_cpc;                                // ceil(2^32 / cells_per_chunk)
    StreamGeom g;
    BlockMaps maps;
};

namespace {

__device__ __forceinline__ bool try_slot(uint32_t addr, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(addr), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __noinline__ bool wait_slot_slow(uint32_t addr, uint32_t parity) {
#pragma unroll 1
    for (uint32_t it = 0; it < (1u << 18); ++it) {
        if (try_slot(addr, parity)) return true;
        if (it > 128) __nanosleep(32);
    }
    return false;
}
__device__ __forceinline__ bool wait_slot(uint32_t addr, uint32_t parity) {
    return try_slot(addr, parity) || wait_slot_slow(addr, parity);
}
__device__ __forceinline__ void arrive(uint32_t addr) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(addr) : "memory");
}
// D(16x8,f32) += A(16x8,tf32,row) * B(8x8,tf32,col)
__device__ __forceinline__ void mma_1688_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                              uint32_t b1) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Shared memory by 32-bit address (offsets known at compile time become part of the instruction).
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts32(uint32_t a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
template <int W>
__device__ __forceinline__ void lds_packed(uint32_t a, uint32_t (&w)[W]) {
    if constexpr (W == 1) {
        w[0] = lds32(a);
    } else if constexpr (W == 2) {
        const uint2 v = lds64(a);
        w[0] = v.x; w[1] = v.y;
    } else {
        const uint4 v = lds128(a);
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    }
}

// Which of the eight rows of a box this lane's MMA row g is: the rows that one shared-memory wavefront reads then
// lie in different 16-byte columns of the 128-byte swizzle.
template <int WORDS>
__device__ __forceinline__ uint32_t box_row(uint32_t g) {
    return WORDS == 4 ? (g >> 1) | ((g & 1u) << 2) : WORDS == 2 ? ((g & 3u) << 1) | (g >> 2) : g;
}

// {sum x, sum x, sum offset*x, sum offset*x} of columns 2t, 2t+1 over one group: rows 0..7 of the tile are ones, rows
// 8..15 the offsets of the unpacked integers.
template <int BITS, int GROUP>
__device__ __forceinline__ void column_sums(const uint32_t (&b)[GROUP / 8], float (&r)[4]) {
    constexpr uint32_t kOnes = 0x3C003C00u, kEven = 0x64006400u, kOdd = BITS == 4 ? 0x54005400u : 0x64006400u;
    r[0] = r[1] = r[2] = r[3] = 0.f;
#pragma unroll
    for (int m = 0; m < GROUP / 16; ++m) mma_16816(r, kOnes, kEven, kOnes, kOdd, b[2 * m], b[2 * m + 1]);
}


__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
// Bytes of an instance buffer and its parts: [group][half][column][t] 16 bytes of operands, [quad][column][t] sums,
// [group][t] initial values.
struct BufferLayout {
    uint32_t z_off, cq_off, bytes;
    __device__ BufferLayout(uint32_t groups, uint32_t halves, uint32_t count) {
        z_off = groups * halves * count * 64;
        cq_off = z_off + (groups + 3) / 4 * count * 64;
        bytes = cq_off + groups * 64;
    }
};

// One group of one instance's columns, by a warp: lane (g, t) holds quarter t of column g (columns past the count repeat
// a row of the instance; they are not stored).
template <int GROUP>
__device__ __forceinline__ void load_group(const uint16_t* row, uint32_t j, uint32_t t, uint32_t (&b)[GROUP / 8]) {
#pragma unroll
    for (int h = 0; h < GROUP / 32; ++h) {
        const uint4 v = *((const uint4*)(row + (size_t)j * GROUP + t * (GROUP / 4)) + h);
        b[4 * h] = v.x; b[4 * h + 1] = v.y; b[4 * h + 2] = v.z; b[4 * h + 3] = v.w;
    }
}
template <int BITS, int GROUP>
__device__ __forceinline__ void stage_group(const uint32_t (&b)[GROUP / 8], uint32_t j, uint32_t groups, uint32_t count, uint32_t buf,
                                            const BufferLayout& lay, uint32_t lane) {
    const uint32_t g = lane >> 2, t = lane & 3;
    float mine = 0.f;
    if (j < groups) {
#pragma unroll
        for (int h = 0; h < GROUP / 32; ++h)
            if (g < count) sts128(buf + (j * (GROUP / 32) + h) * count * 64 + lane * 16, b[4 * h], b[4 * h + 1], b[4 * h + 2], b[4 * h + 3]);
        float r[4];
        column_sums<BITS, GROUP>(b, r);
        if (lane < 4)
            sts128(buf + lay.cq_off + j * 64 + lane * 16, __float_as_uint(-r[2]), __float_as_uint(-r[3]), __float_as_uint(-r[2]), __float_as_uint(-r[3]));
        // column g's sum sits in lane g / 2
        const float v0 = __shfl_sync(0xffffffffu, r[0], g >> 1), v1 = __shfl_sync(0xffffffffu, r[1], g >> 1);
        mine = (g & 1u) ? v1 : v0;
    }
    if (t == (j & 3u) && g < count) {   // 11 + 11 + the rest of the bits: exact tf32 operands
        const float hi = __uint_as_float(__float_as_uint(mine) & 0xffffe000u), rest = mine - hi;
        const float mid = __uint_as_float(__float_as_uint(rest) & 0xffffe000u);
        sts128(buf + lay.z_off + (j >> 2) * count * 64 + lane * 16, __float_as_uint(hi), __float_as_uint(mid), __float_as_uint(rest - mid), 0u);
    }
}

// The groups of one 128-byte piece: acc += sum over groups of scale * sum(q x) + bias * sum(x), rows g and g + 8 of the
// tile against the 8 columns. w: the lane's row g in the piece, its swizzled first byte included (row g + 8 is 1024
// bytes further); sc: row g's scales of the piece, d_s / d_z bytes further row g + 8's / the biases; b, cq: this lane's
// operands of the first group in the instance's buffer, z: of its quad, sB: bytes from one 16-byte part of the operands
// to the next and from quad to quad; TAIL: a row's last piece, n of the GP groups (and rows of scales that are only
// whole 32-bit words); k0: the first group's place in its quad.
template <int BITS, int GROUP, int META, bool TAIL>
__device__ __forceinline__ void piece_tiles(uint32_t w, uint32_t sc, uint32_t d_s, uint32_t d_z, uint32_t b, uint32_t cq,
                                            uint32_t z, uint32_t sB, uint32_t n, uint32_t k0, uint32_t t, float (&acc)[4]) {
    using Q = FQ<BITS, GROUP>;
    constexpr int GB = Q::kGroupBytes, GP = 128 / GB;
    auto f32 = [](uint32_t v) {                        // the low 16 bits as a scale
        return META == SHRIKE_DTYPE_FP16 ? f16_bits_to_f32((uint16_t)(v & 0xffffu)) : __uint_as_float(v << 16);
    };
    auto f32hi = [](uint32_t v) {
        return META == SHRIKE_DTYPE_FP16 ? f16_bits_to_f32((uint16_t)(v >> 16)) : __uint_as_float(v & 0xffff0000u);
    };
    uint32_t vs[2][GP / 2];                            // scales, two 16-bit values a word
    if constexpr (!TAIL) {
        lds_packed<GP / 2>(sc, vs[0]);
        lds_packed<GP / 2>(sc + d_s, vs[1]);
    } else {
#pragma unroll
        for (int j = 0; j < GP / 2; ++j) {
            if ((uint32_t)(2 * j) < n) {
                vs[0][j] = lds32(sc + 4 * j);
                vs[1][j] = lds32(sc + d_s + 4 * j);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < (GP + 3) / 4; ++q) {           // zero points, against the sums' high parts and the next, then the rest
        if (TAIL && q > 0 && (uint32_t)(4 * q) >= n) break;
        const uint32_t k = 4 * q + t - k0;
        uint32_t za = 0, zb = 0;
        if ((!TAIL && GP >= 4) || k < (TAIL ? n : (uint32_t)GP)) {
            za = __float_as_uint(f32(lds16(sc + d_z + 2 * k)));
            zb = __float_as_uint(f32(lds16(sc + d_z + d_s + 2 * k)));
        }
        const uint4 v = lds128(z + q * sB);
        mma_1688_tf32(acc, za, zb, za, zb, v.x, v.y);
        mma_1688_tf32(acc, za, zb, 0u, 0u, v.z, 0u);
    }
#pragma unroll
    for (int i = 0; i < GP; i += 2) {                  // two groups side by side: two independent chains of tiles
        if (TAIL && (uint32_t)i >= n) break;
        uint32_t wa[2][Q::kWords], wb[2][Q::kWords], bf[2][GROUP / 8];
        float c0[2][4], c[2][4];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const uint32_t at = w ^ ((i + e) * GB);
            lds_packed<Q::kWords>(at, wa[e]);
            lds_packed<Q::kWords>(at + 1024, wb[e]);
#pragma unroll
            for (int h = 0; h < GROUP / 32; ++h) {
                const uint4 v = lds128(b);
                b += sB;
                bf[e][4 * h] = v.x; bf[e][4 * h + 1] = v.y; bf[e][4 * h + 2] = v.z; bf[e][4 * h + 3] = v.w;
            }
            const uint4 v = lds128(cq + (i + e) * 64);
            c0[e][0] = __uint_as_float(v.x); c0[e][1] = __uint_as_float(v.y);
            c0[e][2] = __uint_as_float(v.z); c0[e][3] = __uint_as_float(v.w);
        }
#pragma unroll
        for (int m = 0; m < Q::kMmas; ++m) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                uint32_t lo0, hi0, lo1, hi1;
                unpack2<BITS>(wa[e], m, lo0, hi0);
                unpack2<BITS>(wb[e], m, lo1, hi1);
                if (m == 0) mma_16816_from(c[e], lo0, lo1, hi0, hi1, bf[e][0], bf[e][1], c0[e]);
                else mma_16816(c[e], lo0, lo1, hi0, hi1, bf[e][2 * m], bf[e][2 * m + 1]);
            }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const float s0 = e ? f32hi(vs[0][i / 2]) : f32(vs[0][i / 2]), s1 = e ? f32hi(vs[1][i / 2]) : f32(vs[1][i / 2]);
            acc[0] = fmaf(s0, c[e][0], acc[0]);
            acc[1] = fmaf(s0, c[e][1], acc[1]);
            acc[2] = fmaf(s1, c[e][2], acc[2]);
            acc[3] = fmaf(s1, c[e][3], acc[3]);
        }
    }
}

__device__ __noinline__ float glu_of(float gate, float up, uint32_t activation) { return glu(gate, up, activation); }

// Everything this block did so far is visible to the blocks that have passed the same counter.
__device__ __forceinline__ bool grid_sync(uint32_t* counter) {
    bool ok = true;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        // the counter only grows: every launch adds the grid's size once
        const uint32_t goal = (atomicAdd(counter, 1u) / gridDim.x + 1u) * gridDim.x;
        ok = false;
#pragma unroll 1
        for (uint32_t it = 0; it < (1u << 18) && !ok; ++it) {
            uint32_t v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
            ok = (int32_t)(v - goal) >= 0;
            if (!ok && it > 8) __nanosleep(it > 1024 ? 256 : 20);
        }
    }
    __syncthreads();
    return ok;
}

}  // namespace

template <int BITS, int GROUP, int META, bool AL>
__global__ void __launch_bounds__(kThreads, 1) expert_stream_kernel(const __grid_constant__ StreamArgs a) {
    using Q = FQ<BITS, GROUP>;
    constexpr uint32_t GP = 128 / Q::kGroupBytes, H = GROUP / 32;   // groups of a piece; 16-byte operand parts of a group
    extern __shared__ __align__(128) uint8_t dsm_raw[];
    uint8_t* const dsm = dsm_raw + ((1024u - (smem_u32(dsm_raw) & 1023u)) & 1023u);   // the swizzle follows the address
    __shared__ uint64_t full1[kMaxSlots], done1[kMaxSlots], full2[kMaxSlots2], done2[kMaxSlots2];
    __shared__ uint32_t s_failed;
    const StreamGeom& G = a.g;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    uint8_t* const ring = dsm + G.off_ring;
    const uint32_t dsm0 = smem_u32(dsm), ring0 = smem_u32(ring);
    const uint32_t D = a.d;
    const bool do1 = a.phases & 1u, do2 = a.phases & 2u;

    if (tid < G.n_slots) { mbar_init(&full1[tid], 1); mbar_init(&done1[tid], G.w1); }
    if (tid < G.n_slots2) { mbar_init(&full2[tid], 1); mbar_init(&done2[tid], G.w2); }
    if (tid < kMaxSlots2) fence_mbar_init();
    if (tid == 0) s_failed = 0;
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();   // (the next kernel waits for this one to end; its blocks find no room before that)
    const uint32_t n_inst = *a.n_inst, n_sh = min(a.n_shared, n_inst);
    auto give_up = [&]() {
        report_status(a.status, kStatusWaitTimeout);
        s_failed = 1;
    };
    // this lane's row g of the eight, and its first byte in the row's piece
    const uint32_t pr = box_row<Q::kWords>(g), w_lane = pr * 128 + ((t * (Q::kWords * 4)) ^ (pr << 4));
    // where its partial sums go, [column][row mod 4]{row r, r + 4, r + 8, r + 12 of the 16}
    const uint32_t my_red = (pr & 3) * 16 + (pr >> 2) * 4 + 2 * t * (kRedCol * 4);

    auto phase = [&](auto which) {
        constexpr bool P1 = decltype(which)::value == 1;
        const uint32_t W = P1 ? G.w1 : G.w2, nT = kWarps / W;
        // a finishing warp serves every kFinish-th team
        const bool finisher = warp >= kWarps;
        const uint32_t team = finisher ? warp - kWarps : warp / W, wi = finisher ? 0u : warp % W;
        const uint32_t pace = finisher ? min(kFinish, nT) : nT;   // from one of this warp's units to the next
        const uint32_t n_slots = P1 ? G.n_slots : G.n_slots2;
        const uint32_t full = smem_u32(P1 ? full1 : full2), done = smem_u32(P1 ? done1 : done2);
        const uint32_t su = P1 ? a.f_shared / 8 : D / 16, ru = P1 ? a.f / 8 : D / 16, sh_units = n_sh * su;
        // this block's units: [v0, v0 + n) of [shared instances' | routed instances']
        const uint32_t total = sh_units + (n_inst - n_sh) * ru;
        const uint32_t v0 = (uint32_t)((uint64_t)total * blockIdx.x / gridDim.x);
        const uint32_t n = (uint32_t)((uint64_t)total * (blockIdx.x + 1) / gridDim.x) - v0;
        auto find = [&](uint32_t j, uint32_t& i, uint32_t& k) {   // unit j -> instance, unit in it
            const uint32_t v = v0 + j;
            if (v < sh_units) { i = v / su; k = v - i * su; }
            else { const uint32_t w = v - sh_units, q = w / ru; i = n_sh + q; k = w - q * ru; }
        };
        auto step = [&](uint32_t& i, uint32_t& k) {
            k += pace;
            for (;;) {
                const uint32_t cur = i < n_sh ? su : ru;
                if (k < cur) break;
                k -= cur;
                ++i;
            }
        };

        // ---- one lane asks for one unit ----
        uint32_t have = 0xffffffffu, mi = 0;
        int32_t cc = 0;
        const uint8_t* base = nullptr;
        auto ask = [&](uint32_t slot, uint32_t i, uint32_t k) {
            const bool sh = i < n_sh;
            if (i != have) {
                const uint32_t cell = sh ? 0u : a.inst[i].slot, ch = __umulhi(cell, a.rcp_cpc);
                mi = sh ? SHRIKE_MAX_POOL_CHUNKS : ch;
                cc = sh ? 0 : (int32_t)(cell - ch * a.pool.cells_per_chunk);
                base = sh ? a.shared_block : pool_cell_base(a.pool, cell);
                have = i;
            }
            const Offsets3& off = sh ? a.shared : a.routed;
            if constexpr (P1) {
                uint64_t* bar = &full1[slot];
                const uint32_t at = slot * G.slot_bytes;
                mbar_expect_tx(bar, 2048 * ((D * BITS / 8 + 127) / 128) + 64 * (D / GROUP) + (a.expert_bias ? 32u : 0u));
                tma_5d(ring0 + at + G.meta_off, &a.maps.m1[mi], 0, (int32_t)k, 0, 0, cc, bar);
                tma_5d(ring0 + at, &a.maps.l1[mi], 0, (int32_t)(k * 8), 0, 0, cc, bar);
                if (a.expert_bias) {
                    bulk_g2s(ring + at + G.ab_off, base + off.ab[0] + (size_t)k * 16, 16, bar);
                    bulk_g2s(ring + at + G.ab_off + 16, base + off.ab[1] + (size_t)k * 16, 16, bar);
                }
            } else {
                const uint32_t F = sh ? a.f_shared : a.f, mt = G.n_slots2 * G.w_bytes2 + slot * G.m_bytes2;
                uint64_t* bar = &full2[slot];
                mbar_expect_tx(bar, 2048 * ((F * BITS / 8 + 127) / 128) + 64 * (F / GROUP) + (a.expert_bias ? 32u : 0u));
                tma_4d(ring0 + mt, &a.maps.m2[mi], 0, (int32_t)(k * 2), 0, cc, bar);
                tma_4d(ring0 + slot * G.w_bytes2, &a.maps.l2[mi], 0, (int32_t)(k * 16), 0, cc, bar);
                if (a.expert_bias) bulk_g2s(ring + mt + G.ab_off2[sh], base + off.ab[2] + (size_t)k * 32, 32, bar);
            }
        };
        {   // the first round: unit j by lane j / 20 of warp j % 20
            const uint32_t j = warp + lane * (kWarps + kFinish);
            if (j < min(n_slots, n)) {
                uint32_t i, k;
                find(j, i, k);
                ask(j, i, k);
            }
            __syncwarp();
        }
        // ---- the instance of this warp's units ----
        uint32_t i = 0, k = 0, cur = 0xffffffffu, count = 0, G2 = 0, groups_left = 0, pieces = 0;
        uint32_t b0 = 0, cq0 = 0, z0 = 0, sB = 0, w_at = 0, s_at = 0, ab_at = 0, d_s = 0, d_z = 0, k0 = 0;
        uint16_t* dst = nullptr;   // gate/up: where column g's activations go
        float* out0 = nullptr;     // down: where the rows of column g (W == 1: columns 2t and 2t + 1) go, and their weights
        float* out1 = nullptr;
        float wt0 = 0.f, wt1 = 0.f;
        const uint32_t meta0 = ring0 + (P1 ? G.meta_off : G.n_slots2 * G.w_bytes2);
        auto open_instance = [&](uint32_t buf) {
            cur = i;
            const bool sh = i < n_sh;
            const uint32_t K = P1 ? D : sh ? a.f_shared : a.f, P = (K * BITS / 8 + 127) / 128;
            G2 = K / GROUP;
            count = a.inst[i].count;
            const uint32_t p0 = P * wi / W;
            pieces = P * (wi + 1) / W - p0;
            groups_left = G2 - min(G2, p0 * GP);
            const BufferLayout lay(G2, H, count);
            const uint32_t col = min(g, count - 1u);
            sB = count * 64;
            b0 = buf + col * 64 + t * 16 + p0 * GP * H * sB;
            cq0 = buf + lay.cq_off + t * 16 + p0 * GP * 64;
            z0 = buf + lay.z_off + col * 64 + t * 16 + (GP == 2 ? p0 / 2 : p0 * (GP / 4)) * sB;
            k0 = GP == 2 ? 2 * (p0 & 1) : 0u;
            w_at = ring0 + w_lane + p0 * 2048;
            s_at = meta0 + (pr * G2 + p0 * GP) * 2;
            d_s = P1 ? 32 * G2 : 16 * G2;
            d_z = P1 ? 16 * G2 : 32 * G2;
            ab_at = meta0 - (P1 ? G.meta_off : 0u) + (P1 ? G.ab_off : G.ab_off2[sh]) + pr * 2;
            if constexpr (P1) {
                const uint32_t pair = a.inst[i].pair[g];
                const uint32_t F = sh ? a.f_shared : a.f;
                dst = g < count ? (sh ? a.acts_shared : a.acts) + (size_t)pair * F + (BITS == 4 ? 2 * t : t) : nullptr;
            } else {
                auto target = [&](uint32_t c, float*& out, float& w) {
                    const uint32_t pair = a.inst[i].pair[c];
                    w = sh ? (a.shared_gate ? a.shared_gate[pair] : 1.0f) : a.route_w[pair];
                    float* rows = a.accumulate ? a.yacc + (size_t)(sh ? pair : pair / a.top_k) * D
                                               : a.parts + ((size_t)pair + (sh ? a.T * a.top_k : 0u)) * D;
                    out = c < count ? rows + (W == 1 ? pr : t) : nullptr;
                };
                target(W == 1 ? 2 * t : g, out0, wt0);
                target(W == 1 ? 2 * t + 1 : g, out1, wt1);
            }
        };
        auto put = [&](float* at, float v) {
            if (a.accumulate) atomicAdd(at, v);
            else *at = v;
        };

        uint32_t i0 = 0, i_end = 0;   // the first staged instance, the end of the block's
        if (n) {
            uint32_t dummy;
            find(0, i0, dummy);
            find(n - 1, i_end, dummy);
            ++i_end;
        }
        // (W == 1: the warps finish their units themselves; fewer teams than finishing warps: some have none)
        uint32_t u = finisher && (W == 1 || team >= nT) ? n : team, slot = team, par = 0;
        if (u < n) find(u, i, k);
        uint32_t pend = 0;            // units of `cur` whose activations this warp wrote and has not announced
        auto announce = [&]() {
            if (P1 && do2 && pend) {
                __syncwarp();
                if (lane == 0) asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(a.inst_done + cur), "r"(pend) : "memory");
                pend = 0;
            }
        };
        bool later = false;
        while (i0 < i_end) {
            // every warp works out for itself which instances fit: lane l has instance i0 + l
            uint32_t at = 0, i1 = i0;
            {
                const uint32_t ii = i0 + lane;
                uint32_t bytes = 0;
                if (ii < i_end) {
                    const uint32_t K = P1 ? D : ii < n_sh ? a.f_shared : a.f;
                    bytes = BufferLayout(K / GROUP, H, a.inst[ii].count).bytes;
                }
                uint32_t end = bytes;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(0xffffffffu, end, o);
                    if (lane >= (uint32_t)o) end += v;
                }
                at = end - bytes;   // (a prefix of the lanes fits; at least one: the region holds eight columns)
                i1 += __popc(__ballot_sync(0xffffffffu, ii < i_end && end <= G.off_red));
            }
            if (later) __syncthreads();   // the buffers' last readers are done
            later = true;
            {   // groups of the instances in turn over all warps, two at a time
                uint32_t ii = i0, j = warp;
                auto next = [&](const uint16_t*& row, uint32_t& ji, uint32_t& groups, uint32_t& cnt, uint32_t& buf) {
                    for (;;) {
                        if (ii >= i1) return false;
                        groups = (P1 ? D : ii < n_sh ? a.f_shared : a.f) / GROUP;
                        const uint32_t g4 = (groups + 3) & ~3u;
                        if (j < g4) break;
                        j -= g4;
                        ++ii;
                    }
                    const bool sh = ii < n_sh;
                    const uint32_t mine = a.inst[ii].pair[g];
                    cnt = a.inst[ii].count;
                    const uint32_t p = __shfl_sync(0xffffffffu, mine, 4 * min(g, cnt - 1u) + t);   // past the count: the last row
                    if constexpr (P1) {
                        row = a.xh + (size_t)(sh ? p : p / a.top_k) * D;
                    } else {
                        const uint32_t F = sh ? a.f_shared : a.f;
                        row = (sh ? a.acts_shared : a.acts) + (size_t)p * F;
                        if (do1) {   // the instance's activations, whoever wrote them
                            bool ok = false;
#pragma unroll 1
                            for (uint32_t it = 0; it < (1u << 18) && !ok; ++it) {
                                uint32_t v;
                                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a.inst_done + ii) : "memory");
                                ok = v >= F / 8;
                                if (!ok) __nanosleep(it > 1024 ? 256 : 20);
                            }
                            if (!ok) give_up();
                        }
                    }
                    ji = j;
                    buf = dsm0 + __shfl_sync(0xffffffffu, at, ii - i0);
                    j += kWarps + kFinish;
                    return true;
                };
                for (;;) {
                    const uint16_t *ra, *rb2;
                    uint32_t ja, jb, ga, gb, ca, cb, ba, bb;
                    uint32_t xa[GROUP / 8], xb[GROUP / 8];
                    if (!next(ra, ja, ga, ca, ba)) break;
                    if (ja < ga) load_group<GROUP>(ra, ja, t, xa);
                    const bool two = next(rb2, jb, gb, cb, bb);
                    if (two && jb < gb) load_group<GROUP>(rb2, jb, t, xb);
                    stage_group<BITS, GROUP>(xa, ja, ga, ca, ba, BufferLayout(ga, H, ca), lane);
                    if (!two) break;
                    stage_group<BITS, GROUP>(xb, jb, gb, cb, bb, BufferLayout(gb, H, cb), lane);
                }
            }
            if (u < n && i < i1 && i != cur) {   // (its loads run while the others stage)
                announce();
                open_instance(dsm0 + __shfl_sync(0xffffffffu, at, i - i0));
            }
            __syncthreads();
            for (; u < n && i < i1; u += pace) {
                if (i != cur) {
                    announce();
                    open_instance(dsm0 + __shfl_sync(0xffffffffu, at, i - i0));
                }
                const uint32_t bar_at = slot * 8, rb = dsm0 + G.off_red + slot * W * (kRedWarp * 4);
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);   // column g, rows t, t + 4, t + 8, t + 12
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
                if (!finisher) {
                    if (!try_slot(full + bar_at, par) && !wait_slot_slow(full + bar_at, par)) give_up();
                    const uint32_t mo = slot * (P1 ? G.slot_bytes : G.m_bytes2);
                    if (a.expert_bias && wi == 0) {
                        acc[0] = acc[1] = bf16_bits_to_f32((uint16_t)lds16(ab_at + mo));
                        acc[2] = acc[3] = bf16_bits_to_f32((uint16_t)lds16(ab_at + mo + 16));
                    }
                    uint32_t w = w_at + slot * (P1 ? G.slot_bytes : G.w_bytes2), sc = s_at + mo, b = b0, cq = cq0, z = z0, kk = k0, left = groups_left;
#pragma unroll 1
                    for (uint32_t p = 0; p < pieces; ++p) {
                        piece_tiles<BITS, GROUP, META, !AL>(w, sc, d_s, d_z, b, cq, z, sB, min(GP, left), kk, t, acc);
                        w += 2048;
                        sc += 2 * GP;
                        b += GP * H * sB;
                        cq += GP * 64;
                        if constexpr (GP == 2) {
                            kk ^= 2u;
                            z += kk ? 0u : sB;
                        } else {
                            z += GP / 4 * sB;
                        }
                        left -= GP;
                    }
                    if (P1 || W > 1) {
                        const uint32_t at = rb + wi * (kRedWarp * 4) + my_red;
                        sts32(at, acc[0]);
                        sts32(at + kRedCol * 4, acc[1]);
                        sts32(at + 8, acc[2]);
                        sts32(at + kRedCol * 4 + 8, acc[3]);
                    }
                    __syncwarp();
                    if (W > 1 && lane == 0) arrive(done + bar_at);
                } else {
                    if (!try_slot(done + bar_at, par) && !wait_slot_slow(done + bar_at, par)) give_up();
                }
                if (finisher || W == 1) {
                    if (P1 || W > 1) {
#pragma unroll 4
                        for (uint32_t w = 0; w < W; ++w) {
                            const uint4 p = lds128(rb + w * (kRedWarp * 4) + g * (kRedCol * 4) + t * 16);
                            v.x += __uint_as_float(p.x); v.y += __uint_as_float(p.y); v.z += __uint_as_float(p.z); v.w += __uint_as_float(p.w);
                        }
                        __syncwarp();
                    }
                    if (lane == 0 && u + n_slots < n) {
                        uint32_t ri, rk;
                        find(u + n_slots, ri, rk);
                        ask(slot, ri, rk);
                    }
                    __syncwarp();
                    if constexpr (P1) {
                        const uint16_t h0 = act_to_half_bits(glu_of(v.x, v.z, a.activation), a.status);
                        const uint16_t h1 = act_to_half_bits(glu_of(v.y, v.w, a.activation), a.status);
                        if (dst) {
                            if constexpr (BITS == 4) {   // rows t and t + 4 are neighbours in the operand order
                                *(uint32_t*)(dst + k * 8) = h0 | ((uint32_t)h1 << 16);
                            } else {
                                dst[k * 8] = h0;
                                dst[k * 8 + 4] = h1;
                            }
                        }
                        ++pend;
                    } else if (W == 1) {
                        if (out0) {
                            put(out0 + k * 16, wt0 * acc[0]);
                            put(out0 + k * 16 + 8, wt0 * acc[2]);
                        }
                        if (out1) {
                            put(out1 + k * 16, wt1 * acc[1]);
                            put(out1 + k * 16 + 8, wt1 * acc[3]);
                        }
                    } else if (out0) {
                        float* o = out0 + k * 16;
                        put(o, wt0 * v.x);
                        put(o + 4, wt0 * v.y);
                        put(o + 8, wt0 * v.z);
                        put(o + 12, wt0 * v.w);
                    }
                }
                step(i, k);
                slot += pace;
                if (slot >= n_slots) { slot -= n_slots; par ^= 1u; }
            }
            i0 = i1;
        }
        announce();
    };

    if (do1) phase(std::integral_constant<int, 1>());
    __syncthreads();   // the ring changes hands
    if (do2) phase(std::integral_constant<int, 2>());
    if (s_failed) {
        // a copy of this block may still be in flight: give it a bounded time to land
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
    }
    if (!do2 || a.accumulate) return;
    // ================= y = the rows' parts; hidden += y =================
    // one output element pair per thread over all blocks; what does not depend on the parts is read ahead of the wait
    // (warps go round the blocks, so that a small call keeps every SM busy)
    const uint32_t half = D / 2, items = a.T * half, stride = gridDim.x * kThreads;
    uint32_t j = (warp * gridDim.x + blockIdx.x) * 32 + lane;
    auto live_of = [&](uint32_t tk) {
        uint32_t live = 0;
#pragma unroll
        for (uint32_t q = 0; q < SHRIKE_MAX_TOP_K; ++q)
            if (q < a.top_k && a.pair_cell[tk * a.top_k + q] != SHRIKE_SLOT_MISS) live |= 1u << q;
        return live;
    };
    uint32_t live = 0;
    float h0 = 0.f, h1 = 0.f;
    if (j < items) {
        live = live_of(j / half);
        if (a.hidden) {
            h0 = load_act(a.hidden, (size_t)j * 2, a.act_dtype);
            h1 = load_act(a.hidden, (size_t)j * 2 + 1, a.act_dtype);
        }
    }
    if (!grid_sync(a.arrived)) give_up();
    for (bool first = true; j < items; j += stride, first = false) {
        const uint32_t tk = j / half, c = j - tk * half;
        if (!first) live = live_of(tk);
        float2 s = make_float2(0.f, 0.f), p[SHRIKE_MAX_TOP_K];
        if (n_sh) s = __ldcg((const float2*)(a.parts + ((size_t)a.T * a.top_k + tk) * D) + c);
#pragma unroll
        for (uint32_t q = 0; q < SHRIKE_MAX_TOP_K; ++q)
            if (live >> q & 1u) p[q] = __ldcg((const float2*)(a.parts + ((size_t)tk * a.top_k + q) * D) + c);
        const size_t o = (size_t)j * 2;
        if (!first && a.hidden) {
            h0 = load_act(a.hidden, o, a.act_dtype);
            h1 = load_act(a.hidden, o + 1, a.act_dtype);
        }
#pragma unroll
        for (uint32_t q = 0; q < SHRIKE_MAX_TOP_K; ++q)
            if (live >> q & 1u) { s.x += p[q].x; s.y += p[q].y; }
        store_act(a.y, o, a.y_dtype, s.x);
        store_act(a.y, o + 1, a.y_dtype, s.y);
        if (a.hidden) {
            store_act(a.hidden, o, a.act_dtype, h0 + round_act(a.y_dtype, s.x));
            store_act(a.hidden, o + 1, a.act_dtype, h1 + round_act(a.y_dtype, s.y));
        }
    }
}

// ---- host ----------------------------------------------------------------------------------

namespace {

inline uint32_t align_up(uint32_t v, uint32_t a) { return (v + a - 1) / a * a; }

// Shared-memory layout; false when the shape does not fit.
bool stream_geometry(const shrike_moe_config& c, uint32_t smem_optin, StreamGeom& g) {
    memset(&g, 0, sizeof g);
    const uint32_t G1 = c.d / c.group_size, G2 = c.f / c.group_size, Gs = c.has_shared ? c.shared_f / c.group_size : 0;
    if ((G1 | G2 | Gs) & 1u) return false;   // rows of scales are read as 32-bit words
    auto pieces = [&](uint32_t K) { return (K * c.weight_bits / 8 + 127) / 128; };
    auto buffer = [&](uint32_t groups) { return groups * (c.group_size / 32) * 512 + (groups + 3) / 4 * 512 + groups * 64; };   // eight columns
    g.meta_off = 2048 * pieces(c.d);
    g.ab_off = align_up(g.meta_off + 64 * G1, 128);
    g.slot_bytes = align_up(g.ab_off + (c.expert_bias ? 128 : 0), 1024);
    for (int sh = 0; sh < (c.has_shared ? 2 : 1); ++sh) {
        const uint32_t F = sh ? c.shared_f : c.f;
        g.w_bytes2 = std::max(g.w_bytes2, 2048 * pieces(F));
        g.ab_off2[sh] = align_up(64 * (F / c.group_size), 128);
        g.m_bytes2 = std::max(g.m_bytes2, g.ab_off2[sh] + (c.expert_bias ? 128u : 0u));
    }
    const uint32_t least = std::max(buffer(G1), buffer(std::max(G2, Gs))), most_pieces2 = g.w_bytes2 / 2048;
    const uint32_t budget = smem_optin - 3072 - 1024;   // less the static part, the reserved kilobyte, the ring's alignment
    if (least > budget) return false;
    // Teams as small as leaves every team two slots (more warps on a unit mean more partial sums), no smaller than four
    // pieces a warp needs. Slots are a multiple of the teams: a team that runs ahead then cannot take an older round of
    // a slot for its own.
    auto team_of = [&](uint32_t P, uint32_t bytes, uint32_t most_slots, uint32_t& W, uint32_t& slots) {
        for (W = 1; W <= kWarps; W *= 2) {
            const uint32_t nT = kWarps / W, per = bytes + (W > 1 ? W * kRedWarp * 4 : 0), fit = std::min(most_slots, (budget - least) / per);
            if (W < kWarps && P > 4 * W) continue;
            if (fit >= 2 * nT) {
                slots = fit / nT * nT;
                if (slots > 3 * nT) slots = 3 * nT;
                return true;
            }
        }
        return false;
    };
    if (!team_of(pieces(c.d), g.slot_bytes, kMaxSlots, g.w1, g.n_slots)) return false;
    if (!team_of(most_pieces2, g.w_bytes2 + g.m_bytes2, kMaxSlots2, g.w2, g.n_slots2)) return false;
    const uint32_t ring = std::max(g.n_slots * g.slot_bytes, g.n_slots2 * (g.w_bytes2 + g.m_bytes2));
    const uint32_t red = std::max(g.n_slots * g.w1, g.w2 > 1 ? g.n_slots2 * g.w2 : 0u) * kRedWarp * 4;
    if (ring + red + least > budget) return false;
    g.off_red = (budget - ring - red) / 128 * 128;
    g.off_ring = align_up(g.off_red + red, 1024);
    if (g.off_ring > budget + 1023 - ring) { g.off_red -= 1024; g.off_ring -= 1024; }
    if (g.off_red < least) return false;
    g.smem_bytes = g.off_ring + ring + 1024;
    return true;
}

template <int BITS, int GROUP, int META, bool AL>
cudaError_t launch_stream_t(const shrike_moe* m, cudaStream_t st, StreamArgs& a, bool pdl) {
    auto k = expert_stream_kernel<BITS, GROUP, META, AL>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)a.g.smem_bytes);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)m->sm_count);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = a.g.smem_bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    unsigned n = 0;
    if (a.phases == 3u || ((a.phases & 2u) && !a.accumulate)) {   // the blocks wait for each other between the phases
        attr[n].id = cudaLaunchAttributeCooperative;
        attr[n].val.cooperative = 1;
        ++n;
    }
    if (pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, k, a);
}

template <int BITS, int GROUP, int META>
cudaError_t launch_stream_m(const shrike_moe* m, cudaStream_t st, StreamArgs& a, bool pdl) {
    // every row whole 128-byte pieces?
    const shrike_moe_config& c = m->cfg;
    const uint32_t gp = 128 / (GROUP * BITS / 8);
    const bool al = c.d / GROUP % gp == 0 && c.f / GROUP % gp == 0 && (!c.has_shared || c.shared_f / GROUP % gp == 0);
    return al ? launch_stream_t<BITS, GROUP, META, true>(m, st, a, pdl) : launch_stream_t<BITS, GROUP, META, false>(m, st, a, pdl);
}

}  // namespace

size_t stream_parts_bytes(const shrike_moe_config& c) {
    const size_t T = std::min(c.max_tokens, (uint32_t)SHRIKE_MAX_DECODE_TOKENS);
    return T * (c.top_k + (c.has_shared ? 1u : 0u)) * c.d * 4;
}

// phases: 1, 2 or both. accumulate: phase 2 adds into ea.yacc (prefill) instead of writing y and hidden.
// cudaErrorNotSupported when the shape does not fit: nothing was launched.
cudaError_t launch_expert_stream(const shrike_moe* m, cudaStream_t st, const ExpertArgs& ea, uint32_t T, uint32_t n_shared,
                                 uint32_t phases, bool accumulate, void* y, void* hidden, bool pdl) {
    const shrike_moe_config& c = m->cfg;
    const uint64_t cpc = ea.pool.cells_per_chunk ? ea.pool.cells_per_chunk : 1;
    if (cpc < 2 || (uint64_t)ea.pool.cells * cpc >= (1ull << 32)) return cudaErrorNotSupported;
    const BlockMaps* maps = block_maps_for(m, ea);
    if (!maps) return cudaErrorNotSupported;
    StreamArgs a;
    memset(&a, 0, sizeof a);
    a.maps = *maps;
    if (!stream_geometry(c, m->smem_optin, a.g)) return cudaErrorNotSupported;
    a.pool = ea.pool; a.routed = ea.routed; a.shared = ea.shared; a.shared_block = ea.shared_block;
    a.d = c.d; a.f = c.f; a.f_shared = c.has_shared ? c.shared_f : 0; a.top_k = c.top_k;
    a.activation = c.activation; a.expert_bias = c.expert_bias; a.act_dtype = c.act_dtype; a.y_dtype = c.y_dtype;
    a.inst = ea.inst; a.n_inst = ea.n_inst; a.n_shared = n_shared;
    a.xh = ea.xh; a.acts = ea.acts; a.acts_shared = ea.acts_shared; a.yacc = ea.yacc;
    a.parts = m->ws.parts; a.pair_cell = m->ws.pair_cell;
    a.route_w = ea.route_w; a.shared_gate = ea.shared_gate; a.status = ea.status; a.arrived = m->ws.arrived; a.inst_done = m->ws.inst_done;
    a.T = T; a.y = y; a.hidden = hidden; a.phases = phases; a.accumulate = accumulate ? 1u : 0u;
    a.rcp_cpc = (uint32_t)(((1ull << 32) + cpc - 1) / cpc);
    const uint32_t bits = c.weight_bits, grp = c.group_size;
    const bool f16 = c.meta_dtype == SHRIKE_DTYPE_FP16;
    if (bits == 4 && grp == 64 && !f16) return launch_stream_m<4, 64, SHRIKE_DTYPE_BF16>(m, st, a, pdl);
    if (bits == 4 && grp == 64 && f16) return launch_stream_m<4, 64, SHRIKE_DTYPE_FP16>(m, st, a, pdl);
    if (bits == 4 && grp == 32 && !f16) return launch_stream_m<4, 32, SHRIKE_DTYPE_BF16>(m, st, a, pdl);
    if (bits == 4 && grp == 32 && f16) return launch_stream_m<4, 32, SHRIKE_DTYPE_FP16>(m, st, a, pdl);
    if (bits == 8 && grp == 64 && !f16) return launch_stream_m<8, 64, SHRIKE_DTYPE_BF16>(m, st, a, pdl);
    if (bits == 8 && grp == 64 && f16) return launch_stream_m<8, 64, SHRIKE_DTYPE_FP16>(m, st, a, pdl);
    if (bits == 8 && grp == 32 && !f16) return launch_stream_m<8, 32, SHRIKE_DTYPE_BF16>(m, st, a, pdl);
    if (bits == 8 && grp == 32 && f16) return launch_stream_m<8, 32, SHRIKE_DTYPE_FP16>(m, st, a, pdl);
    return cudaErrorInvalidValue;
}

}  // namespace shrike
