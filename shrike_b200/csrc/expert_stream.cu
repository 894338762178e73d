// A decode layer of 2 to 64 rows, or its expert projections alone: router and work list, gate/up + GLU and down at memory
// speed for instances of up to 8 rows that share an expert block.
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
//   * the parts of a row are added up in the order of its picks: results do not depend on timing.
// All phases run in one launch when the call has them: a block asks for its first phase-2 units before it waits for
// the other blocks' activations.
//
// Measured (256 experts of 2048 x 512, top 8, int4, 16 rows: 181 MB of expert blocks): the whole layer 60 us where router,
// gate/up and down launches took 101; gate/up reads 121 MB in 19 us (6.3 TB/s), down 60 MB in 11 (5.5 TB/s), the rest is the
// routing (11 us, 16 with divisions, serial picks and all rows in every block), the first units' way (5 us), the hand-over between the
// projections (5 us) and the row sums (5 us). DRAM reads are the algorithmic bytes (184 MB).
#include "block_maps.cuh"
#include "plan.cuh"
#include "route_args.cuh"
#include "router_math.cuh"
#include "select.cuh"
#include "tile_math.cuh"

#include <algorithm>
#include <type_traits>

namespace shrike {

namespace {

constexpr uint32_t kWarps = 16, kFinish = 4;         // multiplying and finishing warps
constexpr uint32_t kThreads = (kWarps + kFinish) * 32;
constexpr uint32_t kMaxSlots = 32, kMaxSlots2 = 48;
constexpr uint32_t kRedCol = 20;                     // floats per column of a warp's partial sums (16 + padding)
constexpr uint32_t kRedWarp = 8 * kRedCol;
// most instances of a call: each expert once, once more per eight pairs, and the shared expert's
constexpr uint32_t kMaxTable = SHRIKE_MAX_EXPERTS + kPlanMaxPairs / 8 + SHRIKE_MAX_DECODE_TOKENS / 8;
static_assert(kMaxTable <= 65536 && kThreads >= SHRIKE_MAX_EXPERTS, "work list");

}  // namespace

// Shared memory: [instance buffers][partial sums][ring]. An instance buffer holds the B operands of the instance's rows
// (columns; lanes past the count read the last one's), per four groups their sums as tf32 operands, and per group
// the accumulators' initial values. Buffers are packed: most instances of a decode call have one or two rows.
struct StreamGeom {
    uint32_t meta_off, ab_off, slot_bytes, n_slots, w1;   // phase 1: scales/biases and additive biases in a slot; warps of a team
    uint32_t ab_off2[2], w_bytes2, m_bytes2, n_slots2, w2;   // phase 2, [0] routed, [1] shared; [slot] weights, then [slot] the rest
    uint32_t off_red, off_ring, ring_bytes, smem_bytes;
};

// The call's work list as every block keeps it: instance i is block cell[i] (the first n_shared: the shared expert's) for
// count[i] rows, the pairs sorted[first[i]] and on (shared: the rows first[i] and on).
struct StreamTable {
    uint32_t cell[kMaxTable];
    uint16_t first[kMaxTable];
    uint8_t count[kMaxTable];
    uint16_t sorted[kPlanMaxPairs];
    float weight[kPlanMaxPairs];                     // a routing launch: the pairs' route weights
    uint8_t live[SHRIKE_MAX_DECODE_TOKENS];          // bit q: the row's pick q has a cell
    uint32_t warp_sum[SHRIKE_MAX_EXPERTS / 32];
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
    float* parts;                                    // [T x top_k routed | T shared][d] weighted rows (decode)
    const uint32_t* sorted;                          // plan of a call that does not route: the pairs by instance
    const uint32_t* pair_cell;                       // and the cell of every pair or SHRIKE_SLOT_MISS
    const float* route_w;
    const float* shared_gate;
    uint32_t* status;
    unsigned long long* arrived;                     // blocks past a grid barrier, over all launches
    uint32_t* inst_done;                             // both phases: finished gate/up units of every instance
    uint32_t T;
    void* y;
    void* hidden;
    uint32_t phases;                                 // bit 0, bit 1 (with phase 3); both: this launch routes its rows first
    uint32_t rcp_cpc;                                // ceil(2^32 / cells_per_chunk)
    // Reciprocals as quotient() takes them: of the grid, the shared and routed instances' units in phase 1, an instance's in phase
    // 2, top_k, half a row and the blocks of a token group.
    uint32_t rcp_grid, rcp_su, rcp_ru, rcp_u2, rcp_top_k, rcp_half, rcp_nbx;
    uint32_t token_groups_log2;                      // of the logits: a block takes one group's rows against its share of the experts
    RouterArgs r;
    StreamGeom g;
};

// Scratch of the routing, in front of the ring: the pairs of every expert as a bit mask, the experts' residency words
// and the cells of those picked.
struct RouteScratch {
    uint32_t mask[kPlanMaxPairs / 32][SHRIKE_MAX_EXPERTS];
    uint64_t word[SHRIKE_MAX_EXPERTS];
    uint32_t cell[SHRIKE_MAX_EXPERTS];
    RowScratch row[kWarps + kFinish];
};
// Bytes of the kernel's static shared memory: the table, the barriers and two words.
constexpr uint32_t kStaticBytes = (sizeof(StreamTable) + 15) / 16 * 16 + (2 * (kMaxSlots + kMaxSlots2) + 1) * 8 + 24;

namespace {

// v / d by the reciprocal ceil(2^32 / d), exact while v * d < 2^32; 0 stands for d = 1. (A warp's division by a variable
// takes a few hundred cycles here, the two 64-bit ones of a phase's share a thousand: most of the instructions are waited for.)
__device__ __forceinline__ uint32_t quotient(uint32_t v, uint32_t rcp) { return rcp ? __umulhi(v, rcp) : v; }

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
__device__ __forceinline__ uint32_t lds8(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
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
__device__ __forceinline__ void sts64(uint32_t a, uint32_t x, uint32_t y) {
    asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
// Bytes of an instance buffer and its parts: [group][half][column][t] 16 bytes of operands, [quad][column][t] sums,
// [group][t] 8 bytes of initial values (columns 2t and 2t + 1; a tile's rows have the same).
struct BufferLayout {
    uint32_t z_off, cq_off, bytes;
    __device__ BufferLayout(uint32_t groups, uint32_t halves, uint32_t count) {
        z_off = groups * halves * count * 64;
        cq_off = z_off + (groups + 3) / 4 * count * 64;
        bytes = (cq_off + groups * 32 + 15u) & ~15u;
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
        if (lane < 4) sts64(buf + lay.cq_off + j * 32 + lane * 8, __float_as_uint(-r[2]), __float_as_uint(-r[3]));
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
            const uint2 v = lds64(cq + (i + e) * 32);
            c0[e][0] = c0[e][2] = __uint_as_float(v.x);
            c0[e][1] = c0[e][3] = __uint_as_float(v.y);
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
__device__ __forceinline__ bool grid_sync(unsigned long long* counter) {
    bool ok = true;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        // the counter only grows (for more launches than there is time for): every barrier adds the grid's size once
        const unsigned long long goal = (atomicAdd(counter, 1ull) / gridDim.x + 1ull) * gridDim.x;
        ok = false;
#pragma unroll 1
        for (uint32_t it = 0; it < (1u << 18) && !ok; ++it) {
            unsigned long long v;
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(counter) : "memory");
            ok = v >= goal;
            if (!ok && it > 8) __nanosleep(it > 1024 ? 256 : 20);
        }
    }
    __syncthreads();
    return ok;
}

// Lane sums of two rows against two activation rows (fp32, scaled where the router scales columns), all in shared memory:
// acc[row][x]. fp32 rows in the order of lane_dot_f32; a lane's chunks past the row's end are left out.
__device__ __forceinline__ void dots_f32(uint32_t w0, uint32_t w1, uint32_t x0, uint32_t x1, uint32_t chunks, uint32_t lane, float (&acc)[2][2]) {
#pragma unroll 2
    for (uint32_t c = lane; c < chunks; c += 32) {
        uint32_t w[2][4], x[2][4];
        lds_packed<4>(w0 + c * 16, w[0]);
        lds_packed<4>(w1 + c * 16, w[1]);
        lds_packed<4>(x0 + c * 16, x[0]);
        lds_packed<4>(x1 + c * 16, x[1]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int u = 0; u < 2; ++u) acc[k][u] = __fmaf_rn(__uint_as_float(w[k][i]), __uint_as_float(x[u][i]), acc[k][u]);
    }
}
// Affine rows (their packed integers and {scale, bias} pairs), in the order of lane_dot_affine.
__device__ __forceinline__ void dots_affine(uint32_t w0, uint32_t w1, uint32_t sb0, uint32_t sb1, uint32_t x0, uint32_t x1, uint32_t groups,
                                            uint32_t bits, uint32_t lane, float (&acc)[2][2]) {
#pragma unroll 2
    for (uint32_t gi = 0; gi < groups; ++gi) {
        const uint2 xr[2] = {lds64(x0 + (gi * 32 + lane) * 8), lds64(x1 + (gi * 32 + lane) * 8)};
        const uint2 sb[2] = {lds64(sb0 + gi * 8), lds64(sb1 + gi * 8)};
        uint32_t q[2];
        if (bits == 4) {
            q[0] = lds8(w0 + gi * 32 + lane); q[1] = lds8(w1 + gi * 32 + lane);
            q[0] = (q[0] & 0xfu) | (q[0] & 0xf0u) << 4; q[1] = (q[1] & 0xfu) | (q[1] & 0xf0u) << 4;
        } else {
            q[0] = lds16(w0 + gi * 64 + lane * 2); q[1] = lds16(w1 + gi * 64 + lane * 2);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float q0 = (float)(q[k] & 0xffu), q1 = (float)(q[k] >> 8), sc = __uint_as_float(sb[k].x), bi = __uint_as_float(sb[k].y);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const float xa = __uint_as_float(xr[u].x), xb = __uint_as_float(xr[u].y);
                acc[k][u] = __fmaf_rn(sc, __fadd_rn(__fmul_rn(q0, xa), __fmul_rn(q1, xb)), acc[k][u]);
                acc[k][u] = __fmaf_rn(bi, __fadd_rn(xa, xb), acc[k][u]);
            }
        }
    }
}

// The call's work list into `tab`: routed here, or read from the plan of an earlier launch. Returns the number of
// instances. (Inlined: what a call saves of its caller's registers goes through an L1 that the ring leaves 28 KB.)
__device__ __forceinline__ uint32_t work_list(const StreamArgs& a, uint8_t* dsm, uint8_t* ring, StreamTable& tab, uint64_t* rows_here,
                                           uint32_t* failed) {
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, ring0 = smem_u32(ring), D = a.d;
    auto give_up = [&]() {
        report_status(a.status, kStatusWaitTimeout);
        *failed = 1;
    };
    uint32_t n_inst;
    const uint32_t n_sh = a.n_shared;
    if (a.phases == 3u) {
        // ================= router, selection, lookup, work list =================
        // A block has a share of the expert rows (they go to the ring's memory, asked for ahead of the wait) and of the
        // activation rows; what follows the logits every block does for itself: another hand-over between blocks costs
        // more than the work (a row's picks 2 us by one warp, the list 1 us).
        const RouterArgs& r = a.r;
        const uint32_t rows = r.ne + (r.gate_row ? 1u : 0u), tg = a.token_groups_log2, bx = blockIdx.x >> tg, by = blockIdx.x & ((1u << tg) - 1u);
        const uint32_t nbx = gridDim.x >> tg, e0 = bx < nbx ? quotient(rows * bx, a.rcp_nbx) : 0u, e1 = bx < nbx ? quotient(rows * (bx + 1), a.rcp_nbx) : 0u;
        const uint32_t t0 = (a.T * by) >> tg, nt = ((a.T * (by + 1)) >> tg) - t0;
        const uint32_t row_bytes = r.bits ? D * r.bits / 8 : D * 4, n_exp = min(e1, r.ne) - min(e0, r.ne), groups = D / 64;
        const bool gate_here = r.gate_row && e1 == rows && e1 > e0;
        const uint32_t gate_at = ring0 + n_exp * row_bytes, sb_at = gate_at + (gate_here ? D * 4 : 0u);
        if (tid == 0 && e1 > e0) {
            mbar_expect_tx(rows_here, n_exp * row_bytes + (gate_here ? D * 4 : 0u));
            if (n_exp) bulk_g2s(ring, (const uint8_t*)r.w + (size_t)e0 * row_bytes, n_exp * row_bytes, rows_here);
            if (gate_here) bulk_g2s(ring + n_exp * row_bytes, r.gate_row, D * 4, rows_here);
        }
        if (r.bits)
            for (uint32_t j = tid; j < n_exp * groups; j += kThreads) {
                const float2 v = make_float2(bf16_bits_to_f32(r.scales[(size_t)e0 * groups + j]), bf16_bits_to_f32(r.biases[(size_t)e0 * groups + j]));
                *(float2*)(ring + (sb_at - ring0) + j * 8) = v;
            }
        pdl_wait();
        pdl_launch_dependents();   // (the next kernel waits for this one to end; its blocks find no room before that)
        RouteScratch& rs = *(RouteScratch*)dsm;
        const uint32_t n_pairs = a.T * r.top_k, n_words = (n_pairs + 31) / 32;
        uint32_t io = 1u;
        if (r.io_status) io = *r.io_status;
        if (tid < r.ne) rs.word[tid] = r.table[tid];
        for (uint32_t j = tid; j < n_words * SHRIKE_MAX_EXPERTS; j += kThreads) (&rs.mask[0][0])[j] = 0;
        if (blockIdx.x == gridDim.x - 1)
            for (uint32_t j = tid; j < kMaxTable; j += kThreads) a.inst_done[j] = 0;
        // The block's activation rows go to shared memory too, as many at a time as there is room for: read where they
        // are used, every batch of a row costs a round trip to L2 of its own.
        const bool x32 = r.dt == SHRIKE_DTYPE_FP32;
        const size_t x_stride = (size_t)r.stride * (x32 ? 4 : 2);
        const uint32_t x_bytes = D * 4, xs_at = (sb_at + (r.bits ? n_exp * groups * 8 : 0u) + 15u) & ~15u, quads = D / 4;
        const uint32_t room = ((a.g.ring_bytes - (xs_at - ring0)) / x_bytes) & ~1u;
        const uint32_t n_f = r.bits ? 0u : n_exp, pairs_a = r.bits ? (n_exp + 1) / 2 : 0u;
        const uint32_t n_f32 = n_f + (gate_here ? 1u : 0u), f_at = gate_at - n_f * row_bytes;   // (the gate row follows the expert rows)
        for (uint32_t s0 = 0; s0 < nt; s0 += room) {
            const uint32_t here = min(room, nt - s0);
            if (s0) __syncthreads();
            if (e1 > e0) {
                for (uint32_t c = tid; c < quads; c += kThreads) {
                    float es[4] = {1.f, 1.f, 1.f, 1.f};
                    if (r.eff_scale) {
                        const uint2 e = __ldg((const uint2*)r.eff_scale + c);
                        es[0] = __uint_as_float(e.x << 16); es[1] = __uint_as_float(e.x & 0xffff0000u);
                        es[2] = __uint_as_float(e.y << 16); es[3] = __uint_as_float(e.y & 0xffff0000u);
                    }
#pragma unroll 8
                    for (uint32_t row = 0; row < here; ++row) {
                        float x[4];
                        load_act4((const uint8_t*)r.hidden + (t0 + s0 + row) * x_stride, c, r.dt, x);
                        if (r.eff_scale)
#pragma unroll
                            for (int i = 0; i < 4; ++i) x[i] = __fmul_rn(x[i], es[i]);
                        sts128(xs_at + row * x_bytes + c * 16, __float_as_uint(x[0]), __float_as_uint(x[1]), __float_as_uint(x[2]), __float_as_uint(x[3]));
                    }
                }
            }
            if (s0 == 0)   // the fp16 operand copy of all rows, by all blocks
                for (uint32_t j0 = (warp * gridDim.x + blockIdx.x) * 32, items = a.T * (D / 8); j0 < items; j0 += kThreads * gridDim.x)
                    xprep_item(r.hidden, x_stride, D, r.group, r.dt, r.int4 != 0, j0 + lane, j0 + lane < items, r.xh, r.xsum, r.status);
            __syncthreads();
            const uint32_t n_tok2 = (here + 1) / 2, tasks = e1 > e0 ? (pairs_a + (n_f32 + 1) / 2) * n_tok2 : 0u;
            if (warp < tasks && !wait_slot(smem_u32(rows_here), 0)) give_up();
            for (uint32_t task = warp; task < tasks; task += kWarps + kFinish) {
                const uint32_t rp = task / n_tok2, tp = (task - rp * n_tok2) * 2;
                const uint32_t tp2 = min(tp + 1, here - 1), ta = t0 + s0 + tp, tb = t0 + s0 + tp2;
                const uint32_t xa = xs_at + tp * x_bytes, xb = xs_at + tp2 * x_bytes;
                float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
                uint32_t ea, eb;
                if (rp < pairs_a) {
                    const uint32_t ja = 2 * rp, jb = min(ja + 1, n_exp - 1);
                    ea = e0 + ja; eb = e0 + jb;
                    dots_affine(ring0 + ja * row_bytes, ring0 + jb * row_bytes, sb_at + ja * groups * 8, sb_at + jb * groups * 8, xa, xb, groups, r.bits, lane, acc);
                } else {
                    const uint32_t ja = 2 * (rp - pairs_a), jb = min(ja + 1, n_f32 - 1);
                    ea = e0 + n_exp - n_f + ja; eb = e0 + n_exp - n_f + jb;
                    dots_f32(f_at + ja * D * 4, f_at + jb * D * 4, xa, xb, quads, lane, acc);
                }
                if (r.eff_scale && eb == r.ne) {   // the gate row takes no column scale
                    const uint32_t w = gate_at;
                    float ga = 0.f, gb = 0.f;
#pragma unroll 1
                    for (uint32_t c = lane; c < quads; c += 32) {
                        uint32_t wr[4];
                        float xf[4], xg[4];
                        lds_packed<4>(w + c * 16, wr);
                        load_act4((const uint8_t*)r.hidden + ta * x_stride, c, r.dt, xf);
                        load_act4((const uint8_t*)r.hidden + tb * x_stride, c, r.dt, xg);
#pragma unroll
                        for (int i = 0; i < 4; ++i) { ga = __fmaf_rn(__uint_as_float(wr[i]), xf[i], ga); gb = __fmaf_rn(__uint_as_float(wr[i]), xg[i], gb); }
                    }
                    acc[1][0] = ga; acc[1][1] = gb;
                    if (ea == r.ne) { acc[0][0] = ga; acc[0][1] = gb; }
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) acc[k >> 1][k & 1] = butterfly_sum(acc[k >> 1][k & 1]);
                if (lane < 4) {
                    const float v = lane == 0 ? acc[0][0] : lane == 1 ? acc[0][1] : lane == 2 ? acc[1][0] : acc[1][1];
                    const uint32_t e = lane >> 1 ? eb : ea, tk = lane & 1 ? tb : ta;
                    if (e == r.ne) r.gate_out[tk] = sigmoid_det(v);
                    else r.logits[(size_t)tk * r.ne + e] = v;
                }
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the ring's next writers are copies
        if (!grid_sync(a.arrived)) give_up();
        const bool ready = io == 1u || io == 3u;
        for (uint32_t row = warp; row < a.T; row += kWarps + kFinish) {
            uint32_t id;
            float w;
            select_row_ranked<true>(r.logits + (size_t)row * r.ne, r, lane, rs.row[warp], id, w);
            const uint32_t p = row * r.top_k + lane, e = min(id, r.ne - 1u);
            bool live = false;
            if (lane < r.top_k) {
                const uint64_t word = rs.word[e];
                uint32_t slot = (uint32_t)(word & 0xffffffffu);
                if ((uint32_t)(word >> 32) != 2u) slot = SHRIKE_SLOT_MISS;
                const bool inside = slot < r.pool_cells;
                live = inside && ready;
                tab.weight[p] = w;
                if (live) {
                    rs.cell[e] = slot;
                    atomicOr(&rs.mask[p >> 5][e], 1u << (p & 31u));
                }
                if (blockIdx.x == row) {
                    r.ids[p] = id;
                    r.weights[p] = w;
                    if (r.slots) r.slots[p] = slot;
                    if (slot != SHRIKE_SLOT_MISS && !inside) report_status(a.status, kStatusBadIndex);
                }
            }
            const uint32_t bits = __ballot_sync(0xffffffffu, live);
            if (lane == 0) tab.live[row] = (uint8_t)bits;
        }
        __syncthreads();
        uint32_t cnt = 0, incl = 0;   // thread e: pairs of expert e, and {instances, pairs} of the experts up to it
        if (tid < SHRIKE_MAX_EXPERTS) {
            for (uint32_t w = 0; w < n_words; ++w) cnt += __popc(rs.mask[w][tid]);
            incl = ((cnt + 7) / 8) << 16 | cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += v;
            }
            if (lane == 31) tab.warp_sum[warp] = incl;
        }
        __syncthreads();
        uint32_t before = 0, total = 0;
#pragma unroll
        for (uint32_t w = 0; w < SHRIKE_MAX_EXPERTS / 32; ++w) {
            const uint32_t v = tab.warp_sum[w];
            if (w < warp) before += v;
            total += v;
        }
        n_inst = n_sh + (total >> 16);
        if (cnt) {
            const uint32_t ni = (cnt + 7) / 8, at = before + incl - (ni << 16 | cnt), i0 = n_sh + (at >> 16), p0 = at & 0xffffu;
            for (uint32_t c = 0; c < ni; ++c) {
                tab.cell[i0 + c] = rs.cell[tid];
                tab.first[i0 + c] = (uint16_t)(p0 + 8 * c);
                tab.count[i0 + c] = (uint8_t)min(8u, cnt - 8 * c);
            }
            uint32_t j = p0;
            for (uint32_t w = 0; w < n_words; ++w)
                for (uint32_t m = rs.mask[w][tid]; m; m &= m - 1) tab.sorted[j++] = (uint16_t)(w * 32 + __ffs(m) - 1);
        }
    } else {
        pdl_wait();
        pdl_launch_dependents();
        n_inst = min(*a.n_inst, kMaxTable);
        for (uint32_t j = tid; j < kMaxTable; j += kThreads) {
            const uint4 h = *(const uint4*)&a.inst[j < n_inst ? j : 0];
            if (j < n_inst) { tab.cell[j] = h.y; tab.first[j] = (uint16_t)h.z; tab.count[j] = (uint8_t)h.w; }
        }
        for (uint32_t j = tid; j < a.T * a.top_k; j += kThreads) tab.sorted[j] = (uint16_t)a.sorted[j];
        if ((a.phases & 2u) && tid < a.T) {
            uint32_t live = 0;
            for (uint32_t q = 0; q < a.top_k; ++q)
                if (a.pair_cell[tid * a.top_k + q] != SHRIKE_SLOT_MISS) live |= 1u << q;
            tab.live[tid] = (uint8_t)live;
        }
    }
    if (tid < n_sh) {
        tab.cell[tid] = 0;
        tab.first[tid] = (uint16_t)(8 * tid);
        tab.count[tid] = (uint8_t)min(8u, a.T - 8 * tid);
    }
    return n_inst;
}

}  // namespace

template <int BITS, int GROUP, int META, bool AL>
__global__ void __launch_bounds__(kThreads, 1) expert_stream_kernel(const __grid_constant__ StreamArgs a, const __grid_constant__ PieceMaps maps) {
    using Q = FQ<BITS, GROUP>;
    constexpr uint32_t GP = 128 / Q::kGroupBytes, H = GROUP / 32;   // groups of a piece; 16-byte operand parts of a group
    // The warps of a team share a row by whole pieces, or by halves of pieces of eight groups where rows end within a piece: of 12
    // pieces (2880 columns in groups of 32) eight warps have one or two, of 23 halves two or three. 32 experts of 2880 x 2880, 64 rows, us
    // over four layers: 960 by pieces, 848 by halves (970 by pieces with initial values of 16 bytes a lane instead of 8: half of the
    // loops' cycles are reads of shared memory). The parts of a row's sum meet in another order, no further off: error against 64 bits 7.2e-5
    // by pieces, 7.1e-5 by halves, fp32 rows, 2 to 64 of them alike.
    constexpr uint32_t kHalves = GP == 8 && !AL ? 2 : 1;
    extern __shared__ __align__(128) uint8_t dsm_raw[];
    uint8_t* const dsm = dsm_raw + ((1024u - (smem_u32(dsm_raw) & 1023u)) & 1023u);   // the swizzle follows the address
    __shared__ uint64_t full1[kMaxSlots], done1[kMaxSlots], full2[kMaxSlots2], done2[kMaxSlots2];
    __shared__ uint64_t rows_here;
    __shared__ StreamTable tab;
    __shared__ uint32_t s_failed;
    const StreamGeom& G = a.g;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    uint8_t* const ring = dsm + G.off_ring;
    const uint32_t dsm0 = smem_u32(dsm), ring0 = smem_u32(ring);
    const uint32_t D = a.d;
    const bool do1 = a.phases & 1u, do2 = a.phases & 2u;

    if (tid < G.n_slots) { mbar_init(&full1[tid], 1); mbar_init(&done1[tid], G.w1); }
    if (tid < G.n_slots2) { mbar_init(&full2[tid], 1); mbar_init(&done2[tid], G.w2); }
    if (tid == 0) mbar_init(&rows_here, 1);
    if (tid < kMaxSlots2) fence_mbar_init();
    if (tid == 0) s_failed = 0;
    // (no prefetch of the tensor maps here: fetched ahead by a warp of each block they cost 1.2 us of a layer of 4 rows, 38.6 us
    // against 37.4, and 0.7 of one of 16; the first copies come long after, behind the routing)
    __syncthreads();
    auto give_up = [&]() {
        report_status(a.status, kStatusWaitTimeout);
        s_failed = 1;
    };
    const uint32_t n_inst = work_list(a, dsm, ring, tab, &rows_here, &s_failed);
    const uint32_t n_sh = min(a.n_shared, n_inst);
    __syncthreads();
    const float* const pair_weight = a.phases == 3u ? tab.weight : a.route_w;
    // the row of pairs (shared: of rows) behind column c of instance i
    auto pair_of = [&](uint32_t i, uint32_t c) -> uint32_t { return i < n_sh ? tab.first[i] + c : tab.sorted[tab.first[i] + c]; };
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
        const uint32_t each = quotient(total, a.rcp_grid), over = total - each * gridDim.x;
        const uint32_t v0 = each * blockIdx.x + min(blockIdx.x, over), n = each + (blockIdx.x < over ? 1u : 0u);
        const uint32_t rcp_su = P1 ? a.rcp_su : a.rcp_u2, rcp_ru = P1 ? a.rcp_ru : a.rcp_u2;
        auto find = [&](uint32_t j, uint32_t& i, uint32_t& k) {   // unit j -> instance, unit in it
            const uint32_t v = v0 + j;
            if (v < sh_units) { i = quotient(v, rcp_su); k = v - i * su; }
            else { const uint32_t w = v - sh_units, q = quotient(w, rcp_ru); i = n_sh + q; k = w - q * ru; }
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
        auto ask = [&](uint32_t slot, uint32_t i, uint32_t k) {
            const bool sh = i < n_sh;
            const uint32_t cell = sh ? 0u : tab.cell[i], ch = __umulhi(cell, a.rcp_cpc);
            const uint32_t mi = sh ? SHRIKE_MAX_POOL_CHUNKS : ch;
            const int32_t cc = sh ? 0 : (int32_t)(cell - ch * a.pool.cells_per_chunk);
            const uint8_t* base = sh || !a.expert_bias ? a.shared_block : pool_cell_base(a.pool, cell);
            const Offsets3& off = sh ? a.shared : a.routed;
            if constexpr (P1) {
                uint64_t* bar = &full1[slot];
                const uint32_t at = slot * G.slot_bytes;
                mbar_expect_tx(bar, 2048 * ((D * BITS / 8 + 127) / 128) + 64 * (D / GROUP) + (a.expert_bias ? 32u : 0u));
                tma_5d_once(ring0 + at + G.meta_off, &maps.m1[mi], 0, (int32_t)k, 0, 0, cc, bar, evict_first_policy());
                tma_5d_once(ring0 + at, &maps.l1[mi], 0, (int32_t)(k * 8), 0, 0, cc, bar, evict_first_policy());
                if (a.expert_bias) {
                    bulk_g2s(ring + at + G.ab_off, base + off.ab[0] + (size_t)k * 16, 16, bar);
                    bulk_g2s(ring + at + G.ab_off + 16, base + off.ab[1] + (size_t)k * 16, 16, bar);
                }
            } else {
                const uint32_t F = sh ? a.f_shared : a.f, mt = G.n_slots2 * G.w_bytes2 + slot * G.m_bytes2;
                uint64_t* bar = &full2[slot];
                mbar_expect_tx(bar, 2048 * ((F * BITS / 8 + 127) / 128) + 64 * (F / GROUP) + (a.expert_bias ? 32u : 0u));
                tma_4d_once(ring0 + mt, &maps.m2[mi], 0, (int32_t)(k * 2), 0, cc, bar, evict_first_policy());
                tma_4d_once(ring0 + slot * G.w_bytes2, &maps.l2[mi], 0, (int32_t)(k * 16), 0, cc, bar, evict_first_policy());
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
        const uint32_t meta0 = ring0 + (P1 ? G.meta_off : G.n_slots2 * G.w_bytes2);

        uint32_t i0 = 0, i_end = 0;   // the first staged instance, the end of the block's
        if (n) {
            uint32_t dummy;
            find(0, i0, dummy);
            find(n - 1, i_end, dummy);
            ++i_end;
        }
        // (W == 1: the warps finish their units themselves; fewer teams than finishing warps: some have none)
        uint32_t u = finisher && (W == 1 || team >= nT) ? n : team, slot = team, par = 0;
        uint32_t i = 0, k = 0;        // unit u: instance, unit in it
        if (u < n) find(u, i, k);
        bool later = false;
        while (i0 < i_end) {
            // every warp works out for itself which instances fit: lane l has instance i0 + l
            uint32_t at = 0, i1 = i0;
            {
                const uint32_t ii = i0 + lane;
                uint32_t bytes = 0;
                if (ii < i_end) {
                    const uint32_t K = P1 ? D : ii < n_sh ? a.f_shared : a.f;
                    bytes = BufferLayout(K / GROUP, H, tab.count[ii]).bytes;
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
            {   // the instances' groups, in shares of neighbours over all warps (two or more at a time cost registers that the
                // loops below then spill: 16 rows 500 us over eight layers, 508 and 516)
                const uint32_t n_s = i0 < n_sh ? min(n_sh, i1) - i0 : 0u;
                const uint32_t gs = ((P1 ? D : a.f_shared) / GROUP + 3) & ~3u, gr = ((P1 ? D : a.f) / GROUP + 3) & ~3u;
                const uint32_t all = n_s * gs + (i1 - i0 - n_s) * gr;
                uint32_t left = all * (warp + 1) / (kWarps + kFinish), ii = i0, j = all * warp / (kWarps + kFinish);
                left -= j;
                while (left) {
                    const bool sh = ii < n_sh;
                    const uint32_t g4 = sh ? gs : gr;
                    if (j >= g4) {
                        j -= g4;
                        ++ii;
                        continue;
                    }
                    const uint32_t groups = (P1 ? D : sh ? a.f_shared : a.f) / GROUP, cnt = tab.count[ii];
                    const uint32_t p = pair_of(ii, min(g, cnt - 1u));   // past the count: the last row
                    const uint16_t* row;
                    if constexpr (P1) {
                        row = a.xh + (size_t)(sh ? p : quotient(p, a.rcp_top_k)) * D;
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
                    const uint32_t buf = dsm0 + __shfl_sync(0xffffffffu, at, ii - i0);
                    const BufferLayout lay(groups, H, cnt);
                    const uint32_t end = min(j + left, g4);
                    left -= end - j;
                    for (; j < end; ++j) {
                        uint32_t x[GROUP / 8];
                        if (j < groups) load_group<GROUP>(row, j, t, x);
                        stage_group<BITS, GROUP>(x, j, groups, cnt, buf, lay, lane);
                    }
                }
            }
            __syncthreads();
            // The units of the staged instances, by what the warp does with them (a copy of the loop each: it holds only
            // that role's registers): multiplies, finishes, or, in a team of one, both.
            auto units = [&](auto role) {
                constexpr bool MUL = decltype(role)::value != 1, FIN = decltype(role)::value != 0, ONE = MUL && FIN;
                uint32_t cur = 0xffffffffu, count = 0, groups_left = 0, pieces = 0, first_half = 0;
                uint32_t b0 = 0, cq0 = 0, z0 = 0, sB = 0, w_at = 0, s_at = 0, ab_at = 0, d_s = 0, d_z = 0, k0 = 0;
                uint16_t* dst = nullptr;   // gate/up: where column g's activations go
                float* out0 = nullptr;     // down: where the rows of column g (ONE: columns 2t and 2t + 1) go, and their weights
                float* out1 = nullptr;
                float wt0 = 0.f, wt1 = 0.f;
                uint32_t pend = 0;         // units of `cur` whose activations this warp wrote and has not announced
                auto announce = [&]() {
                    if (P1 && FIN && do2 && pend) {
                        __syncwarp();
                        if (lane == 0) asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(a.inst_done + cur), "r"(pend) : "memory");
                        pend = 0;
                    }
                };
                auto open_instance = [&](uint32_t buf) {
                    cur = i;
                    const bool sh = i < n_sh;
                    count = tab.count[i];
                    const uint32_t col = min(g, count - 1u);
                    if constexpr (MUL) {
                        const uint32_t K = P1 ? D : sh ? a.f_shared : a.f, G2 = K / GROUP, P = (G2 + GP / kHalves - 1) / (GP / kHalves);
                        const uint32_t h0 = P * wi / W, h1 = P * (wi + 1) / W, p0 = h0 / kHalves;
                        first_half = h0 % kHalves;
                        pieces = h1 > h0 ? (h1 + kHalves - 1) / kHalves - p0 : 0u;
                        groups_left = (kHalves == 1 ? G2 : min(G2, h1 * 4)) - min(G2, h0 * (GP / kHalves));
                        const BufferLayout lay(G2, H, count);
                        sB = count * 64;
                        b0 = buf + col * 64 + t * 16 + h0 * (GP / kHalves) * H * sB;
                        cq0 = buf + lay.cq_off + t * 8 + h0 * (GP / kHalves) * 32;
                        z0 = buf + lay.z_off + col * 64 + t * 16 + (GP == 2 ? h0 / 2 : h0 * (GP / kHalves / 4)) * sB;
                        k0 = GP == 2 ? 2 * (h0 & 1) : 0u;
                        w_at = (ring0 + w_lane + p0 * 2048) ^ (first_half * 64);
                        s_at = meta0 + (pr * G2 + h0 * (GP / kHalves)) * 2;
                        d_s = P1 ? 32 * G2 : 16 * G2;
                        d_z = P1 ? 16 * G2 : 32 * G2;
                        ab_at = meta0 - (P1 ? G.meta_off : 0u) + (P1 ? G.ab_off : G.ab_off2[sh]) + pr * 2;
                    }
                    if constexpr (FIN && P1) {
                        const uint32_t pair = pair_of(i, col);
                        const uint32_t F = sh ? a.f_shared : a.f;
                        dst = g < count ? (sh ? a.acts_shared : a.acts) + (size_t)pair * F + (BITS == 4 ? 2 * t : t) : nullptr;
                    } else if constexpr (FIN) {
                        auto target = [&](uint32_t c, float*& out, float& w) {
                            const uint32_t pair = pair_of(i, min(c, count - 1u));
                            w = sh ? (a.shared_gate ? __ldcg(a.shared_gate + pair) : 1.0f) : pair_weight[pair];
                            float* rows = a.parts + ((size_t)pair + (sh ? a.T * a.top_k : 0u)) * D;
                            out = c < count ? rows + (ONE ? pr : t) : nullptr;
                        };
                        target(ONE ? 2 * t : g, out0, wt0);
                        if constexpr (ONE) target(2 * t + 1, out1, wt1);
                    }
                };
                for (; u < n && i < i1; u += pace) {
                    if (i != cur) {
                        announce();
                        open_instance(dsm0 + __shfl_sync(0xffffffffu, at, i - i0));
                    }
                    const uint32_t bar_at = slot * 8, rb = dsm0 + G.off_red + slot * W * (kRedWarp * 4);
                    float acc[4] = {0.f, 0.f, 0.f, 0.f};
                    if constexpr (MUL) {
                        if (!try_slot(full + bar_at, par) && !wait_slot_slow(full + bar_at, par)) give_up();
                        const uint32_t mo = slot * (P1 ? G.slot_bytes : G.m_bytes2);
                        if (a.expert_bias && wi == 0) {
                            acc[0] = acc[1] = bf16_bits_to_f32((uint16_t)lds16(ab_at + mo));
                            acc[2] = acc[3] = bf16_bits_to_f32((uint16_t)lds16(ab_at + mo + 16));
                        }
                        uint32_t w = w_at + slot * (P1 ? G.slot_bytes : G.w_bytes2), sc = s_at + mo, b = b0, cq = cq0, z = z0, kk = k0, left = groups_left;
                        uint32_t cap = kHalves == 2 && first_half ? GP / 2 : GP;   // groups from here to the piece's end
#pragma unroll 1
                        for (uint32_t p = 0; p < pieces; ++p) {
                            piece_tiles<BITS, GROUP, META, !AL>(w, sc, d_s, d_z, b, cq, z, sB, min(cap, left), kk, t, acc);
                            w = (kHalves == 2 && cap != GP ? w ^ 64u : w) + 2048;
                            sc += 2 * cap;
                            b += cap * H * sB;
                            cq += cap * 32;
                            if constexpr (GP == 2) {
                                kk ^= 2u;
                                z += kk ? 0u : sB;
                            } else {
                                z += cap / 4 * sB;
                            }
                            left -= cap;
                            if constexpr (kHalves == 2) cap = GP;
                        }
                        if (P1 || !ONE) {
                            const uint32_t to = rb + wi * (kRedWarp * 4) + my_red;
                            sts32(to, acc[0]);
                            sts32(to + kRedCol * 4, acc[1]);
                            sts32(to + 8, acc[2]);
                            sts32(to + kRedCol * 4 + 8, acc[3]);
                        }
                        __syncwarp();
                        if (!FIN && lane == 0) arrive(done + bar_at);
                    } else {
                        if (!try_slot(done + bar_at, par) && !wait_slot_slow(done + bar_at, par)) give_up();
                    }
                    if constexpr (FIN) {
                        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);   // column g, rows t, t + 4, t + 8, t + 12
                        if (P1 || !ONE) {
#pragma unroll 4
                            for (uint32_t w = 0; w < (ONE ? 1u : W); ++w) {
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
                        } else if constexpr (ONE) {
                            if (out0) {
                                *(out0 + k * 16) = wt0 * acc[0];
                                *(out0 + k * 16 + 8) = wt0 * acc[2];
                            }
                            if (out1) {
                                *(out1 + k * 16) = wt1 * acc[1];
                                *(out1 + k * 16 + 8) = wt1 * acc[3];
                            }
                        } else if (out0) {
                            float* o = out0 + k * 16;
                            *o = wt0 * v.x;
                            *(o + 4) = wt0 * v.y;
                            *(o + 8) = wt0 * v.z;
                            *(o + 12) = wt0 * v.w;
                        }
                    }
                    step(i, k);
                    slot += pace;
                    if (slot >= n_slots) { slot -= n_slots; par ^= 1u; }
                }
                announce();
            };
            if (finisher) units(std::integral_constant<int, 1>());
            else if (W == 1) units(std::integral_constant<int, 2>());
            else units(std::integral_constant<int, 0>());
            i0 = i1;
        }
    };

    if (do1) phase(std::integral_constant<int, 1>());
    __syncthreads();   // the ring changes hands
    if (do2) phase(std::integral_constant<int, 2>());
    if (s_failed) {
        // a copy of this block may still be in flight: give it a bounded time to land
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
    }
    if (!do2) return;
    // ================= y = the rows' parts; hidden += y =================
    // one output element pair per thread over all blocks; what does not depend on the parts is read ahead of the wait
    // (warps go round the blocks, so that a small call keeps every SM busy)
    const uint32_t half = D / 2, items = a.T * half, stride = gridDim.x * kThreads;
    uint32_t j = (warp * gridDim.x + blockIdx.x) * 32 + lane;
    uint32_t live = 0;
    float h0 = 0.f, h1 = 0.f;
    if (j < items) {
        live = tab.live[quotient(j, a.rcp_half)];
        if (a.hidden) {
            h0 = load_act(a.hidden, (size_t)j * 2, a.act_dtype);
            h1 = load_act(a.hidden, (size_t)j * 2 + 1, a.act_dtype);
        }
    }
    if (!grid_sync(a.arrived)) give_up();
    for (bool first = true; j < items; j += stride, first = false) {
        const uint32_t tk = quotient(j, a.rcp_half), c = j - tk * half;
        if (!first) live = tab.live[tk];
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
// What quotient() takes for a division by d (nothing is divided by a zero).
inline uint32_t reciprocal(uint32_t d) { return d < 2 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d); }

// Shared-memory layout; false when the shape does not fit.
bool stream_geometry(const shrike_moe_config& c, uint32_t smem_optin, StreamGeom& g) {
    memset(&g, 0, sizeof g);
    const uint32_t G1 = c.d / c.group_size, G2 = c.f / c.group_size, Gs = c.has_shared ? c.shared_f / c.group_size : 0;
    if ((G1 | G2 | Gs) & 1u) return false;   // rows of scales are read as 32-bit words
    auto pieces = [&](uint32_t K) { return (K * c.weight_bits / 8 + 127) / 128; };
    auto buffer = [&](uint32_t groups) { return groups * (c.group_size / 32) * 512 + (groups + 3) / 4 * 512 + (groups * 32 + 15) / 16 * 16; };   // eight columns
    g.meta_off = 2048 * pieces(c.d);
    g.ab_off = align_up(g.meta_off + 64 * G1, 128);
    g.slot_bytes = align_up(g.ab_off + (c.expert_bias ? 128 : 0), 1024);
    for (int sh = 0; sh < (c.has_shared ? 2 : 1); ++sh) {
        const uint32_t F = sh ? c.shared_f : c.f;
        g.w_bytes2 = std::max(g.w_bytes2, 2048 * pieces(F));
        g.ab_off2[sh] = align_up(64 * (F / c.group_size), 128);
        g.m_bytes2 = std::max(g.m_bytes2, g.ab_off2[sh] + (c.expert_bias ? 128u : 0u));
    }
    const uint32_t least = std::max({buffer(G1), buffer(std::max(G2, Gs)), (uint32_t)sizeof(RouteScratch)}), most_pieces2 = g.w_bytes2 / 2048;
    const uint32_t budget = smem_optin - kStaticBytes - 1024;   // less the static part and the ring's alignment
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
    // quotient()'s products: units of all instances times those of one or the blocks, pairs of elements times those of a row
    const uint64_t units = std::max(std::max(c.f, c.has_shared ? c.shared_f : 0u) / 8, c.d / 16);
    if (kMaxTable * units * std::max<uint64_t>(units, 4096) >= 1ull << 32 || (uint64_t)SHRIKE_MAX_DECODE_TOKENS * c.d / 2 * (c.d / 2) >= 1ull << 32) return false;
    const uint32_t ring = std::max(g.n_slots * g.slot_bytes, g.n_slots2 * (g.w_bytes2 + g.m_bytes2));
    const uint32_t red = std::max(g.n_slots * g.w1, g.w2 > 1 ? g.n_slots2 * g.w2 : 0u) * kRedWarp * 4;
    if (ring + red + least > budget) return false;
    g.off_ring = (budget - ring) / 1024 * 1024;
    if (g.off_ring < red + least) return false;
    g.off_red = (g.off_ring - red) / 128 * 128;
    if (g.off_red < least) return false;
    g.ring_bytes = ring;
    g.smem_bytes = g.off_ring + ring + 1024;
    return true;
}

template <int BITS, int GROUP, int META, bool AL>
cudaError_t launch_stream_t(const shrike_moe* m, cudaStream_t st, const StreamArgs& a, const PieceMaps& maps, bool pdl) {
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
    if (a.phases & 2u) {   // the blocks wait for each other
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
    return cudaLaunchKernelEx(&cfg, k, a, maps);
}

template <int BITS, int GROUP, int META>
cudaError_t launch_stream_m(const shrike_moe* m, cudaStream_t st, const StreamArgs& a, const PieceMaps& maps, bool pdl) {
    // every row whole 128-byte pieces?
    const shrike_moe_config& c = m->cfg;
    const uint32_t gp = 128 / (GROUP * BITS / 8);
    const bool al = c.d / GROUP % gp == 0 && c.f / GROUP % gp == 0 && (!c.has_shared || c.shared_f / GROUP % gp == 0);
    return al ? launch_stream_t<BITS, GROUP, META, true>(m, st, a, maps, pdl) : launch_stream_t<BITS, GROUP, META, false>(m, st, a, maps, pdl);
}

}  // namespace

// Whether calls of some rows run here, pools of single-cell chunks and parts of a GPU aside.
bool stream_takes_shape(const shrike_moe* m) {
    StreamGeom g;
    return stream_geometry(m->cfg, m->smem_optin, g);
}

size_t stream_parts_bytes(const shrike_moe_config& c) {
    const size_t T = std::min(c.max_tokens, (uint32_t)SHRIKE_MAX_DECODE_TOKENS);
    return T * (c.top_k + (c.has_shared ? 1u : 0u)) * c.d * 4;
}

size_t stream_done_bytes() { return kMaxTable * 4; }

// How many groups the call's rows form for the logits: with more than a few rows a block takes a part of them against more
// expert rows. Its own activation rows are what it waits for (us over eight layers, 16 rows: 1 group 529, 2 groups 516, 4 groups 508;
// over four layers of 32 experts of 2880 x 2880, 64 rows: 4 groups 989, 8 groups 968). 0 when a
// block's rows of the router do not fit into the ring, or there is no block for every row (block t writes row t's picks): both
// only on a part of a GPU.
static uint32_t stream_token_groups(const shrike_moe_config& c, uint32_t sm_count, uint32_t T, uint32_t ring_bytes) {
    const uint32_t rows = c.num_experts + (c.shared_gated ? 1u : 0u), bits = c.router_weight_bits;
    const uint32_t row_bytes = bits ? c.d * bits / 8 + c.d / 64 * 8 : c.d * 4;
    if (T > sm_count) return 0;
    for (uint32_t n = T <= 2 ? 1 : T <= 4 ? 2 : T <= 16 ? 4 : 8; n; n /= 2) {
        const uint32_t nbx = sm_count / n, most = (rows + nbx - 1) / nbx;
        if (nbx && most * row_bytes + c.d * 4 + 16 + 2 * c.d * 4 <= ring_bytes) return n;
    }
    return 0;
}

// phases: 1 or 2, by the plan of an earlier launch, or both, with `route`: the launch then routes the rows itself.
// cudaErrorNotSupported when the shape does not fit: nothing was launched.
cudaError_t launch_expert_stream(const shrike_moe* m, cudaStream_t st, const ExpertArgs& ea, uint32_t T, uint32_t n_shared,
                                 void* y, void* hidden, bool pdl, uint32_t phases, const RouterArgs* route) {
    const shrike_moe_config& c = m->cfg;
    const uint64_t cpc = ea.pool.cells_per_chunk ? ea.pool.cells_per_chunk : 1;
    if (cpc < 2 || (uint64_t)ea.pool.cells * cpc >= (1ull << 32)) return cudaErrorNotSupported;
    const PieceMaps* maps = piece_maps_for(m, ea);
    if (!maps) return cudaErrorNotSupported;
    StreamArgs a;
    memset(&a, 0, sizeof a);
    if (!stream_geometry(c, m->smem_optin, a.g)) return cudaErrorNotSupported;
    a.pool = ea.pool; a.routed = ea.routed; a.shared = ea.shared; a.shared_block = ea.shared_block;
    a.d = c.d; a.f = c.f; a.f_shared = c.has_shared ? c.shared_f : 0; a.top_k = c.top_k;
    a.activation = c.activation; a.expert_bias = c.expert_bias; a.act_dtype = c.act_dtype; a.y_dtype = c.y_dtype;
    a.inst = ea.inst; a.n_inst = ea.n_inst; a.n_shared = n_shared;
    a.xh = ea.xh; a.acts = ea.acts; a.acts_shared = ea.acts_shared;
    a.parts = m->ws.parts; a.sorted = ea.sorted; a.pair_cell = m->ws.pair_cell;
    if (route) {
        a.r = *route;
        const uint32_t groups = stream_token_groups(c, m->sm_count, T, a.g.ring_bytes);
        if (!groups) return cudaErrorNotSupported;
        while ((2u << a.token_groups_log2) <= groups) ++a.token_groups_log2;
        a.rcp_nbx = reciprocal(m->sm_count / groups);
    }
    a.route_w = ea.route_w; a.shared_gate = ea.shared_gate; a.status = ea.status; a.arrived = m->ws.arrived; a.inst_done = m->ws.inst_done;
    a.T = T; a.y = y; a.hidden = hidden; a.phases = phases;
    a.rcp_cpc = (uint32_t)(((1ull << 32) + cpc - 1) / cpc);
    a.rcp_grid = reciprocal(m->sm_count);
    a.rcp_su = reciprocal(a.f_shared / 8);
    a.rcp_ru = reciprocal(c.f / 8);
    a.rcp_u2 = reciprocal(c.d / 16);
    a.rcp_top_k = reciprocal(c.top_k);
    a.rcp_half = reciprocal(c.d / 2);
    const uint32_t bits = c.weight_bits, grp = c.group_size;
    const bool f16 = c.meta_dtype == SHRIKE_DTYPE_FP16;
    if (bits == 4 && grp == 64 && !f16) return launch_stream_m<4, 64, SHRIKE_DTYPE_BF16>(m, st, a, *maps, pdl);
    if (bits == 4 && grp == 64 && f16) return launch_stream_m<4, 64, SHRIKE_DTYPE_FP16>(m, st, a, *maps, pdl);
    if (bits == 4 && grp == 32 && !f16) return launch_stream_m<4, 32, SHRIKE_DTYPE_BF16>(m, st, a, *maps, pdl);
    if (bits == 4 && grp == 32 && f16) return launch_stream_m<4, 32, SHRIKE_DTYPE_FP16>(m, st, a, *maps, pdl);
    if (bits == 8 && grp == 64 && !f16) return launch_stream_m<8, 64, SHRIKE_DTYPE_BF16>(m, st, a, *maps, pdl);
    if (bits == 8 && grp == 64 && f16) return launch_stream_m<8, 64, SHRIKE_DTYPE_FP16>(m, st, a, *maps, pdl);
    if (bits == 8 && grp == 32 && !f16) return launch_stream_m<8, 32, SHRIKE_DTYPE_BF16>(m, st, a, *maps, pdl);
    if (bits == 8 && grp == 32 && f16) return launch_stream_m<8, 32, SHRIKE_DTYPE_FP16>(m, st, a, *maps, pdl);
    return cudaErrorInvalidValue;
}

}  // namespace shrike
