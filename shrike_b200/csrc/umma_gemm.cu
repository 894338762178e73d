// Ragged prefill on the 5th-generation tensor cores: an expert-grouped GEMM with
// the dequantisation in the producer warps (the B200 counterpart of
// mpp_prefill_affine_grouped_f16, tensorops.metal:145-248, and of
// encodeGroupedExpertGEMMs, PrefillGroupedRoutedMoE.swift:925-1035).
//
// One tile = 256 weight rows of one expert against up to 256 of the rows routed
// to it ("swap-AB": the weights are the M operand -- two 128-row tiles, each
// with its own TMEM accumulator -- and the activation rows the N operand, so an
// expert with few rows still fills the MMA's M dimension). A 256 x 256 block
// reads each activation byte once per 256 weight rows and dequantises each
// weight once per 256 activation rows.
//
//   warp 18    one thread streams the packed weights (64 bytes of every row
//              per copy: a 3-D TMA box of 128 rows of one matrix of one pool
//              cell, 64-byte swizzle) and the group scales / biases (16 bytes
//              of every row per copy) into shared-memory rings. Whole-line TMA
//              requests keep the packed experts streaming at HBM speed where
//              per-thread 32-byte loads ran out of outstanding requests.
//   warp 17    one thread copies the activation tiles: one or two boxes of 64 x
//              16 to 256 of the expert-sorted fp16 rows per K block, 128-byte
//              swizzle.
//   warps 0-15 converters: two threads per weight row; per 64-wide K block
//              they turn the packed nibbles/bytes into fp16 (q - Z) * scale +
//              (bias + Z*scale) -- the reference's half(fma(q, scale, bias)),
//              tensorops.metal:106 -- and write them to TMEM (instances of up
//              to 128 rows) or, 16 bytes at a time, into the K-major
//              128-byte-swizzled tile in shared memory that the MMA reads.
//              After the K loop the same warps run the epilogue.
//   warp 16    one elected thread issues tcgen05.mma (M 128, N = rows, K 16, fp16 in,
//              fp32 accumulate in TMEM) for both tiles and commits to the
//              mbarriers that free the converted tile and the activation tile.
//
// PHASE 0: tile 0 = 128 gate rows, tile 1 = the matching 128 up rows; epilogue
//          GLU -> fp16 activations in operand layout, one row per sorted pair.
// PHASE 1: tiles = 256 consecutive down rows; epilogue (+ additive bias) x route
//          weight -> red.global.add into the token's fp32 accumulator row (the
//          weighted reduce, with no per-(row, rank) partial rows in between).
//
// What bounds it (256 experts of 2048 x 512): a K block takes 0.43 us at 16 rows, the converters' chain of waits, loads,
// arithmetic and stores, and 0.74 to 0.76 us at 256 rows. That is 8.39 MFLOP on each of 148 SMs: 1.63 to 1.68 PFLOP/s, as fast as
// the measured burst rate of a library GEMM (1.67). What is left of full tiles lies outside the K loop: 9 of a down tile's 14 us.
//
// Every wait is bounded; a wait that gives up sets the status word and the
// block falls through to the TMEM release.
#include <cuda.h>
#include <algorithm>

#include "internal.h"

namespace shrike {

constexpr uint32_t kUmmaMaxN = 256;
constexpr int kActBoxes = 5;
constexpr uint32_t kConverters = 512;                  // two threads per weight row
constexpr uint32_t kConvWarps = kConverters / 32;
constexpr uint32_t kUmmaThreads = kConverters + 96;    // + MMA warp, activation-copy warp, weight-copy warp
constexpr uint32_t kAStages = 2, kMaxAStages = 4, kBStages = 3, kPkSlots = 3;   // kAStages: at the widest activation tile
constexpr uint32_t kTileBytes = 128 * 128;             // 128 rows x 64 fp16, one swizzle-128B K block
constexpr uint32_t kAStageBytes = 2 * kTileBytes;      // both weight tiles
constexpr uint32_t kBTileBytes = kUmmaMaxN * 128;      // 256 rows x 64 fp16
constexpr uint32_t kPkSlotBytes = 256 * 64;            // 64 packed bytes of 256 rows
constexpr uint32_t kScHalfBytes = 256 * 16;            // 8 scales (or biases) of 256 rows
constexpr uint32_t kOffA = kBStages * kBTileBytes;
constexpr uint32_t kOffPk = kOffA + kAStages * kAStageBytes;
constexpr uint32_t kOffSc = kOffPk + kPkSlots * kPkSlotBytes;
constexpr uint32_t kOffBar = kOffSc + 2 * kScHalfBytes;
constexpr uint32_t kNumBars = 2 * kMaxAStages + 2 * kBStages + 2 * kPkSlots + 3 + 5;
constexpr uint32_t kUmmaSmemBytes = kOffBar + kNumBars * 8 + 4 * kUmmaMaxN * 4 + 16 + 1024 /*alignment slack*/;

struct WeightMaps {       // TMA descriptors of the two 128-row tiles of a block
    CUtensorMap w[2];     // packed weights   [cells][rows][row bytes]
    CUtensorMap s[2];     // group scales     [cells][rows][groups]
    CUtensorMap b[2];     // group biases
};
struct UmmaMaps {
    WeightMaps routed[SHRIKE_MAX_POOL_CHUNKS];
    WeightMaps shared;
    CUtensorMap act_routed[kActBoxes], act_shared[kActBoxes];   // boxes of 16, 32, 64, 128 and 256 activation rows
};

// ---- tcgen05 wrappers -------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// The same with A in TMEM: row = lane, two fp16 a column.
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// One lane of the converged warp, the same one every time.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// K-major, 128-byte swizzle, rows packed at 128 bytes: 8-row atoms 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);   // start address
    d |= (uint64_t)1 << 16;                          // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;                // stride byte offset
    d |= (uint64_t)1 << 46;                          // descriptor version
    d |= (uint64_t)2 << 61;                          // 128-byte swizzle
    return d;
}
// D fp32, A/B fp16, both K-major, M 128, N n.
__device__ __forceinline__ uint32_t umma_idesc(uint32_t n) {
    return (1u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}

// 8 packed nibbles -> 8 fp16 weights in operand order {0,4,1,5,2,6,3,7}; 4 bytes -> 4 fp16 in order.
template <int BITS>
__device__ __forceinline__ void dequant_word(uint32_t w, uint32_t s2, uint32_t z2, uint32_t* out) {
    if constexpr (BITS == 4) {
        // nibbles j and j + 4 of the word make pair j. A nibble in bits 0..3 of a half is read as the fp16
        // value 1024 + q, one in bits 4..7 as 64 + q (64's unit in the last place sits at bit 4): one shift
        // per word instead of three.
        const uint32_t v = w >> 8;
        const uint32_t h0 = hsub2_u32(lop3_and_or(w, 0x000F000Fu, 0x64006400u), 0x64086408u);   // (1024 + q) - 1032
        const uint32_t h1 = hsub2_u32(lop3_and_or(w, 0x00F000F0u, 0x54005400u), 0x54805480u);   // (64 + q) - 72
        const uint32_t h2 = hsub2_u32(lop3_and_or(v, 0x000F000Fu, 0x64006400u), 0x64086408u);
        const uint32_t h3 = hsub2_u32(lop3_and_or(v, 0x00F000F0u, 0x54005400u), 0x54805480u);
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(out[0]) : "r"(h0), "r"(s2), "r"(z2));
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(out[1]) : "r"(h1), "r"(s2), "r"(z2));
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(out[2]) : "r"(h2), "r"(s2), "r"(z2));
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(out[3]) : "r"(h3), "r"(s2), "r"(z2));
    } else {
        const uint32_t lo = hsub2_u32(prmt(w, 0x64646464u, 0x5140u), 0x64806480u);
        const uint32_t hi = hsub2_u32(prmt(w, 0x64646464u, 0x5342u), 0x64806480u);
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(out[0]) : "r"(lo), "r"(s2), "r"(z2));
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(out[1]) : "r"(hi), "r"(s2), "r"(z2));
    }
}

__device__ __forceinline__ uint32_t half2_dup(float v) {
    const uint32_t h = __half_as_ushort(__float2half_rn(v));
    return h | (h << 16);
}

__device__ __forceinline__ void tmem_ld8_issue(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Tiled TMA loads (no multicast). x is the element column, then row, then cell.
__device__ __forceinline__ void tma_load_2d(uint32_t smem_dst, const CUtensorMap* map, int32_t x, int32_t y,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_dst), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t smem_dst, const CUtensorMap* map, int32_t x, int32_t y, int32_t z,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}

// SiLU / clamped-SwiGLU gates with the fast exponential and reciprocal: the
// epilogue runs one per output element, and the result is rounded to fp16.
__device__ __forceinline__ float glu_epilogue(float gate, float up, uint32_t activation) {
    if (activation == SHRIKE_ACT_CLAMPED_SWIGLU) {
        const float gc = fminf(gate, 7.0f);
        const float uc = fmaxf(-7.0f, fminf(up, 7.0f));
        return __fdividef(gc, 1.0f + __expf(-1.702f * gc)) * (uc + 1.0f);
    }
    if (activation == SHRIKE_ACT_GELU_TANH) return glu(gate, up, activation);
    return __fdividef(gate, 1.0f + __expf(-gate)) * up;
}

// Bounded wait for the pipeline barriers: these are on the critical path of every K block, so the
// first polls do not sleep.
__device__ __forceinline__ bool pipe_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t it = 0; it < (1u << 21); ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(addr), "r"(parity) : "memory");
        if (ok) return true;
        if (it > 256) __nanosleep(32);
    }
    return false;
}

// 16-bit field `idx` (0..7) of four registers.
__device__ __forceinline__ uint16_t pick16(const uint32_t (&v)[4], uint32_t idx) {
    const uint32_t lo = (idx & 2u) ? v[1] : v[0], hi = (idx & 2u) ? v[3] : v[2];
    const uint32_t w = (idx & 4u) ? hi : lo;
    return (uint16_t)((idx & 1u) ? (w >> 16) : (w & 0xffffu));
}

struct alignas(16) ChunkInstance {  // up to 256 rows that share one expert block
    uint32_t kind, slot, first, count;
};

// The instance's rows as one or two boxes of 16 << i rows (the largest that fits, then the smallest that holds the
// rest), and the layout of the activation and weight stages. An instance with few rows needs narrow activation tiles and
// gets more weight stages instead: what paces such a tile is the round trip converters -> tensor core -> converters.
struct TileShape {
    uint32_t N, n1, b1, n2, b2, b_stage, off_a, a_stages, acc_step;
    bool in_tmem;   // converted weights: stages of 64 TMEM columns from column 256 on
    __device__ explicit TileShape(uint32_t count) {
        N = (count + 15u) & ~15u;           // MMA N: rows padded to 16
        n1 = 16; b1 = 0;
        while ((n1 << 1) <= N && b1 + 1 < (uint32_t)kActBoxes) { n1 <<= 1; ++b1; }
        n2 = 0; b2 = 0;
        if (N > n1) {
            n2 = 16;
            while (n2 < N - n1) { n2 <<= 1; ++b2; }
        }
        // three layouts: 64, 128 or 256 activation rows a stage
        b_stage = N <= 64 ? 64u * 128u : N <= 128 ? 128u * 128u : 256u * 128u;
        off_a = kBStages * b_stage;
        // Up to 128 rows the accumulators leave TMEM room for the converted weights. From shared memory the tensor core
        // needs 85 cycles to fetch the weights of an instruction, whatever its N; and the converters' stores and their
        // fence fall away.
        in_tmem = N <= 128;
        acc_step = in_tmem ? 128u : kUmmaMaxN;
        a_stages = in_tmem ? kMaxAStages : (kOffPk - off_a) / kAStageBytes;
    }
};

// A persistent block per SM; tiles (instance, 128 or 256 weight rows) come from a counter, in list order. The copy
// threads run ahead into the next tile while the converters finish this one: as one block per tile, set-up, the first
// copies' way and the launch gap cost 4 us of every tile's 8 (512 x 16 columns) to 37 (2048 x 256).
template <int BITS, int GROUP, int META, int PHASE>
__global__ void __launch_bounds__(kUmmaThreads, 1)
umma_expert_kernel(const ExpertArgs a, const ChunkInstance* __restrict__ inst, uint32_t* __restrict__ n_inst,
                   const uint32_t row_tiles, const __grid_constant__ UmmaMaps maps) {
    constexpr uint32_t kRowBlockBytes = 64 * BITS / 8;  // packed bytes of one row per K block (32 or 64)
    constexpr uint32_t kWordsPerBlock = kRowBlockBytes / 4;
    constexpr uint32_t kGroupsPerBlock = 64 / GROUP;    // 1 (g64) or 2 (g32)
    constexpr uint32_t kKbPerPk = 64 / kRowBlockBytes;  // K blocks per packed copy (2 or 1)
    constexpr uint32_t kKbPerSc = 8 / kGroupsPerBlock;  // K blocks per scale copy (8 or 4)
    constexpr float kZero = BITS == 4 ? 8.0f : 128.0f;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    pdl_launch_dependents();
    // Scale rows that are whole 16-byte units come by TMA; others (groups % 8 != 0) are read by the converters. One way for
    // all instances: both use the same memory, which the copy thread would fill a tile ahead.
    const bool sc_tma = PHASE == 0 ? (a.d / GROUP & 7u) == 0 : ((a.f / GROUP | a.f_shared / GROUP) & 7u) == 0;

    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
    uint64_t* bars = (uint64_t*)(smem + kOffBar);
    uint64_t* a_full = bars;                       // converters -> MMA
    uint64_t* a_empty = a_full + kMaxAStages;      // MMA -> converters
    uint64_t* b_full = a_empty + kMaxAStages;      // activation copy -> MMA
    uint64_t* b_empty = b_full + kBStages;         // MMA -> activation copy
    uint64_t* pk_full = b_empty + kBStages;        // weight copy -> converters
    uint64_t* pk_empty = pk_full + kPkSlots;       // converters -> weight copy
    uint64_t* sc_full = pk_empty + kPkSlots;
    uint64_t* sc_empty = sc_full + 1;
    uint64_t* accum = sc_empty + 1;                // all of a tile's MMAs are done
    uint64_t* next_full = accum + 1;               // [2] weight copy -> everyone: the next tile's number
    uint64_t* next_empty = next_full + 2;
    uint64_t* conv = next_empty + 2;               // the converter warps among themselves (a named barrier has no bounded wait)
    uint32_t* rowid = (uint32_t*)(bars + kNumBars);                 // [2][column] token of a column, tiles in turn
    float* roww = (float*)(rowid + 2 * kUmmaMaxN);                  // [2][column] route weight (routed) or gate (shared)
    uint32_t* next_tile = (uint32_t*)(roww + 2 * kUmmaMaxN);        // [2]
    uint32_t* tmem_slot = next_tile + 2;
    __shared__ uint32_t s_failed;

    if (tid == 0) {
        for (uint32_t s = 0; s < kMaxAStages; ++s) { mbar_init(&a_full[s], kConvWarps); mbar_init(&a_empty[s], 1); }
        for (uint32_t s = 0; s < kBStages; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 1); }
        for (uint32_t s = 0; s < kPkSlots; ++s) { mbar_init(&pk_full[s], 1); mbar_init(&pk_empty[s], kConvWarps); }
        mbar_init(sc_full, 1);
        mbar_init(sc_empty, kConvWarps);
        mbar_init(accum, 1);
        mbar_init(conv, kConvWarps);
        for (uint32_t s = 0; s < 2; ++s) { mbar_init(&next_full[s], 1); mbar_init(&next_empty[s], kConvWarps + 2); }
        fence_mbar_init();
        s_failed = 0;
    }
    // two accumulators of up to 256 columns: all of TMEM (a block per SM)
    if (warp == kConvWarps) tmem_alloc(smem_u32(tmem_slot), 2 * kUmmaMaxN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();   // all of the above runs while the last kernel ends
    const uint32_t n_tiles = n_inst[0] * row_tiles;
    auto give_up = [&]() {
        report_status(a.status, kStatusWaitTimeout);
        *(volatile uint32_t*)&s_failed = 1;
    };
    auto failed = [&]() { return *(volatile uint32_t*)&s_failed != 0; };
    // Every barrier's use is counted in one bit per stage, kept by each role for itself: full barriers are waited for
    // with the bit, empty ones with its complement (the first use of a stage finds it empty).
    // The tile after `turn` others; n_tiles and above: none.
    auto take_tile = [&](uint32_t turn) -> uint32_t {
        const uint32_t s = turn & 1;
        if (!__all_sync(0xffffffffu, pipe_wait(&next_full[s], (turn >> 1) & 1))) { give_up(); return 0xffffffffu; }
        const uint32_t t = *(volatile uint32_t*)&next_tile[s];
        __syncwarp();
        if (lane == 0) mbar_arrive(&next_empty[s]);
        return __shfl_sync(0xffffffffu, t, 0);
    };
    struct Work {
        ChunkInstance in;
        bool shared;
        uint32_t F, KB, out_rows, r0;
    };
    auto open_tile = [&](uint32_t t, Work& w) {   // false: no such rows (a narrower shared or routed expert)
        const uint32_t ii = t / row_tiles;
        const uint4 v = __ldg((const uint4*)(inst + ii));
        w.in.kind = v.x; w.in.slot = v.y; w.in.first = v.z; w.in.count = v.w;
        w.shared = w.in.kind == 1;
        w.F = w.shared ? a.f_shared : a.f;
        w.KB = (PHASE == 0 ? a.d : w.F) / 64;
        w.out_rows = PHASE == 0 ? w.F : a.d;       // rows of the weight matrix
        w.r0 = (t - ii * row_tiles) * (PHASE == 0 ? 128u : 256u);
        return w.r0 < w.out_rows;
    };

    if (warp < kConvWarps) {
        // ---------------- converters, then the tile's epilogue ----------------
        uint32_t a_use = 0, pk_use = 0, sc_use = 0, slot = 0, acc_use = 0, conv_use = 0, odd = 0;
        auto converters_meet = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(conv);
            const bool ok = pipe_wait(conv, conv_use);
            conv_use ^= 1;
            if (!ok) give_up();
            return ok;
        };
        // Two threads per weight row: thread `half` converts 32 of the K block's 64 weights. A lane is a row: the TMEM lanes
        // that a warp reaches.
        const uint32_t tile = (warp >> 2) & 1, r = (warp & 3) * 32 + lane, half = warp >> 3;
        const uint32_t a_tmem = tmem_base + 256u + (((warp & 3) * 32) << 16) + tile * 32 + half * 16;
        constexpr uint32_t kWordsPerThread = kWordsPerBlock / 2;   // 4 (int4) or 8 (int8)
        const uint32_t pk_row = kOffPk + tile * (kPkSlotBytes / 2) + r * 64, pk_xor = (r >> 1) & 3;
        // What does not change along K: this thread's chunk positions in a packed slot and in the converted
        // tile (both swizzled by the row).
        uint32_t pk_off[kKbPerPk * (kWordsPerThread / 4)];
#pragma unroll
        for (uint32_t sub = 0; sub < kKbPerPk; ++sub)
#pragma unroll
            for (uint32_t q = 0; q < kWordsPerThread / 4; ++q) {
                // 16-byte chunk of the 64-byte row: the K block's share, then this thread's half of it
                const uint32_t c = sub * (kRowBlockBytes / 16) + half * (kWordsPerThread / 4) + q;
                pk_off[sub * (kWordsPerThread / 4) + q] = pk_row + ((c ^ pk_xor) << 4);
            }
        uint32_t a_pos[4];
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i)   // A row r: 8 chunks of 8 fp16; chunk c lives at position c ^ (r & 7)
            a_pos[i] = tile * kTileBytes + r * 128 + (((half * 4 + i) ^ (r & 7)) << 4);

        bool wide = false;   // the last tile's accumulators took all of TMEM
        for (uint32_t turn = 0;; ++turn) {
            const uint32_t t = take_tile(turn);
            if (t >= n_tiles || failed()) break;
            Work wk;
            if (!open_tile(t, wk)) continue;
            const ChunkInstance& in = wk.in;
            const bool shared = wk.shared;
            const uint32_t F = wk.F, KB = wk.KB, out_rows = wk.out_rows, r0 = wk.r0, G = KB * 64 / GROUP;
            const TileShape ts(in.count);
            const Offsets3& off = shared ? a.shared : a.routed;
            const uint8_t* base = shared ? a.shared_block : pool_cell_base(a.pool, in.slot);
            uint32_t* const ids = rowid + odd * kUmmaMaxN;
            float* const wts = roww + odd * kUmmaMaxN;
            odd ^= 1;
            // the tokens and route weights of the columns: the epilogue reads them, long after these loads
            if (PHASE == 1 && tid < kUmmaMaxN) {
                const uint32_t src = tid < in.count ? tid : 0;
                if (shared) {
                    ids[tid] = in.first + src;
                    wts[tid] = a.shared_gate ? a.shared_gate[in.first + src] : 1.0f;
                } else {
                    const uint32_t pair = a.sorted[in.first + src];
                    ids[tid] = pair / a.top_k;
                    wts[tid] = a.route_w[pair];
                }
            }
            uint32_t sreg[4] = {0, 0, 0, 0}, breg[4] = {0, 0, 0, 0};
            uint32_t snext[4] = {0, 0, 0, 0}, bnext[4] = {0, 0, 0, 0};
            const uint32_t mrow = r0 + (PHASE == 0 ? r : tile * 128 + r);
            const int mat = PHASE == 0 ? (int)tile : 2;
            const uint16_t* srow = (const uint16_t*)(base + off.s[mat]) + (size_t)mrow * G;
            const uint16_t* brow = (const uint16_t*)(base + off.b[mat]) + (size_t)mrow * G;
            // Groups 8*blk .. 8*blk+7 straight from global memory (rows past the matrix and groups past the row read as
            // zero: the converted weights are then zero). An even number of groups: the warp's 32 rows in 32-bit words, four
            // lanes a row, handed to the rows' lanes when they are needed; read by each row's threads in 16-bit pieces
            // they kept L1 busy for 1.3 us per K block of 90-group rows.
            const bool words = (G & 1u) == 0;
            const uint32_t my_rows = r0 + (PHASE == 0 ? 0u : tile * 128u) + (warp & 3) * 32 + (lane >> 2);
            auto fetch_scales = [&](uint32_t blk) {
                if (words) {
                    const uint32_t gi = blk * 8 + 2 * (lane & 3);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t row = my_rows + 8 * i;
                        const bool there = row < out_rows && gi < G;
                        const size_t at = (size_t)row * G + gi;
                        snext[i] = there ? __ldg((const uint32_t*)((const uint16_t*)(base + off.s[mat]) + at)) : 0u;
                        bnext[i] = there ? __ldg((const uint32_t*)((const uint16_t*)(base + off.b[mat]) + at)) : 0u;
                    }
                    return;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t gi = blk * 8 + 2 * i;
                    uint32_t sv = 0, bv = 0;
                    if (mrow < out_rows && gi < G) {
                        sv = __ldg(srow + gi);
                        bv = __ldg(brow + gi);
                        if (gi + 1 < G) {
                            sv |= (uint32_t)__ldg(srow + gi + 1) << 16;
                            bv |= (uint32_t)__ldg(brow + gi + 1) << 16;
                        }
                    }
                    snext[i] = sv;
                    bnext[i] = bv;
                }
            };
            if (!sc_tma) fetch_scales(0);
            // A scale block (8 groups of the row) at a time, its K blocks unrolled: the position in the packed slot
            // and the group of a K block are then constants of the instruction stream.
            // (a warp may write the stages while others still read the columns that they take of the last accumulators)
            if (wide && ts.in_tmem && !converters_meet()) break;
            wide = !ts.in_tmem;
            uint32_t st = 0;
            for (uint32_t kb0 = 0; kb0 < KB; kb0 += kKbPerSc) {
                if (failed()) break;
                if (sc_tma) {
                    if (!pipe_wait(sc_full, sc_use)) { give_up(); break; }
                    sc_use ^= 1;
                    const uint4 sv = *(const uint4*)(smem + kOffSc + tile * (kScHalfBytes / 2) + r * 16);
                    const uint4 bv = *(const uint4*)(smem + kOffSc + kScHalfBytes + tile * (kScHalfBytes / 2) + r * 16);
                    sreg[0] = sv.x; sreg[1] = sv.y; sreg[2] = sv.z; sreg[3] = sv.w;
                    breg[0] = bv.x; breg[1] = bv.y; breg[2] = bv.z; breg[3] = bv.w;
                    // the values are in registers: the copy thread may fetch the next block's
                    __syncwarp();
                    if (lane == 0) mbar_arrive(sc_empty);
                } else {
                    // this block's 8 groups were fetched one block ago; fetch the next block's now
                    if (words) {
                        __syncwarp();   // the last block's have been read
                        if constexpr (GROUP == 32) {
                            // through the scales' memory: a thread's half has the even or the odd groups, so the two warps
                            // of a row write 16 bits of every word each
                            uint8_t* const to = smem + kOffSc + (tile * 128 + (warp & 3) * 32 + (lane >> 2)) * 16 + (lane & 3) * 4 + half * 2;
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                *(uint16_t*)(to + i * 128) = (uint16_t)(half ? snext[i] >> 16 : snext[i]);
                                *(uint16_t*)(to + kScHalfBytes + i * 128) = (uint16_t)(half ? bnext[i] >> 16 : bnext[i]);
                            }
                            __syncwarp();
                            const uint4 sv = *(const uint4*)(smem + kOffSc + (tile * 128 + r) * 16), bv = *(const uint4*)(smem + kOffSc + kScHalfBytes + (tile * 128 + r) * 16);
                            sreg[0] = sv.x; sreg[1] = sv.y; sreg[2] = sv.z; sreg[3] = sv.w;
                            breg[0] = bv.x; breg[1] = bv.y; breg[2] = bv.z; breg[3] = bv.w;
                        } else {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {   // lane 4 (row mod 8) + word of load row / 8
#pragma unroll
                                for (int w = 0; w < 4; ++w) {
                                    const uint32_t sv = __shfl_sync(0xffffffffu, snext[i], 4 * (lane & 7) + w);
                                    const uint32_t bv = __shfl_sync(0xffffffffu, bnext[i], 4 * (lane & 7) + w);
                                    if ((lane >> 3) == (uint32_t)i) { sreg[w] = sv; breg[w] = bv; }
                                }
                            }
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i) { sreg[i] = snext[i]; breg[i] = bnext[i]; }
                    }
                    fetch_scales(kb0 / kKbPerSc + 1);
                }
#pragma unroll
                for (uint32_t j = 0; j < kKbPerSc; ++j) {
                    const uint32_t kb = kb0 + j;
                    if (kb >= KB) break;
                    constexpr uint32_t kSubMask = kKbPerPk - 1;
                    const uint32_t sub = j & kSubMask;         // K block within its packed slot
                    if (sub == 0 && !pipe_wait(&pk_full[slot], (pk_use >> slot) & 1)) { give_up(); break; }
                    uint32_t pk[kWordsPerThread];
#pragma unroll
                    for (uint32_t q = 0; q < kWordsPerThread / 4; ++q) {
                        const uint4 v = *(const uint4*)(smem + slot * kPkSlotBytes + pk_off[sub * (kWordsPerThread / 4) + q]);
                        pk[4 * q] = v.x; pk[4 * q + 1] = v.y; pk[4 * q + 2] = v.z; pk[4 * q + 3] = v.w;
                    }
                    // a thread's half of a 64-wide block lies inside one group of 32 or 64
                    const uint32_t gsel = j * kGroupsPerBlock + (GROUP == 64 ? 0u : half);
                    const float sc = meta_to_f32<META>(pick16(sreg, gsel));
                    const float zf = fmaf(kZero, sc, meta_to_f32<META>(pick16(breg, gsel)));
                    const uint32_t s2 = half2_dup(sc), z2 = half2_dup(zf);
                    if (!pipe_wait(&a_empty[st], ((a_use >> st) & 1) ^ 1)) { give_up(); break; }
                    a_use ^= 1u << st;
                    uint32_t o[16];   // 32 weights
#pragma unroll
                    for (uint32_t i = 0; i < kWordsPerThread; ++i) {
                        uint32_t w4[4];
                        dequant_word<BITS>(pk[i], s2, z2, w4);
#pragma unroll
                        for (uint32_t e = 0; e < 16 / kWordsPerThread; ++e) o[i * (16 / kWordsPerThread) + e] = w4[e];
                    }
                    if (ts.in_tmem) {
                        __syncwarp();
                        tc_fence_after();   // the stage's last readers are done
                        tmem_st16(a_tmem + st * 64, o);
                        tc_fence_before();
                    } else {
                        uint8_t* a_stage = smem + ts.off_a + st * kAStageBytes;
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i)
                            *(uint4*)(a_stage + a_pos[i]) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                        fence_async_smem();
                    }
                    __syncwarp();
                    const bool slot_done = sub == kSubMask || kb + 1 == KB;
                    if (lane == 0) {
                        // one arrival per warp: 512 arrivals on one barrier word would serialise every K block
                        mbar_arrive(&a_full[st]);
                        // The ring slots are handed back only here: by now the values read from them have been
                        // consumed, so the reads are complete before the copy thread may overwrite the slot.
                        if (slot_done) mbar_arrive(&pk_empty[slot]);
                    }
                    if (slot_done) {
                        pk_use ^= 1u << slot;
                        if (++slot == kPkSlots) slot = 0;
                    }
                    if (++st == ts.a_stages) st = 0;
                }
            }
            // ---------------- epilogue (warp w: TMEM lanes 32*(w & 3) .. +31, every fourth 16-column group) ----------------
            bool ok = pipe_wait(accum, acc_use);
            acc_use ^= 1;
            if (!ok) give_up();
            if (failed()) break;
            tc_fence_after();
            // the columns' tokens and weights were written by other converter threads at the start of the tile
            if (PHASE == 1 && !converters_meet()) break;
            // (eight columns at a time and loops that are not unrolled further: the code runs once per tile, and fetching
            // it takes longer than what unrolling saves)
            const uint32_t q = warp & 3, h = warp >> 2, N = ts.N;
            const uint32_t trow = q * 32 + lane;                       // row inside each 128-row tile
            const uint32_t taddr = tmem_base + ((q * 32) << 16);
            constexpr uint32_t kColStep = 8 * (kConvWarps / 4);
            if (PHASE == 0) {
                const uint32_t f = r0 + trow;
                float gab = 0.f, uab = 0.f;
                if (a.expert_bias && f < F) {
                    gab = bf16_bits_to_f32(((const uint16_t*)(base + off.ab[0]))[f]);
                    uab = bf16_bits_to_f32(((const uint16_t*)(base + off.ab[1]))[f]);
                }
                uint16_t* const dst = (shared ? a.acts_shared : a.acts) + (size_t)in.first * F + perm_index(f, BITS == 4);
                auto columns = [&](auto glu_of) {
                    bool over = false;
#pragma unroll 1
                    for (uint32_t c0 = h * 8; c0 < N; c0 += kColStep) {
                        uint32_t g[8], u[8];
                        tmem_ld8_issue(taddr + c0, g);
                        tmem_ld8_issue(taddr + ts.acc_step + c0, u);
                        tmem_ld_wait();
                        uint16_t* p = dst + (size_t)c0 * F;
                        const uint32_t live = f < F ? min(8u, in.count > c0 ? in.count - c0 : 0u) : 0u;   // rows of this group
#pragma unroll
                        for (int j = 0; j < 8; j += 2) {
                            float v[2];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                v[e] = glu_of(__uint_as_float(g[j + e]) + gab, __uint_as_float(u[j + e]) + uab);
                                if (fabsf(v[e]) > kHalfMax) {   // false for NaN, which passes through
                                    over |= (uint32_t)(j + e) < live;
                                    v[e] = copysignf(kHalfMax, v[e]);
                                }
                            }
                            const __half2 hv = __floats2half2_rn(v[0], v[1]);
                            if ((uint32_t)j < live) *p = __half_as_ushort(__low2half(hv));
                            p += F;
                            if ((uint32_t)j + 1 < live) *p = __half_as_ushort(__high2half(hv));
                            p += F;
                        }
                    }
                    if (over) report_status(a.status, kStatusOperandRange);
                };
                if (a.activation == SHRIKE_ACT_CLAMPED_SWIGLU) columns([](float x, float y) { return glu_epilogue(x, y, SHRIKE_ACT_CLAMPED_SWIGLU); });
                else if (a.activation == SHRIKE_ACT_GELU_TANH) columns([](float x, float y) { return glu_epilogue(x, y, SHRIKE_ACT_GELU_TANH); });
                else columns([](float x, float y) { return glu_epilogue(x, y, SHRIKE_ACT_SILU); });
            } else {
                const uint32_t d0 = r0 + trow, d1 = d0 + 128;
                float ab0 = 0.f, ab1 = 0.f;
                if (a.expert_bias) {
                    const uint16_t* dab = (const uint16_t*)(base + off.ab[2]);
                    if (d0 < a.d) ab0 = bf16_bits_to_f32(dab[d0]);
                    if (d1 < a.d) ab1 = bf16_bits_to_f32(dab[d1]);
                }
                const bool ok0 = d0 < a.d, ok1 = d1 < a.d;
#pragma unroll 1
                for (uint32_t c0 = h * 8; c0 < N; c0 += kColStep) {
                    uint32_t v0[8], v1[8];
                    tmem_ld8_issue(taddr + c0, v0);
                    tmem_ld8_issue(taddr + ts.acc_step + c0, v1);
                    tmem_ld_wait();
                    const uint32_t live = min(8u, in.count > c0 ? in.count - c0 : 0u);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if ((uint32_t)j < live) {
                            // lanes hold consecutive output rows: one 128-byte reduction per warp and column
                            float* o = a.yacc + (size_t)ids[c0 + j] * a.d + d0;
                            const float w = wts[c0 + j];
                            if (ok0) atomicAdd(o, w * (__uint_as_float(v0[j]) + ab0));
                            if (ok1) atomicAdd(o + 128, w * (__uint_as_float(v1[j]) + ab1));
                        }
                    }
                }
            }
            tc_fence_before();   // these reads of the accumulators come before the next tile's instructions
        }
    } else if (warp == kConvWarps) {
        // ---------------- MMA issue ----------------
        // The whole warp walks the loop on warp-uniform values and one elected lane issues: behind a branch on the lane
        // number every descriptor was a per-thread value, and all tiles ran at 0.7 us per K block (0.5 now at 16 columns).
        uint32_t a_use = 0, b_use = 0;
        for (uint32_t turn = 0;; ++turn) {
            const uint32_t t = take_tile(turn);
            if (t >= n_tiles || failed()) break;
            Work wk;
            if (!open_tile(t, wk)) continue;
            const TileShape ts(wk.in.count);
            const uint32_t idesc = __shfl_sync(0xffffffffu, umma_idesc(ts.N), 0), acc0 = __shfl_sync(0xffffffffu, tmem_base, 0);
            const uint32_t acc1 = acc0 + __shfl_sync(0xffffffffu, ts.acc_step, 0), stages = __shfl_sync(0xffffffffu, ts.a_stages, 0);
            const uint32_t b_smem = __shfl_sync(0xffffffffu, smem_base, 0), a_smem = b_smem + __shfl_sync(0xffffffffu, ts.off_a, 0);
            const uint32_t b_step = __shfl_sync(0xffffffffu, ts.b_stage, 0), n_kb = __shfl_sync(0xffffffffu, wk.KB, 0);
            const bool in_tmem = __shfl_sync(0xffffffffu, (uint32_t)ts.in_tmem, 0) != 0;
            uint32_t sa = 0, sb = 0;
            for (uint32_t kb = 0; kb < n_kb; ++kb) {
                // (the first stage of converted weights also says that the last tile's accumulators have been read)
                const bool got = pipe_wait(&b_full[sb], (b_use >> sb) & 1) && pipe_wait(&a_full[sa], (a_use >> sa) & 1);
                if (!__all_sync(0xffffffffu, got)) {
                    give_up();
                    break;
                }
                a_use ^= 1u << sa;
                b_use ^= 1u << sb;
                __syncwarp();
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t db = umma_smem_desc(b_smem + sb * b_step);
                    if (in_tmem) {
                        const uint32_t ta = acc0 + 256u + sa * 64;   // 16 of K are eight columns
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k) {
                            umma_f16_ts(acc0, ta + 8 * k, db + 2 * k, idesc, (kb | k) != 0);
                            umma_f16_ts(acc1, ta + 32 + 8 * k, db + 2 * k, idesc, (kb | k) != 0);
                        }
                    } else {
                        const uint64_t da0 = umma_smem_desc(a_smem + sa * kAStageBytes), da1 = umma_smem_desc(a_smem + sa * kAStageBytes + kTileBytes);
                        // 4 x K16 per 64-wide block: 32 bytes further along the row. The two tiles alternate: consecutive
                        // instructions then add into different accumulators.
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k) {
                            umma_f16(acc0, da0 + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                            umma_f16(acc1, da1 + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                        }
                    }
                    umma_commit(&a_empty[sa]);
                    umma_commit(&b_empty[sb]);
                }
                __syncwarp();
                if (++sa == stages) sa = 0;
                if (++sb == kBStages) sb = 0;
            }
            if (elect_one()) umma_commit(accum);
            __syncwarp();
        }
    } else if (warp == kConvWarps + 1) {
        // ---------------- activation tiles ----------------
        // One or two boxes per K block: these tiles are most of what a block pulls out of L2, and a short instance
        // does not pay for 256 rows, nor one of 80 rows for 128.
        uint32_t b_use = 0, last_stage = 0;
        for (uint32_t turn = 0;; ++turn) {
            const uint32_t t = take_tile(turn);
            if (t >= n_tiles || failed()) break;
            Work wk;
            if (!open_tile(t, wk)) continue;
            const TileShape ts(wk.in.count);
            const CUtensorMap* maps_b = wk.shared ? maps.act_shared : maps.act_routed;
            if (lane == 0) {
                // Another layout: the last use of the old stages that its stages lie across has to be done. (The stages
                // themselves are waited for, not the tile: a tile of two K blocks leaves the third stage to the tile before it, so
                // the tile barrier could still be two phases behind, where its one parity bit reads as passed. By the lane
                // that copies: with the wait and a vote by the whole warp, 333 rows took 297 us for 291.)
                const uint32_t over = last_stage && ts.b_stage != last_stage ?
                                          min(kBStages, (kBStages * ts.b_stage + last_stage - 1) / last_stage) : 0u;
                last_stage = ts.b_stage;
#pragma unroll 1
                for (uint32_t s = 0; s < over; ++s)
                    if (!pipe_wait(&b_empty[s], ((b_use >> s) & 1) ^ 1)) { give_up(); break; }
                const uint32_t b_bytes = (ts.n1 + ts.n2) * 128u;
                uint32_t sb = 0;
                for (uint32_t kb = 0; kb < wk.KB; ++kb) {
                    if (failed()) break;
                    if (!pipe_wait(&b_empty[sb], ((b_use >> sb) & 1) ^ 1)) { give_up(); break; }
                    b_use ^= 1u << sb;
                    mbar_expect_tx(&b_full[sb], b_bytes);
                    tma_load_2d(smem_base + sb * ts.b_stage, &maps_b[ts.b1], (int32_t)(kb * 64), (int32_t)wk.in.first, &b_full[sb]);
                    if (ts.n2)
                        tma_load_2d(smem_base + sb * ts.b_stage + ts.n1 * 128u, &maps_b[ts.b2], (int32_t)(kb * 64),
                                    (int32_t)(wk.in.first + ts.n1), &b_full[sb]);
                    if (++sb == kBStages) sb = 0;
                }
            }
            __syncwarp();
        }
    } else if (lane == 0) {
        // ---------------- tile numbers; packed weights, scales, biases ----------------
        uint32_t pk_use = 0, sc_use = 0, slot = 0;
        for (uint32_t turn = 0;; ++turn) {
            const uint32_t s = turn & 1;
            const uint32_t t = turn == 0 ? blockIdx.x : gridDim.x + atomicAdd(n_inst + 1 + PHASE, 1u);
            if (!pipe_wait(&next_empty[s], ((turn >> 1) & 1) ^ 1)) { give_up(); break; }
            *(volatile uint32_t*)&next_tile[s] = t;
            mbar_arrive(&next_full[s]);
            if (t >= n_tiles || failed()) break;
            Work wk;
            if (!open_tile(t, wk)) continue;
            const ChunkInstance& in = wk.in;
            const WeightMaps* wm = wk.shared ? &maps.shared : &maps.routed[in.slot / a.pool.cells_per_chunk];
            const int32_t cell = wk.shared ? 0 : (int32_t)(in.slot % a.pool.cells_per_chunk);
            const int32_t y0 = (int32_t)wk.r0, y1 = (int32_t)(PHASE == 0 ? wk.r0 : wk.r0 + 128);
            for (uint32_t kb = 0; kb < wk.KB; ++kb) {
                if (failed()) break;
                if (sc_tma && kb % kKbPerSc == 0) {
                    const int32_t g0 = (int32_t)(kb / kKbPerSc * 8);
                    if (!pipe_wait(sc_empty, sc_use ^ 1)) { give_up(); break; }
                    sc_use ^= 1;
                    mbar_expect_tx(sc_full, 2 * kScHalfBytes);
                    const uint32_t dst = smem_base + kOffSc;
                    tma_load_3d(dst, &wm->s[0], g0, y0, cell, sc_full);
                    tma_load_3d(dst + kScHalfBytes / 2, &wm->s[1], g0, y1, cell, sc_full);
                    tma_load_3d(dst + kScHalfBytes, &wm->b[0], g0, y0, cell, sc_full);
                    tma_load_3d(dst + kScHalfBytes + kScHalfBytes / 2, &wm->b[1], g0, y1, cell, sc_full);
                }
                if (kb % kKbPerPk == 0) {
                    const int32_t x = (int32_t)(kb / kKbPerPk * 64);
                    if (!pipe_wait(&pk_empty[slot], ((pk_use >> slot) & 1) ^ 1)) { give_up(); break; }
                    pk_use ^= 1u << slot;
                    mbar_expect_tx(&pk_full[slot], kPkSlotBytes);
                    const uint32_t dst = smem_base + kOffPk + slot * kPkSlotBytes;
                    tma_load_3d(dst, &wm->w[0], x, y0, cell, &pk_full[slot]);
                    tma_load_3d(dst + kPkSlotBytes / 2, &wm->w[1], x, y1, cell, &pk_full[slot]);
                    if (++slot == kPkSlots) slot = 0;
                }
            }
        }
    }
    if (failed() && lane == 0 && warp > kConvWarps) {
        // a copy of this block may still be in flight: give it a bounded time to land
        for (int i = 0; i < 200; ++i) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kConvWarps) {
        __syncwarp();
        tmem_dealloc(tmem_base, 2 * kUmmaMaxN);
    }
}

// One thread per expert: ceil(count/256) chunk instances each, then the shared expert's.
// n_inst[0] = instances, [1], [2]: tiles handed out in phase 0, 1.
__global__ void __launch_bounds__(256)
chunk_instances_kernel(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ counts,
                       const uint32_t* __restrict__ slot_of_expert, uint32_t ne, uint32_t T, uint32_t with_shared,
                       uint32_t pool_cells, ChunkInstance* __restrict__ inst, uint32_t* __restrict__ n_inst,
                       uint32_t* status) {
    pdl_wait();
    pdl_launch_dependents();
    __shared__ uint32_t warp_sums[8], by_size[256];
    __shared__ __align__(16) uint32_t key[256];
    // Experts with the most rows first: a tile of 256 rows takes twice the time of one of 16, and a list that ends on long
    // ones leaves SMs idle (4096 rows: the last ended a tenth after the median SM).
    key[threadIdx.x] = (threadIdx.x < ne ? counts[threadIdx.x] << 8 : 0u) | (255u - threadIdx.x);
    __syncthreads();
    {
        const uint32_t mine = key[threadIdx.x];
        uint32_t rank = 0;
        for (uint32_t j = 0; j < 256; j += 4) {
            const uint4 v = *(const uint4*)&key[j];
            rank += (v.x > mine) + (v.y > mine) + (v.z > mine) + (v.w > mine);
        }
        by_size[rank] = threadIdx.x;
    }
    __syncthreads();
    const uint32_t e = by_size[threadIdx.x];
    uint32_t n = 0, slot = SHRIKE_SLOT_MISS, c = 0;
    if (e < ne && counts[e] > 0) {
        c = counts[e];
        slot = slot_of_expert[e];
        if (slot != SHRIKE_SLOT_MISS && slot >= pool_cells) {
            report_status(status, kStatusBadIndex);
            slot = SHRIKE_SLOT_MISS;
        }
        if (slot != SHRIKE_SLOT_MISS) n = (c + kUmmaMaxN - 1) / kUmmaMaxN;
    }
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
    // The shared expert's instances come first in the list: they are full (256 rows), and the blocks of the
    // list's end are the last to start -- a launch that ends on its longest blocks ends late.
    const uint32_t n_shared = with_shared ? (T + kUmmaMaxN - 1) / kUmmaMaxN : 0;
    base += inc - n + n_shared;
    for (uint32_t j = 0; j < n; ++j) {
        ChunkInstance in;
        in.kind = 0; in.slot = slot; in.first = offsets[e] + kUmmaMaxN * j; in.count = min(kUmmaMaxN, c - kUmmaMaxN * j);
        inst[base + j] = in;
    }
    for (uint32_t j = threadIdx.x; j < n_shared; j += blockDim.x) {
        ChunkInstance in;
        in.kind = 1; in.slot = 0; in.first = kUmmaMaxN * j; in.count = min(kUmmaMaxN, T - kUmmaMaxN * j);
        inst[j] = in;
    }
    if (threadIdx.x == 0) {
        n_inst[0] = total + n_shared;
        n_inst[1] = n_inst[2] = 0;   // tiles handed out, per phase
    }
}

// ---- tensor maps -------------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) != cudaSuccess ||
            qres != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (EncodeTiledFn)p;
    }();
    return fn;
}

// fp16 activation rows [rows][cols]: box = 64 columns (one 128-byte swizzle row) x box_rows rows.
static bool make_rows_map(CUtensorMap* map, const uint16_t* base, uint64_t cols, uint64_t rows, uint32_t box_rows) {
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return encode_tiled_fn()(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, (void*)base, dims, strides, box, elem,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// One matrix of every cell of a pool chunk: [cells][rows][row_bytes] bytes (packed weights, 64-byte
// boxes of 128 rows, 64-byte swizzle) or [cells][rows][groups] 16-bit (scales / biases, 8 per row).
static bool make_matrix_map(CUtensorMap* map, const uint8_t* base, bool meta, uint64_t row_elems, uint64_t rows,
                            uint64_t cells, uint64_t cell_stride) {
    const uint64_t esz = meta ? 2 : 1;
    const cuuint64_t dims[3] = {row_elems, rows, cells};
    // a single cell (the shared expert's block) still needs a valid outer pitch
    const cuuint64_t strides[2] = {row_elems * esz, cells > 1 ? cell_stride : row_elems * esz * rows};
    const cuuint32_t box[3] = {meta ? 8u : 64u, 128, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    return encode_tiled_fn()(map, meta ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, (void*)base,
                             dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             meta ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_64B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The two tiles of one phase: gate + up (phase 0) or down twice (phase 1).
static bool make_weight_maps(WeightMaps* wm, const uint8_t* base, const Offsets3& off, int phase, uint32_t kdim,
                             uint32_t rows, uint32_t bits, uint32_t group, uint64_t cells, uint64_t cell_stride) {
    for (int t = 0; t < 2; ++t) {
        const int mat = phase == 0 ? t : 2;
        if (!make_matrix_map(&wm->w[t], base + off.w[mat], false, (uint64_t)kdim * bits / 8, rows, cells, cell_stride))
            return false;
        if ((kdim / group) % 8 != 0) continue;   // such scale rows are read by the converter threads
        if (!make_matrix_map(&wm->s[t], base + off.s[mat], true, kdim / group, rows, cells, cell_stride) ||
            !make_matrix_map(&wm->b[t], base + off.b[mat], true, kdim / group, rows, cells, cell_stride))
            return false;
    }
    return true;
}

// K in whole 64-wide blocks (packed rows are then whole 16-byte units, which the TMA copies need).
bool umma_supported(const shrike_moe_config& c) {
    if (c.d % 64 || c.f % 64) return false;
    if (c.has_shared && c.shared_f % 64) return false;
    return encode_tiled_fn() != nullptr;
}

// Called once per handle, after the workspace exists: the activation operands' maps.
cudaError_t umma_prepare(shrike_moe* m) {
    const shrike_moe_config& c = m->cfg;
    Workspace& ws = m->ws;
    if (!ws.xs || !umma_supported(c)) return cudaSuccess;
    // maps[operand][box]: operands xs, acts, xh, acts_shared; boxes of 16, 32, 64, 128, 256 rows
    CUtensorMap* am = (CUtensorMap*)ws.tensor_maps;
    const uint64_t pairs = (uint64_t)c.max_tokens * c.top_k;
    bool ok = true;
    for (int bi = 0; bi < kActBoxes && ok; ++bi) {
        const uint32_t box_rows = 16u << bi;
        ok = make_rows_map(&am[0 * kActBoxes + bi], ws.xs, c.d, pairs, box_rows) &&
             make_rows_map(&am[1 * kActBoxes + bi], ws.acts, c.f, pairs, box_rows);
        if (ok && c.has_shared)
            ok = make_rows_map(&am[2 * kActBoxes + bi], ws.xh, c.d, c.max_tokens, box_rows) &&
                 make_rows_map(&am[3 * kActBoxes + bi], ws.acts_shared, c.shared_f, c.max_tokens, box_rows);
    }
    return ok ? cudaSuccess : cudaErrorInvalidValue;
}

template <int BITS, int GROUP, int META>
static cudaError_t launch_umma_t(const shrike_moe* m, cudaStream_t st, const ExpertArgs& a, const ChunkInstance* inst,
                                 uint32_t* n_inst, uint32_t max_inst, const UmmaMaps& m0, const UmmaMaps& m1) {
    auto k0 = umma_expert_kernel<BITS, GROUP, META, 0>;
    auto k1 = umma_expert_kernel<BITS, GROUP, META, 1>;
    cudaError_t e = cudaFuncSetAttribute(k0, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kUmmaSmemBytes);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kUmmaSmemBytes);
    if (e != cudaSuccess) return e;
    const uint32_t fmax = a.f_shared > a.f ? a.f_shared : a.f;
    const uint32_t sm_count = (uint32_t)m->sm_count;
    const uint32_t t0 = (fmax + 127) / 128, t1 = (a.d + 255) / 256;
    e = launch_after(m, st, k0, dim3(std::min(sm_count, max_inst * t0)), kUmmaThreads, kUmmaSmemBytes, a, inst, n_inst, t0, m0);
    if (e != cudaSuccess) return e;
    return launch_after(m, st, k1, dim3(std::min(sm_count, max_inst * t1)), kUmmaThreads, kUmmaSmemBytes, a, inst, n_inst, t1, m1);
}

uint32_t umma_max_chunk_instances(const shrike_moe_config& c, uint32_t T) {
    const uint32_t pairs = T * c.top_k;
    uint32_t routed = c.num_experts + pairs / kUmmaMaxN;
    if (routed > pairs) routed = pairs;
    return routed + (c.has_shared ? (T + kUmmaMaxN - 1) / kUmmaMaxN : 0);
}

size_t umma_chunk_instance_bytes() { return sizeof(ChunkInstance); }
size_t umma_tensor_map_bytes() { return 4 * kActBoxes * sizeof(CUtensorMap); }

// Gate/up + GLU, then down, for the instances built from the grouping the
// prefill plan left in the workspace.
cudaError_t launch_umma_prefill(const shrike_moe* m, cudaStream_t st, const ExpertArgs& a, uint32_t T,
                                uint32_t pool_cells) {
    const shrike_moe_config& c = m->cfg;
    const Workspace& ws = m->ws;
    const CUtensorMap* am = (const CUtensorMap*)ws.tensor_maps;
    if (!am || !umma_supported(c)) return cudaErrorNotSupported;
    // descriptors of this call's pool and shared block (host work only)
    UmmaMaps maps[2];
    for (int phase = 0; phase < 2; ++phase) {
        UmmaMaps& mp = maps[phase];
        memset(&mp, 0, sizeof mp);
        const uint32_t kdim = phase == 0 ? c.d : c.f, rows = phase == 0 ? c.f : c.d;
        uint32_t left = a.pool.cells;
        for (uint32_t ch = 0; ch < SHRIKE_MAX_POOL_CHUNKS && a.pool.base[ch] && left; ++ch) {
            const uint32_t cells = left < a.pool.cells_per_chunk ? left : a.pool.cells_per_chunk;
            if (!make_weight_maps(&mp.routed[ch], a.pool.base[ch], a.routed, phase, kdim, rows, c.weight_bits,
                                  c.group_size, cells, a.pool.stride))
                return cudaErrorInvalidValue;
            left -= cells;
        }
        for (int bi = 0; bi < kActBoxes; ++bi) mp.act_routed[bi] = am[phase * kActBoxes + bi];
        if (c.has_shared) {
            const uint32_t kds = phase == 0 ? c.d : c.shared_f, rws = phase == 0 ? c.shared_f : c.d;
            if (!make_weight_maps(&mp.shared, a.shared_block, a.shared, phase, kds, rws, c.weight_bits, c.group_size, 1,
                                  16))
                return cudaErrorInvalidValue;
            for (int bi = 0; bi < kActBoxes; ++bi) mp.act_shared[bi] = am[(2 + phase) * kActBoxes + bi];
        } else {
            mp.shared = mp.routed[0];
            for (int bi = 0; bi < kActBoxes; ++bi) mp.act_shared[bi] = mp.act_routed[bi];
        }
    }
    ChunkInstance* inst = (ChunkInstance*)ws.chunk_inst;
    const uint32_t max_inst = umma_max_chunk_instances(c, T);
    cudaError_t e = launch_after(m, st, chunk_instances_kernel, dim3(1), 256, 0, ws.expert_offsets, ws.expert_counts, ws.slot_of_expert,
                                 c.num_experts, T, (uint32_t)c.has_shared, pool_cells, inst, ws.n_chunk_inst, ws.status);
    if (e != cudaSuccess) return e;
    const uint32_t bits = c.weight_bits, grp = c.group_size;
    const bool f16 = c.meta_dtype == SHRIKE_DTYPE_FP16;
#define SHRIKE_UMMA(B, G, M) \
    return launch_umma_t<B, G, M>(m, st, a, inst, ws.n_chunk_inst, max_inst, maps[0], maps[1])
    if (bits == 4 && grp == 64 && !f16) SHRIKE_UMMA(4, 64, SHRIKE_DTYPE_BF16);
    if (bits == 4 && grp == 64 && f16) SHRIKE_UMMA(4, 64, SHRIKE_DTYPE_FP16);
    if (bits == 4 && grp == 32 && !f16) SHRIKE_UMMA(4, 32, SHRIKE_DTYPE_BF16);
    if (bits == 4 && grp == 32 && f16) SHRIKE_UMMA(4, 32, SHRIKE_DTYPE_FP16);
    if (bits == 8 && grp == 64 && !f16) SHRIKE_UMMA(8, 64, SHRIKE_DTYPE_BF16);
    if (bits == 8 && grp == 64 && f16) SHRIKE_UMMA(8, 64, SHRIKE_DTYPE_FP16);
    if (bits == 8 && grp == 32 && !f16) SHRIKE_UMMA(8, 32, SHRIKE_DTYPE_BF16);
    if (bits == 8 && grp == 32 && f16) SHRIKE_UMMA(8, 32, SHRIKE_DTYPE_FP16);
#undef SHRIKE_UMMA
    return cudaErrorInvalidValue;
}

}  // namespace shrike
