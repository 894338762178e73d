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
//   warp 19    takes tiles, streams the packed weights (64 or, for narrow tiles, 128
//              bytes of every row per copy: a 3-D TMA box of 128 rows of one matrix of one pool
//              cell, swizzled) and the group scales / biases (16 or 32 bytes
//              of every row per copy, or words of every row) into shared-memory rings. Whole-line TMA
//              requests keep the packed experts streaming at HBM speed where
//              per-thread 32-byte loads ran out of outstanding requests.
//   warp 18    copies the activation tiles: one or two boxes of 64 x
//              16 to 256 of the expert-sorted fp16 rows per K block, 128-byte
//              swizzle.
//   warps 0-15 converters: they turn the packed nibbles/bytes of a 64-wide K block into fp16
//              q * scale + bias (nibbles: (q - 8) * scale + (bias + 8 scale)) -- the reference's half(fma(q,
//              scale, bias)), tensorops.metal:106 -- and write them to TMEM (narrow tiles) or, 16 bytes at a
//              time, into the K-major 128-byte-swizzled tile in shared memory that the MMA reads.
//              After the K loop of a tile of more than 64 rows the same warps run the epilogue.
//   warps 16, 17  one elected thread of each issues tcgen05.mma (M 128, N = rows, K 16, fp16 in,
//              fp32 accumulate in TMEM) for one of the two tiles and commits to the
//              mbarriers that free the converted tile and the activation tile.
//   warps 20-23   epilogues of tiles of up to 64 rows, while the next tile is converted.
//
// PHASE 0: tile 0 = 128 gate rows, tile 1 = the matching 128 up rows; epilogue
//          GLU -> fp16 activations in operand layout, one row per sorted pair.
// PHASE 1: tiles = 256 consecutive down rows; epilogue (+ additive bias) x route
//          weight -> red.global.add into the token's fp32 accumulator row (the
//          weighted reduce, with no per-(row, rank) partial rows in between).
//
// What bounds it (256 experts of 2048 x 512, int4): at 256 rows a K block takes 0.74 to 0.76 us. That is 8.39 MFLOP on each of 148
// SMs: 1.63 to 1.68 PFLOP/s, as fast as the measured burst rate of a library GEMM (1.63). What is left of full tiles lies outside
// the K loop: 12,600 of a down tile's 25,800 cycles. With few rows the issue slots of the converters (70 % taken at 10 rows an expert; fp16
// arithmetic and logic run at half the rate there); 10 rows an expert take 93 us for gate/up and 62 for down, 2.9 TB/s.
//
// Every wait is bounded; a wait that gives up sets the status word and the
// block falls through to the TMEM release.
#include <cuda.h>
#include <algorithm>
#include <type_traits>

#include "internal.h"

namespace shrike {

constexpr uint32_t kUmmaMaxN = kChunkRows;
constexpr int kActBoxes = 5;
constexpr uint32_t kConverters = 512;                  // two threads per weight row
constexpr uint32_t kConvWarps = kConverters / 32;
constexpr uint32_t kEpiWarps = 4;
constexpr uint32_t kUmmaThreads = kConverters + 128 + kEpiWarps * 32;   // + two MMA warps, activation-copy warp, weight-copy warp, epilogue warps
constexpr uint32_t kSmallN = 64;                       // rows up to which TMEM holds two pairs of accumulators
constexpr uint32_t kConvRegs = 88, kOtherRegs = 64;    // of the 80 that 768 threads are launched with
static_assert(kConverters * kConvRegs + (kUmmaThreads - kConverters) * kOtherRegs <= kUmmaThreads * 80, "registers of a block");
constexpr uint32_t kTileBytes = 128 * 128;             // 128 rows x 64 fp16, one swizzle-128B K block
constexpr uint32_t kTiles = 4;                         // tiles that the copies may be ahead
// Shared memory of wide tiles (more than 128 rows):
//   [activations 3 x 32 KB][converted weights 2 x 32 KB][packed weights 3 x 16 KB][scales 8 KB]
constexpr uint32_t kWideB = 3, kWideA = 2, kWidePk = 3;
constexpr uint32_t kWideBBytes = kUmmaMaxN * 128, kWideABytes = 2 * kTileBytes;
constexpr uint32_t kWidePkBytes = 256 * 64;            // 64 packed bytes of 256 rows
constexpr uint32_t kWideScBytes = 2 * 256 * 16;        // 8 scales and biases of 256 rows
constexpr uint32_t kWideOffA = kWideB * kWideBBytes, kWideOffPk = kWideOffA + kWideA * kWideABytes;
constexpr uint32_t kWideOffSc = kWideOffPk + kWidePk * kWidePkBytes;
// and of narrow ones, whose converted weights go to TMEM: [activations 5 x 16 KB][packed weights 3 x 32 KB][scales 2 x 16 KB]
constexpr uint32_t kNarrowN = 128, kNarrowA = 2, kNarrowB = 5, kNarrowPk = 3, kNarrowSc = 2;
constexpr uint32_t kNarrowBBytes = kNarrowN * 128;     // a K block of 128 rows, two of 64 or four of 32
constexpr uint32_t kNarrowPkBytes = 256 * 128;         // 128 packed bytes of 256 rows
constexpr uint32_t kNarrowScBytes = 2 * 256 * 32;      // 16 scales and biases of 256 rows
constexpr uint32_t kNarrowOffPk = kNarrowB * kNarrowBBytes, kNarrowOffSc = kNarrowOffPk + kNarrowPk * kNarrowPkBytes;
// Rows of an odd number of scales: every odd row's word past its scale block, [stage][scales, biases][128] (wide tiles: a stage).
constexpr uint32_t kOffPast = kWideOffSc + kWideScBytes, kPastBytes = 128 * 4;
static_assert(kNarrowOffSc + kNarrowSc * kNarrowScBytes <= kOffPast, "narrow tiles' scales");
constexpr uint32_t kOffBar = kOffPast + kNarrowSc * 2 * kPastBytes;
constexpr uint32_t kNumBars = 2 * (kWideB + kWideA + kWidePk + 1) + 1 + 2 * (kNarrowA + kNarrowB + kNarrowPk + kNarrowSc) + 2 + 3 * kTiles + 2;
constexpr uint32_t kOffTiles = (kOffBar + kNumBars * 8 + 15) / 16 * 16;
constexpr uint32_t kUmmaSmemBytes = kOffTiles + kTiles * 16 + 4 * kUmmaMaxN * 4 + 4 * kSmallN * 4 + 16 + 1024 /*alignment slack*/;
static_assert(kUmmaSmemBytes + 1024 <= 227 * 1024, "shared memory of a block");

struct WeightMaps {       // TMA descriptors of the two 128-row tiles of a block
    CUtensorMap w[2];     // packed weights   [cells][rows][row bytes]
    CUtensorMap s[2];     // group scales     [cells][rows][groups]
    CUtensorMap b[2];     // group biases
    CUtensorMap nw[2], ns[2], nb[2];   // the same in the boxes of narrow tiles, twice as wide
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
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
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
__device__ __forceinline__ void mbar_arrive(uint64_t* bar, uint32_t count = 1) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
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

// 8 packed nibbles -> 8 fp16 weights in operand order {0,4,1,5,2,6,3,7}; 4 bytes -> 4 fp16 in order. A byte q in a half's low bits is
// the fp16 number q x 2^-24, below the normal range and exact: it is multiplied as it lies there, by a scale of 2^24 times the
// group's, with one rounding in all and no subtraction of an offset (256 experts of 2304 x 1024, 2064 rows, 707 -> 695 us a call).
// (Nibbles the same way, at bit 4: no faster, 333 rows 177 us with the subtractions, 180 without.)
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
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(out[0]) : "r"(prmt(w, 0u, 0x4140u)), "r"(s2), "r"(z2));
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(out[1]) : "r"(prmt(w, 0u, 0x4342u)), "r"(s2), "r"(z2));
    }
}
// A byte's scale of 2^-9 and above is made 2^-k times as large, the power of two that keeps 2^24 times it below 2^15 and in fp16's
// range, and so are its weights, which are multiplied by 2^k afterwards.
constexpr float kScaleUp = 16777216.0f;
__device__ __forceinline__ float power_of_two(int k) { return __uint_as_float((uint32_t)(127 + k) << 23); }
__device__ __forceinline__ int scale_excess(float scale) {
    return max(0, min((int)((__float_as_uint(scale) >> 23) & 0xffu) - 127 + 24 - 14, 126));
}
template <int N>
__device__ __forceinline__ void scale_weights(uint32_t (&o)[N], int k) {
    uint32_t m0, m1;   // 2^k may be more than fp16 holds
    asm("cvt.rn.f16x2.f32 %0, %1, %1;" : "=r"(m0) : "f"(power_of_two(min(k, 15))));
    asm("cvt.rn.f16x2.f32 %0, %1, %1;" : "=r"(m1) : "f"(power_of_two(max(k - 15, 0))));
#pragma unroll
    for (int i = 0; i < N; ++i) {
        asm("mul.rn.f16x2 %0, %0, %1;" : "+r"(o[i]) : "r"(m0));
        asm("mul.rn.f16x2 %0, %0, %1;" : "+r"(o[i]) : "r"(m1));
    }
}

__device__ __forceinline__ uint32_t half2_dup(float v) {
    uint32_t h;
    asm("cvt.rn.f16x2.f32 %0, %1, %1;" : "=r"(h) : "f"(v));
    return h;
}

template <int C>
__device__ __forceinline__ void tmem_ld_issue(uint32_t taddr, uint32_t (&r)[C]) {
    static_assert(C == 4 || C == 8, "columns");
    if constexpr (C == 4)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
    else
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

// Bounded wait for the pipeline barriers: these are on the critical path of every K block, so the first polls do not sleep.
// False when the time is up, or another role's was. (Inlined: around a call the converters moved their registers.)
__device__ __forceinline__ bool pipe_wait_or(uint64_t* bar, uint32_t parity, const volatile uint32_t* failed) {
    const uint32_t addr = smem_u32(bar);
#pragma unroll 1
    for (uint32_t it = 0; it < (1u << 21); ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(addr), "r"(parity) : "memory");
        if (ok) return true;
        if (it > 256) {
            __nanosleep(32);
            if (*failed) return false;
        }
    }
    return false;
}
// Whether the phase is over, without waiting.
__device__ __forceinline__ bool pipe_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}

template <int N>
__device__ __forceinline__ void load_words(const uint8_t* from, uint32_t (&w)[N]) {
    static_assert(N == 1 || N == 2 || N == 4, "words");
    if constexpr (N == 4) {
        const uint4 v = *(const uint4*)from;
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else if constexpr (N == 2) {
        const uint2 v = *(const uint2*)from;
        w[0] = v.x; w[1] = v.y;
    } else {
        w[0] = *(const uint32_t*)from;
    }
}

// 16-bit field `idx` (0..7) of four registers.
__device__ __forceinline__ uint16_t pick16(const uint32_t (&v)[4], uint32_t idx) {
    const uint32_t lo = (idx & 2u) ? v[1] : v[0], hi = (idx & 2u) ? v[3] : v[2];
    const uint32_t w = (idx & 4u) ? hi : lo;
    return (uint16_t)((idx & 1u) ? (w >> 16) : (w & 0xffffu));
}

// The instance's rows as one or two boxes of 16 << i rows (the largest that fits, then the smallest that holds the rest).
struct TileShape {
    uint32_t N, n1, b1, n2, b2;
    __device__ explicit TileShape(uint32_t count) {
        N = (count + 15u) & ~15u;           // MMA N: rows padded to 16
        n1 = 16; b1 = 0;
        while ((n1 << 1) <= N && b1 + 1 < (uint32_t)kActBoxes) { n1 <<= 1; ++b1; }
        n2 = 0; b2 = 0;
        if (N > n1) {
            n2 = 16;
            while (n2 < N - n1) { n2 <<= 1; ++b2; }
        }
    }
};

// K blocks of activations in a narrow tile's stage, less one. A copy of activations waits in the SM's copy engine behind the packed
// weights, 32 KB at a time: with a K block a stage and four stages the tensor core waited 660 cycles for each of 16 rows.
__device__ __forceinline__ uint32_t narrow_b_mask(uint32_t count) { return count <= 32 ? 3u : count <= 64 ? 1u : 0u; }

// A tile as the weight copy hands it to the other roles: rows r0 and on of the matrix against the rows first .. first + count
// of the sorted pairs (the shared expert: of the call); count 0 ends the list.
struct Tile {
    uint32_t slot, first, r0, count;
    bool shared, narrow;
    __device__ Tile() {}
    __device__ explicit Tile(const uint4& v)
        : slot(v.x), first(v.y), r0(v.z & 0x7fffffffu), count(v.w), shared(v.z >> 31), narrow(v.w <= kNarrowN) {}
};

// A persistent block per SM; tiles (instance, 128 or 256 weight rows) come from a counter, in list order: wide ones (129 to 256
// rows) first. The copy threads run ahead into the next tiles while the converters finish this one: as one block per tile, set-up,
// the first copies' way and the launch gap cost 4 us of every tile's 8 (512 x 16 columns) to 37 (2048 x 256).
//
// Wide tiles are bound by the tensor core, narrow ones by the converters' instructions, and have loops of their own:
//   wide    all converters on every K block, a thread 32 of a row's 64 weights, into shared memory; both accumulators fill TMEM, so
//           a tile ends before the next begins;
//   narrow  the converters in two sets of eight warps on alternate K blocks, a thread all 64 weights of its row, into TMEM: half
//           the waits, arrivals and scales per weight, and while a set waits the other converts. The tensor core is told of two K
//           blocks at a time. Up to 64 rows there are two pairs of accumulators, and warps of their own for the epilogues.
// 10 rows an expert, gate/up and down: 136 + 98 us with all converters on every K block and one loop for both kinds of tile, 121 +
// 100 in two sets, 106 + 82 with an issuing warp per weight tile (a single one needed 650 cycles for a K block), 101 + 72 with
// epilogue warps, 93 + 62 with the questions to barriers asked before their answers are needed. Deeper rings of copies, wider
// boxes and fewer boxes of scales changed nothing: the bytes are there in time.
// SCT: rows of scales are whole 16-byte units and come by TMA; others (groups % 8 != 0) word by word (cp.async), into the same places.
// Read by the converters themselves, a block ahead and through registers, their waits for a stage were waits for DRAM too: 32
// experts of 2880 x 2880 in groups of 32 took 900 cycles for a K block and 6000 until a tile's first one, now 780 and 350 (host
// call of 777 rows 519 -> 492 us).
template <int BITS, int GROUP, int META, int PHASE, bool SCT>
__global__ void __launch_bounds__(kUmmaThreads, 1)
umma_expert_kernel(const ExpertArgs a, const ChunkInstance* __restrict__ inst, uint32_t* __restrict__ n_inst,
                   const uint32_t row_tiles, const __grid_constant__ UmmaMaps maps) {
    constexpr uint32_t kRowBlockBytes = 64 * BITS / 8;  // packed bytes of one row per K block (32 or 64)
    constexpr uint32_t kWordsPerBlock = kRowBlockBytes / 4;
    constexpr uint32_t kGroupsPerBlock = 64 / GROUP;    // 1 (g64) or 2 (g32)
    constexpr uint32_t kKbPerSc = 8 / kGroupsPerBlock;  // K blocks per eight groups (8 or 4)
    constexpr uint32_t kWideKbPerPk = 64 / kRowBlockBytes, kNarrowKbPerPk = 2 * kWideKbPerPk;   // K blocks per packed copy
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    if (PHASE == 1) pdl_launch_dependents();
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (smem_base - smem_u32(smem_raw));
    uint64_t* bars = (uint64_t*)(smem + kOffBar);
    // wide tiles
    uint64_t* a_full = bars;                       // converters -> MMA
    uint64_t* a_empty = a_full + kWideA;           // MMA -> converters
    uint64_t* b_full = a_empty + kWideA;           // activation copy -> MMA
    uint64_t* b_empty = b_full + kWideB;           // MMA -> activation copy
    uint64_t* pk_full = b_empty + kWideB;          // weight copy -> converters
    uint64_t* pk_empty = pk_full + kWidePk;        // converters -> weight copy
    uint64_t* sc_full = pk_empty + kWidePk;
    uint64_t* sc_empty = sc_full + 1;
    uint64_t* wide_over = sc_empty + 1;            // MMA -> copies: nothing reads the wide tiles' memory any more
    // narrow tiles
    uint64_t* na_full = wide_over + 1;
    uint64_t* na_empty = na_full + kNarrowA;
    uint64_t* nb_full = na_empty + kNarrowA;
    uint64_t* nb_empty = nb_full + kNarrowB;
    uint64_t* npk_full = nb_empty + kNarrowB;
    uint64_t* npk_empty = npk_full + kNarrowPk;
    uint64_t* nsc_full = npk_empty + kNarrowPk;
    uint64_t* nsc_empty = nsc_full + kNarrowSc;
    // all
    uint64_t* accum = nsc_empty + kNarrowSc;       // [kTiles] MMA -> epilogue: all of a tile's MMAs are done, tiles in turn
    uint64_t* epi_done = accum + kTiles;                // [2] converters -> MMA: a tile's accumulators have been read
    uint64_t* tile_full = epi_done + 2;            // [kTiles] weight copy -> everyone: the next tile
    uint64_t* tile_empty = tile_full + kTiles;
    uint64_t* conv = tile_empty + kTiles;          // the converter warps among themselves (a named barrier has no bounded wait)
    uint64_t* eids_full = conv + 1;                // the epilogue warps among themselves
    uint4* next_tile = (uint4*)(smem + kOffTiles);                  // [kTiles]
    uint32_t* rowid = (uint32_t*)(next_tile + kTiles);              // token of a column: [2][256], tiles in turn
    float* roww = (float*)(rowid + 2 * kUmmaMaxN);                  // route weight (routed) or gate (shared)
    uint32_t* small_id = (uint32_t*)(roww + 2 * kUmmaMaxN);          // the same of a small tile: [2][64], tiles in turn
    float* small_w = (float*)(small_id + 2 * kSmallN);
    uint32_t* tmem_slot = (uint32_t*)(small_w + 2 * kSmallN);
    __shared__ uint32_t s_failed;

    if (tid == 0) {
        for (uint32_t s = 0; s < kWideA; ++s) { mbar_init(&a_full[s], kConvWarps); mbar_init(&a_empty[s], 2); }
        for (uint32_t s = 0; s < kWideB; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_empty[s], 2); }
        for (uint32_t s = 0; s < kWidePk; ++s) { mbar_init(&pk_full[s], 1); mbar_init(&pk_empty[s], kConvWarps); }
        mbar_init(sc_full, SCT ? 1 : 64);
        mbar_init(sc_empty, kConvWarps);
        mbar_init(wide_over, 2);
        for (uint32_t s = 0; s < kNarrowA; ++s) { mbar_init(&na_full[s], kConvWarps); mbar_init(&na_empty[s], 2); }
        for (uint32_t s = 0; s < kNarrowB; ++s) { mbar_init(&nb_full[s], 1); mbar_init(&nb_empty[s], 2); }
        for (uint32_t s = 0; s < kNarrowPk; ++s) { mbar_init(&npk_full[s], 1); mbar_init(&npk_empty[s], kConvWarps); }
        for (uint32_t s = 0; s < kNarrowSc; ++s) { mbar_init(&nsc_full[s], SCT ? 1 : 64); mbar_init(&nsc_empty[s], kConvWarps); }
        for (uint32_t s = 0; s < 2; ++s) mbar_init(&epi_done[s], kConvWarps);
        for (uint32_t s = 0; s < kTiles; ++s) { mbar_init(&accum[s], 2); mbar_init(&tile_full[s], 1); mbar_init(&tile_empty[s], kConvWarps + 3 + kEpiWarps); }
        mbar_init(conv, kConvWarps);
        mbar_init(eids_full, kEpiWarps);
        fence_mbar_init();
        s_failed = 0;
    }
    // two accumulators of up to 256 columns: all of TMEM (a block per SM)
    if (warp == kConvWarps) tmem_alloc(smem_u32(tmem_slot), 2 * kUmmaMaxN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // All of the above runs while the last kernel ends. The down projection takes its first tiles and converts their weights
    // meanwhile: of what comes before, only the activations are the gate/up launch's, and the warp that copies them waits. The list, the
    // pairs and the cleared rows were there when that launch let this one start (they are read past L1). 333 rows 196 -> 187 us a
    // call, 4096 rows 498 -> 490.
    if (PHASE == 0) {
        pdl_wait();
        pdl_launch_dependents();
    }
    auto give_up = [&]() {
        report_status(a.status, kStatusWaitTimeout);
        *(volatile uint32_t*)&s_failed = 1;
    };
    auto failed = [&]() { return *(volatile uint32_t*)&s_failed != 0; };
    auto pipe_wait = [&](uint64_t* bar, uint32_t parity) { return pipe_wait_or(bar, parity, &s_failed); };
    // Tile number n of this block (all lanes); false: there is none.
    auto release_tile = [&](uint32_t n) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&tile_empty[n % kTiles]);
    };
    auto take_tile = [&](uint32_t n, Tile& t, bool release = true) {
        const uint32_t s = n % kTiles;
        if (!__all_sync(0xffffffffu, pipe_wait(&tile_full[s], (n / kTiles) & 1))) { give_up(); return false; }
        const uint4 v = next_tile[s];
        if (release) release_tile(n);
        t = Tile(v);
        return t.count != 0;
    };
    auto k_blocks = [&](const Tile& t) { return (PHASE == 0 ? a.d : t.shared ? a.f_shared : a.f) / 64; };
    // Epilogue of tile `e`, the block's n-th, by H x 4 warps: warp w reads TMEM lanes 32*(w & 3) .. +31, every H-th group of C columns
    // from the h-th on; accumulators at columns acc0 and acc1, the columns' tokens and weights at `ids` and `wts`.
    auto epilogue = [&](auto width, auto share, uint32_t h, const Tile& e, uint32_t n, uint32_t acc0, uint32_t acc1, const uint32_t* ids, const float* wts) {
        constexpr int C = decltype(width)::value, H = decltype(share)::value;
        if (!pipe_wait(&accum[n % kTiles], (n / kTiles) & 1)) give_up();
        if (failed()) return false;
        __syncwarp();
        tc_fence_after();
        const Offsets3& off = e.shared ? a.shared : a.routed;
        const uint8_t* base = e.shared ? a.shared_block : pool_cell_base(a.pool, e.slot);
        const uint32_t F = e.shared ? a.f_shared : a.f, N = (e.count + 15u) & ~15u;
        // (loops that are not unrolled further: the code runs once per tile, and fetching it takes longer than what
        // unrolling saves)
        const uint32_t q = warp & 3;
        const uint32_t trow = q * 32 + lane;                       // row inside each 128-row tile
        const uint32_t taddr = tmem_base + ((q * 32) << 16);
        constexpr uint32_t kColStep = C * H;
        if (PHASE == 0) {
            const uint32_t f = e.r0 + trow;
            float gab = 0.f, uab = 0.f;
            if (a.expert_bias && f < F) {
                gab = bf16_bits_to_f32(((const uint16_t*)(base + off.ab[0]))[f]);
                uab = bf16_bits_to_f32(((const uint16_t*)(base + off.ab[1]))[f]);
            }
            uint16_t* const dst = (e.shared ? a.acts_shared : a.acts) + (size_t)e.first * F + perm_index(f, BITS == 4);
            auto columns = [&](auto glu_of) {
                bool over = false;
#pragma unroll 1
                for (uint32_t c0 = h * C; c0 < N; c0 += kColStep) {
                    uint32_t g[C], u[C];
                    tmem_ld_issue<C>(taddr + acc0 + c0, g);
                    tmem_ld_issue<C>(taddr + acc1 + c0, u);
                    tmem_ld_wait();
                    uint16_t* p = dst + (size_t)c0 * F;
                    const uint32_t live = f < F ? min((uint32_t)C, e.count > c0 ? e.count - c0 : 0u) : 0u;   // rows of this group
#pragma unroll
                    for (int j = 0; j < C; j += 2) {
                        float v[2];
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            v[k] = glu_of(__uint_as_float(g[j + k]) + gab, __uint_as_float(u[j + k]) + uab);
                            if (fabsf(v[k]) > kHalfMax) {   // false for NaN, which passes through
                                over |= (uint32_t)(j + k) < live;
                                v[k] = copysignf(kHalfMax, v[k]);
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
            const uint32_t d0 = e.r0 + trow, d1 = d0 + 128;
            float ab0 = 0.f, ab1 = 0.f;
            if (a.expert_bias) {
                const uint16_t* dab = (const uint16_t*)(base + off.ab[2]);
                if (d0 < a.d) ab0 = bf16_bits_to_f32(dab[d0]);
                if (d1 < a.d) ab1 = bf16_bits_to_f32(dab[d1]);
            }
            const bool ok0 = d0 < a.d, ok1 = d1 < a.d;
#pragma unroll 1
            for (uint32_t c0 = h * C; c0 < N; c0 += kColStep) {
                uint32_t v0[C], v1[C];
                tmem_ld_issue<C>(taddr + acc0 + c0, v0);
                tmem_ld_issue<C>(taddr + acc1 + c0, v1);
                tmem_ld_wait();
                const uint32_t live = min((uint32_t)C, e.count > c0 ? e.count - c0 : 0u);
#pragma unroll
                for (int j = 0; j < C; ++j) {
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
        tc_fence_before();   // these reads of the accumulators come before the instructions that write them next
        __syncwarp();
        if (lane == 0) mbar_arrive(&epi_done[n & 1], kConvWarps / (4 * H));
        return true;
    };
    // Barriers' parities: a stage's use n (counted by each role for itself) is waited for with n & 1 at its full barrier, and with the
    // complement at the empty one. Accumulators and ids: by the number of the tile.

    if (warp < kConvWarps) {
        // ---------------- converters, and the tiles' epilogues ----------------
        // A lane is a row: the TMEM lanes that a warp reaches. half: of a K block (wide), or which K blocks (narrow).
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kConvRegs));
        const uint32_t tile = (warp >> 2) & 1, r = (warp & 3) * 32 + lane, half = warp >> 3;
        uint32_t conv_use = 0;
        auto converters_meet = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(conv);
            const bool ok = pipe_wait(conv, conv_use);
            conv_use ^= 1;
            if (!ok) give_up();
            return ok;
        };
        // ---- of the tile at hand ----
        Tile t;
        uint32_t KB;
        uint32_t col_pair = 0;              // the pair (shared: row) behind this thread's column, and its weight
        float col_w = 0.f;
        auto open_tile = [&]() {
            KB = k_blocks(t);
            if (PHASE == 1 && t.count > kSmallN && tid < t.count) col_pair = t.shared ? t.first + tid : __ldcg(a.sorted + t.first + tid);
        };
        // The columns' tokens and route weights, for the epilogue: asked for when the tile begins (its weight once the pair is
        // there), stored when its weights are converted -- a store at the start waits for two trips to L2.
        auto ask_weight = [&]() {
            if (PHASE == 1 && tid < t.count) col_w = t.shared ? (a.shared_gate ? __ldcg(a.shared_gate + col_pair) : 1.0f) : __ldcg(a.route_w + col_pair);
        };
        auto own_epilogue = [&](auto width, uint32_t n, uint32_t acc1) {
            const uint32_t at = (n & 1) * kUmmaMaxN;
            if (PHASE == 1) {
                if (tid < t.count) {
                    rowid[at + tid] = t.shared ? col_pair : col_pair / a.top_k;
                    roww[at + tid] = col_w;
                }
                if (!converters_meet()) return false;
            }
            return epilogue(width, std::integral_constant<int, 4>(), warp >> 2, t, n, 0u, acc1, rowid + at, roww + at);
        };
        // Whether this row's scales begin with one of the row before: an odd row of an odd number of them.
        auto past = [&]() { return !SCT && GROUP == 64 && (KB & r & 1u) != 0; };
        // N words of scales become those that begin a half later.
        auto shift_in = [&](auto& v, uint32_t next) {
            constexpr int N = sizeof v / 4;
#pragma unroll
            for (int i = 0; i < N; ++i) v[i] = __funnelshift_r(v[i], i + 1 < N ? v[i + 1 < N ? i + 1 : i] : next, 16);
        };
        // True for the warp when a lane's scale is too large for dequant_word(): the weights then take scale_weights() as well.
        auto scale_words = [&](uint32_t s16, uint32_t b16, uint32_t& s2, uint32_t& z2) {
            const float sc = meta_to_f32<META>((uint16_t)s16), bi = meta_to_f32<META>((uint16_t)b16);
            if constexpr (BITS == 4) {
                s2 = half2_dup(sc);
                z2 = half2_dup(fmaf(8.0f, sc, bi));   // the zero point is 8 less
                return false;
            }
            const float up = sc * kScaleUp;
            s2 = half2_dup(up);
            z2 = half2_dup(bi);
            if (!__any_sync(0xffffffffu, !(fabsf(up) < 32768.0f))) return false;
            const float by = power_of_two(-scale_excess(sc));
            s2 = half2_dup(up * by);
            z2 = half2_dup(bi * by);
            return true;
        };

        uint32_t n = 0;
        bool go = take_tile(0, t), was_wide = false;
        // ---- wide tiles ----
        {
            uint32_t a_use = 0, pk_use = 0, sc_use = 0, slot = 0, st = 0;
            constexpr uint32_t kWordsPerThread = kWordsPerBlock / 2;   // 4 (int4) or 8 (int8)
            const uint32_t pk_row = kWideOffPk + tile * (kWidePkBytes / 2) + r * 64, pk_xor = (r >> 1) & 3;
            // What does not change along K: this thread's chunk positions in a packed slot and in the converted
            // tile (both swizzled by the row).
            uint32_t pk_off[kWideKbPerPk * (kWordsPerThread / 4)];
#pragma unroll
            for (uint32_t sub = 0; sub < kWideKbPerPk; ++sub)
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
            for (; go && !t.narrow; go = take_tile(++n, t)) {
                was_wide = true;
                open_tile();
                // A scale block (8 groups of the row) at a time, its K blocks unrolled: the position in the packed slot
                // and the group of a K block are then constants of the instruction stream.
                for (uint32_t kb0 = 0; kb0 < KB; kb0 += kKbPerSc) {
                    if (failed()) break;
                    if (!pipe_wait(sc_full, sc_use)) { give_up(); break; }
                    sc_use ^= 1;
                    const uint8_t* const from = smem + kWideOffSc + (tile * 128 + r) * 16;
                    uint32_t sreg[4], breg[4];
                    load_words<4>(from, sreg);
                    load_words<4>(from + kWideScBytes / 2, breg);
                    if (past()) {
                        const uint32_t* const more = (const uint32_t*)(smem + kOffPast) + (tile * 128 + r) / 2;
                        shift_in(sreg, more[0]);
                        shift_in(breg, more[kPastBytes / 4]);
                    }
                    // the values are in registers: the copy thread may fetch the next block's
                    __syncwarp();
                    if (lane == 0) mbar_arrive(sc_empty);
#pragma unroll
                    for (uint32_t j = 0; j < kKbPerSc; ++j) {
                        const uint32_t kb = kb0 + j;
                        if (kb >= KB) break;
                        constexpr uint32_t kSubMask = kWideKbPerPk - 1;
                        const uint32_t sub = j & kSubMask;         // K block within its packed slot
                        if (sub == 0 && !pipe_wait(&pk_full[slot], (pk_use >> slot) & 1)) { give_up(); break; }
                        if (j == 2 && kb0 == 0) ask_weight();
                        uint32_t pk[kWordsPerThread];
#pragma unroll
                        for (uint32_t q = 0; q < kWordsPerThread / 4; ++q) {
                            const uint4 v = *(const uint4*)(smem + slot * kWidePkBytes + pk_off[sub * (kWordsPerThread / 4) + q]);
                            pk[4 * q] = v.x; pk[4 * q + 1] = v.y; pk[4 * q + 2] = v.z; pk[4 * q + 3] = v.w;
                        }
                        // a thread's half of a 64-wide block lies inside one group of 32 or 64
                        const uint32_t gsel = j * kGroupsPerBlock + (GROUP == 64 ? 0u : half);
                        uint32_t s2, z2;
                        const uint32_t s16 = pick16(sreg, gsel);
                        const bool large = scale_words(s16, pick16(breg, gsel), s2, z2);
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
                        if (large) scale_weights(o, scale_excess(meta_to_f32<META>((uint16_t)s16)));
                        uint8_t* a_stage = smem + kWideOffA + st * kWideABytes;
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i)
                            *(uint4*)(a_stage + a_pos[i]) = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
                        fence_async_smem();
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
                            if (++slot == kWidePk) slot = 0;
                        }
                        if (++st == kWideA) st = 0;
                    }
                }
                if (KB <= 2) ask_weight();
                if (!own_epilogue(std::integral_constant<int, 8>(), n, kUmmaMaxN)) break;
            }
        }
        // ---- narrow tiles ----
        // (a warp may write weights and columns while others still read what they take of the last accumulators)
        if (go && was_wide && !failed()) go = converters_meet();
        {
            static_assert(kNarrowA == 2, "stages in turn");
            uint32_t a_st = 0, a_par = 1, slot = 0, pk_par = 0, ss = 0, sc_par = 0, in_sc = 0;
            auto next_pair = [&]() { a_st ^= 1u; a_par ^= a_st ^ 1u; };
            const uint32_t a_tmem = tmem_base + 256u + (((warp & 3) * 32) << 16) + half * 64 + tile * 32;
            // 16-byte chunks of this thread's K block in its row of 128 packed bytes: the second of int4's two is 64 bytes on
            constexpr uint32_t kChunks = kRowBlockBytes / 16;
            uint32_t pk_off[kChunks];
#pragma unroll
            for (uint32_t q = 0; q < kChunks; ++q)
                pk_off[q] = kNarrowOffPk + tile * (kNarrowPkBytes / 2) + r * 128 + (((half * kChunks + q) ^ (r & 7)) << 4);
            uint32_t pk[kWordsPerBlock];
            auto load_packed = [&](uint32_t i) {   // of K block i (+ half) in the slot
#pragma unroll
                for (uint32_t q = 0; q < kChunks; ++q) {
                    const uint4 v = *(const uint4*)(smem + slot * kNarrowPkBytes + (pk_off[q] ^ (i * kRowBlockBytes)));
                    pk[4 * q] = v.x; pk[4 * q + 1] = v.y; pk[4 * q + 2] = v.z; pk[4 * q + 3] = v.w;
                }
            };
            // Eight groups' scales are kRawWords words for each of kSlotsPerSc slots.
            constexpr uint32_t kRawWords = kNarrowKbPerPk * kGroupsPerBlock / 2, kSlotsPerSc = kKbPerSc / kNarrowKbPerPk, kOwn = kNarrowKbPerPk / 2;
            const uint32_t sc_row = kNarrowOffSc + (tile * 128 + r) * 32;
            // What the next slot's first own K block needs, asked for as soon as the slot is there.
            uint32_t rs[kRawWords], rb[kRawWords];
            auto open_slot = [&](uint32_t kb0) {
                const uint8_t* const from = smem + sc_row + ss * kNarrowScBytes + in_sc * (kRawWords * 4);
                load_words<kRawWords>(from, rs);
                load_words<kRawWords>(from + kNarrowScBytes / 2, rb);
                if (past()) {
                    const bool end = (in_sc + 1) * kRawWords == 8;
                    const uint8_t* const more = end ? smem + kOffPast + ss * 2 * kPastBytes + (tile * 128 + r) / 2 * 4 : from + kRawWords * 4;
                    shift_in(rs, *(const uint32_t*)more);
                    shift_in(rb, *(const uint32_t*)(more + (end ? kPastBytes : kNarrowScBytes / 2)));
                }
                if (kb0 + half < KB) load_packed(0);
            };
            for (; go; go = take_tile(++n, t)) {
                open_tile();
                if (!pipe_wait(&nsc_full[ss], sc_par)) { give_up(); break; }
                if (!pipe_wait(&npk_full[slot], pk_par)) { give_up(); break; }
                open_slot(0);
                for (uint32_t kb0 = 0; kb0 < KB; kb0 += kNarrowKbPerPk) {
                    const bool last = kb0 + kNarrowKbPerPk >= KB;
                    // ---- the slot's scales and biases: own K block i's in sw[i], bw[i] (in the low bits, or both groups') ----
                    uint32_t sw[kOwn], bw[kOwn];
#pragma unroll
                    for (uint32_t i = 0; i < kOwn; ++i) {
                        if constexpr (GROUP == 32) {
                            sw[i] = half ? rs[2 * i + 1] : rs[2 * i];
                            bw[i] = half ? rb[2 * i + 1] : rb[2 * i];
                        } else {
                            sw[i] = rs[i] >> (16 * half);
                            bw[i] = rb[i] >> (16 * half);
                        }
                    }
                    const uint32_t slot1 = slot + 1 == kNarrowPk ? 0u : slot + 1, pk_par1 = slot1 ? pk_par : pk_par ^ 1;
                    const bool there = pipe_test(&npk_full[slot1], pk_par1);   // (the answer takes its time: looked at below)
                    // ---- its K blocks that are this set's ----
#pragma unroll
                    for (uint32_t i = 0; i < kOwn; ++i) {
                        const uint32_t kb = kb0 + 2 * i + half;
                        if (kb >= KB) break;
                        const bool free = pipe_test(&na_empty[a_st], a_par);
                        uint32_t s2, z2;
                        bool large = scale_words(sw[i] & 0xffffu, bw[i] & 0xffffu, s2, z2);
#pragma unroll
                        for (uint32_t h = 0; h < 2; ++h) {   // 32 weights, 16 columns at a time: half the registers
                            if (GROUP == 32 && h) large = scale_words(sw[i] >> 16, bw[i] >> 16, s2, z2);
                            uint32_t o[16];
#pragma unroll
                            for (uint32_t w = 0; w < kWordsPerBlock / 2; ++w) {
                                uint32_t w4[4];
                                dequant_word<BITS>(pk[h * (kWordsPerBlock / 2) + w], s2, z2, w4);
#pragma unroll
                                for (uint32_t e = 0; e < 32 / kWordsPerBlock; ++e) o[w * (32 / kWordsPerBlock) + e] = w4[e];
                            }
                            if (large) scale_weights(o, scale_excess(meta_to_f32<META>((uint16_t)(GROUP == 32 && h ? sw[i] >> 16 : sw[i]))));
                            if (h == 0) {
                                if (!free && !pipe_wait(&na_empty[a_st], a_par)) { give_up(); break; }
                                __syncwarp();
                                tc_fence_after();   // the stage's last readers are done
                            }
                            tmem_st16(a_tmem + a_st * 128 + h * 16, o);
                        }
                        if (i + 1 < kOwn && kb + 2 < KB) load_packed(2 * (i + 1));
                        tmem_st_wait();
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&na_full[a_st]);
                        next_pair();
                    }
                    // handed back only here: the values read from them have been consumed
                    const bool sc_done = ++in_sc == 2 * kSlotsPerSc || last;
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&npk_empty[slot]);
                        if (sc_done) mbar_arrive(&nsc_empty[ss]);
                    }
                    if (sc_done) {
                        in_sc = 0;
                        if (++ss == kNarrowSc) { ss = 0; sc_par ^= 1; }
                    }
                    slot = slot1;
                    pk_par = pk_par1;
                    if (!last) {
                        if (sc_done && !pipe_wait(&nsc_full[ss], sc_par)) { give_up(); break; }
                        if (!there && !pipe_wait(&npk_full[slot], pk_par)) { give_up(); break; }
                        open_slot(kb0 + kNarrowKbPerPk);
                    }
                    if (kb0 == 0 && t.count > kSmallN) ask_weight();
                }
                if (failed()) break;
                if (half && (KB & 1)) {   // the last pair has no second K block
                    if (!pipe_wait(&na_empty[a_st], a_par)) { give_up(); break; }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&na_full[a_st]);
                    next_pair();
                }
                if (t.count > kSmallN && !own_epilogue(std::integral_constant<int, 4>(), n, 128u)) break;
            }
        }
    } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
    auto wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, pipe_wait(bar, parity)) != 0; };
    auto any_failed = [&]() { return __any_sync(0xffffffffu, failed()) != 0; };
    // Weight tile m: W words of every row's scales and biases from group g0 on, 128 rows from row0 on; of an odd row of an odd number
    // of groups, from the word that the first one shares with the row before, and a word more. What lies past the matrix reads
    // as zero. (By one warp for both weight tiles: 100 rows of 32 experts of 2880 x 2880 239 us a call, by a warp each 197.)
    auto copy_scales = [&](auto width, uint32_t m, const Tile& t, uint32_t g0, uint32_t row0, uint32_t to, uint32_t to_past, uint64_t* bar) {
        constexpr uint32_t W = decltype(width)::value, kStep = 32 / W, kBias = 256 * W * 4;
        const Offsets3& off = t.shared ? a.shared : a.routed;
        const uint8_t* const base = t.shared ? a.shared_block : pool_cell_base(a.pool, t.slot);
        const uint32_t G = k_blocks(t) * 64 / GROUP, odd = G & 1u, stride = kStep * G * 2;
        const int32_t total = (int32_t)((PHASE == 0 ? t.shared ? a.f_shared : a.f : a.d) * G);
        auto word = [&](uint32_t dst, const uint8_t* sp, const uint8_t* bp, int32_t at, uint32_t bias_dst) {
            const uint32_t n = (uint32_t)max(0, min(2 * (total - at), 4));
            const size_t from = n ? (size_t)at * 2 : 0;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(sp + from), "r"(n) : "memory");
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + bias_dst), "l"(bp + from), "r"(n) : "memory");
        };
        const int mat = PHASE == 0 ? (int)m : 2;
        const uint8_t *const sp = base + off.s[mat], *const bp = base + off.b[mat];
        const uint32_t row = lane / W, dst = to + (m * 128 * W + lane) * 4;
        const int32_t at = (int32_t)((row0 + row) * G + g0 + 2 * (lane % W) - (row & odd));
        if ((int32_t)((row0 + 127) * G + g0 + 2 * W) <= total) {   // (most of the warp's instructions; the copies of weights wait for them)
            const uint8_t *s_at = sp + (size_t)at * 2, *b_at = bp + (size_t)at * 2;
#pragma unroll 8
            for (uint32_t q = 0; q < 128 / kStep; ++q, s_at += stride, b_at += stride) {
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + q * 128), "l"(s_at) : "memory");
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + q * 128 + kBias), "l"(b_at) : "memory");
            }
        } else {
#pragma unroll 1
            for (uint32_t q = 0; q < 128 / kStep; ++q) word(dst + q * 128, sp, bp, at + (int32_t)(q * kStep * G), kBias);
        }
        if (odd)
#pragma unroll 1
            for (uint32_t i = lane; i < 64; i += 32)
                word(to_past + (m * 64 + i) * 4, sp, bp, (int32_t)((row0 + 2 * i + 1) * G + g0 + 2 * W - 1), kPastBytes);
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
    };
    if (warp < kConvWarps + 2) {
        // ---------------- MMA issue, a warp for each of the two weight tiles ----------------
        // (one warp for both issued a K block of 16 rows in 650 cycles: it gets a fifth of its scheduler's slots)
        const uint32_t mt = warp - kConvWarps;
        // The whole warp walks the loop on warp-uniform values and one elected lane issues: behind a branch on the lane
        // number every descriptor was a per-thread value, and all tiles ran at 0.7 us per K block (0.5 now at 16 columns).
        Tile t;
        uint32_t n = 0;
        bool go = take_tile(0, t), was_wide = false;
        const uint32_t acc = __shfl_sync(0xffffffffu, tmem_base, 0), sm0 = __shfl_sync(0xffffffffu, smem_base, 0);
        {
            uint32_t a_use = 0, b_use = 0, sa = 0, sb = 0;
            for (; go && !t.narrow; go = take_tile(++n, t)) {
                was_wide = true;
                t.count = __shfl_sync(0xffffffffu, t.count, 0);
                const uint32_t idesc = umma_idesc((t.count + 15u) & ~15u), n_kb = __shfl_sync(0xffffffffu, k_blocks(t), 0);
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
                        const uint64_t db = umma_smem_desc(sm0 + sb * kWideBBytes);
                        const uint64_t da = umma_smem_desc(sm0 + kWideOffA + sa * kWideABytes + mt * kTileBytes);
                        // 4 x K16 per 64-wide block: 32 bytes further along the row
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k) umma_f16(acc + mt * kUmmaMaxN, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                        umma_commit(&a_empty[sa]);
                        umma_commit(&b_empty[sb]);
                    }
                    __syncwarp();
                    if (++sa == kWideA) sa = 0;
                    if (++sb == kWideB) sb = 0;
                }
                if (elect_one()) umma_commit(&accum[n % kTiles]);
                __syncwarp();
            }
        }
        if (was_wide && go) {
            if (elect_one()) umma_commit(wide_over);
            __syncwarp();
        }
        uint32_t kc = 0, sb = 0, b_par = 0;
        bool other_small = true;   // the tile before had accumulators of its own
        for (uint32_t first = n; go; go = take_tile(++n, t)) {
            t.count = __shfl_sync(0xffffffffu, t.count, 0);   // (a value that the compiler knows to be uniform)
            const bool small = t.count <= kSmallN;
            const uint32_t idesc = umma_idesc((t.count + 15u) & ~15u), n_kb = __shfl_sync(0xffffffffu, k_blocks(t), 0);
            const uint32_t b_mask = narrow_b_mask(t.count), b_step = kNarrowBBytes / (b_mask + 1);
            const uint32_t acc_at = acc + (small ? (n & 1) * 2 * kSmallN + mt * kSmallN : mt * 128);
            // the last tiles' epilogues have read these accumulators (a wide tile's: before any narrow weights were converted)
            bool ok = n < first + 2 || pipe_wait(&epi_done[n & 1], ((n >> 1) & 1) ^ 1);
            if (n > first && !(small && other_small)) ok = ok && pipe_wait(&epi_done[(n & 1) ^ 1], ((n - 1) >> 1) & 1);
            if (!__all_sync(0xffffffffu, ok)) { give_up(); break; }
            other_small = small;
            for (uint32_t kb = 0; kb < n_kb; kb += 2, ++kc) {
                const uint32_t st = kc % kNarrowA, here = min(2u, n_kb - kb), in_b = kb & b_mask;   // K block within the activations' stage
                const uint32_t sb1 = b_mask ? sb : sb + 1 == kNarrowB ? 0u : sb + 1, in_b1 = b_mask ? in_b + 1 : 0u;   // the second one's
                bool got = in_b || pipe_wait(&nb_full[sb], b_par);
                if (!b_mask && here == 2) got = got && pipe_wait(&nb_full[sb1], sb1 ? b_par : b_par ^ 1);
                got = got && pipe_wait(&na_full[st], (kc / kNarrowA) & 1);
                if (!__all_sync(0xffffffffu, got)) {
                    give_up();
                    break;
                }
                const bool b_done = in_b1 == b_mask || kb + 2 >= n_kb;   // (of a stage for several K blocks)
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t ta = acc + 256u + st * 128 + mt * 32;   // 16 of K are eight columns
                    const uint64_t db = umma_smem_desc(sm0 + sb * kNarrowBBytes + in_b * b_step);
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k) umma_f16_ts(acc_at, ta + 8 * k, db + 2 * k, idesc, (kb | k) != 0);
                    if (!b_mask) umma_commit(&nb_empty[sb]);   // (its next copy need not wait for the other K block)
                    if (here == 2) {
                        const uint64_t db1 = umma_smem_desc(sm0 + sb1 * kNarrowBBytes + in_b1 * b_step);
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k) umma_f16_ts(acc_at, ta + 64 + 8 * k, db1 + 2 * k, idesc, 1u);
                    }
                    umma_commit(&na_empty[st]);
                    if (b_mask && b_done) umma_commit(&nb_empty[sb]);
                    if (!b_mask && here == 2) umma_commit(&nb_empty[sb1]);
                }
                __syncwarp();
                for (uint32_t i = b_mask ? (b_done ? 1u : 0u) : here; i; --i)
                    if (++sb == kNarrowB) { sb = 0; b_par ^= 1; }
            }
            if (elect_one()) umma_commit(&accum[n % kTiles]);
            __syncwarp();
        }
    } else if (warp == kConvWarps + 2) {
        // ---------------- activation tiles ----------------
        // One or two boxes per K block: these tiles are most of what a block pulls out of L2, and a short instance
        // does not pay for 256 rows, nor one of 80 rows for 128.
        uint32_t b_use = 0, sb = 0, nsb = 0, b_par = 0, ss = 0, sc_par = 0, sc_use = 0;
        bool was_wide = false, in_wide = true, waited = PHASE == 0;
        Tile t;
        for (uint32_t n = 0; take_tile(n, t); ++n) {
            const TileShape ts(t.count);
            const CUtensorMap* maps_b = t.shared ? maps.act_shared : maps.act_routed;
            const uint32_t KB = k_blocks(t), b_bytes = (ts.n1 + ts.n2) * 128u, y1 = PHASE == 0 ? t.r0 : t.r0 + 128;
            if (t.narrow && in_wide) {
                in_wide = false;
                if (was_wide && !wait(wide_over, 0)) give_up();
            }
            was_wide = in_wide;
            auto copy = [&](uint32_t dst, uint32_t kb, uint64_t* bar) {
                tma_load_2d(dst, &maps_b[ts.b1], (int32_t)(kb * 64), (int32_t)t.first, bar);
                if (ts.n2) tma_load_2d(dst + ts.n1 * 128u, &maps_b[ts.b2], (int32_t)(kb * 64), (int32_t)(t.first + ts.n1), bar);
            };
            const uint32_t b_mask = narrow_b_mask(t.count), b_step = kNarrowBBytes / (b_mask + 1);
            for (uint32_t kb = 0; t.narrow && kb < KB; kb += b_mask + 1) {
                if (any_failed()) break;
                if (!SCT && kb % (2 * kKbPerSc) == 0) {
                    if (!wait(&nsc_empty[ss], sc_par ^ 1)) { give_up(); break; }
                    copy_scales(std::integral_constant<uint32_t, 8>(), 1, t, kb * kGroupsPerBlock, y1, smem_base + kNarrowOffSc + ss * kNarrowScBytes,
                                smem_base + kOffPast + ss * 2 * kPastBytes, &nsc_full[ss]);
                    if (++ss == kNarrowSc) { ss = 0; sc_par ^= 1; }
                }
                if (!waited) { pdl_wait(); waited = true; }   // the scales are there before the gate/up launch ends
                if (!wait(&nb_empty[nsb], b_par ^ 1)) { give_up(); break; }
                if (lane == 0) {
                    const uint32_t here = min(b_mask + 1, KB - kb);
                    mbar_expect_tx(&nb_full[nsb], here * b_bytes);
                    for (uint32_t i = 0; i < here; ++i) copy(smem_base + nsb * kNarrowBBytes + i * b_step, kb + i, &nb_full[nsb]);
                }
                if (++nsb == kNarrowB) { nsb = 0; b_par ^= 1; }
            }
            for (uint32_t kb = 0; !t.narrow && kb < KB; ++kb) {
                if (any_failed()) break;
                if (!SCT && kb % kKbPerSc == 0) {
                    if (!wait(sc_empty, sc_use ^ 1)) { give_up(); break; }
                    sc_use ^= 1;
                    copy_scales(std::integral_constant<uint32_t, 4>(), 1, t, kb * kGroupsPerBlock, y1, smem_base + kWideOffSc, smem_base + kOffPast, sc_full);
                }
                if (!waited) { pdl_wait(); waited = true; }
                if (!wait(&b_empty[sb], ((b_use >> sb) & 1) ^ 1)) { give_up(); break; }
                b_use ^= 1u << sb;
                if (lane == 0) {
                    mbar_expect_tx(&b_full[sb], b_bytes);
                    copy(smem_base + sb * kWideBBytes, kb, &b_full[sb]);
                }
                if (++sb == kWideB) sb = 0;
            }
        }
        if (!waited) pdl_wait();   // (no tile here: the launch still ends after the one before)
    } else if (warp > kConvWarps + 3) {
        // ---------------- epilogues of small tiles ----------------
        // (by the converters between two tiles they took 3000 of a tile's 22,000 cycles at 2048 x 16 rows)
        const uint32_t et = tid - (kConvWarps + 4) * 32;
        uint32_t met = 0;
        Tile t;
        // A tile is handed back only when its instructions are done, also one that the converters finish: its barrier then is never
        // more than a phase away from the one that is waited for.
        for (uint32_t n = 0; take_tile(n, t, false); ++n) {
            if (t.count > kSmallN) {
                if (!pipe_wait(&accum[n % kTiles], (n / kTiles) & 1)) { give_up(); break; }
                release_tile(n);
                continue;
            }
            uint32_t* const ids = small_id + (n & 1) * kSmallN;
            float* const wts = small_w + (n & 1) * kSmallN;
            if (PHASE == 1) {
                if (et < t.count) {
                    const uint32_t p = t.shared ? t.first + et : __ldcg(a.sorted + t.first + et);
                    ids[et] = t.shared ? p : p / a.top_k;
                    wts[et] = t.shared ? (a.shared_gate ? __ldcg(a.shared_gate + p) : 1.0f) : __ldcg(a.route_w + p);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(eids_full);
                const bool ok = pipe_wait(eids_full, met);
                met ^= 1;
                if (!ok) { give_up(); break; }
            }
            const uint32_t at = (n & 1) * 2 * kSmallN;
            if (!epilogue(std::integral_constant<int, 4>(), std::integral_constant<int, 1>(), 0u, t, n, at, at + kSmallN, ids, wts)) break;
            release_tile(n);
        }
    } else {
        // ---------------- tiles; packed weights, scales, biases ----------------
        // The number of the tile after next and the instance of the next one are asked for while this one is copied.
        const uint32_t n_tiles = __ldcg(n_inst) * row_tiles;
        auto read_inst = [&](uint32_t tile) { return tile < n_tiles ? __ldcg((const uint4*)(inst + tile / row_tiles)) : make_uint4(0, 0, 0, 0); };
        auto number = [&]() { return lane == 0 ? gridDim.x + atomicAdd(n_inst + 1 + PHASE, 1u) : 0u; };   // (of lane 0)
        uint32_t now = blockIdx.x, next = number();
        uint4 v = read_inst(now);
        uint32_t n = 0, pk_use = 0, sc_use = 0, slot = 0, ss = 0, pk_par = 0, sc_par = 0;
        bool was_wide = false, in_wide = true;
        for (;;) {
            const bool end = now >= n_tiles;
            next = __shfl_sync(0xffffffffu, next, 0);
            const uint4 v_next = end ? v : read_inst(next);
            const uint32_t after = end ? 0u : number();
            Tile t;
            t.shared = v.x == 1;
            t.slot = v.y; t.first = v.z; t.count = end ? 0u : v.w;
            t.r0 = (now % row_tiles) * (PHASE == 0 ? 128u : 256u);
            t.narrow = t.count <= kNarrowN;
            const uint32_t rows = PHASE == 0 ? (t.shared ? a.f_shared : a.f) : a.d, KB = k_blocks(t);
            now = next; next = after; v = v_next;
            if (!end && t.r0 >= rows) continue;   // a narrower shared or routed expert
            const uint32_t s = n % kTiles;
            if (!wait(&tile_empty[s], ((n / kTiles) & 1) ^ 1)) { give_up(); break; }
            ++n;
            if (lane == 0) {
                next_tile[s] = make_uint4(t.slot, t.first, t.r0 | (t.shared ? 0x80000000u : 0u), t.count);
                mbar_arrive(&tile_full[s]);
            }
            if (end || any_failed()) break;
            const WeightMaps* wm = t.shared ? &maps.shared : &maps.routed[t.slot / a.pool.cells_per_chunk];
            const int32_t cell = t.shared ? 0 : (int32_t)(t.slot % a.pool.cells_per_chunk);
            const int32_t y0 = (int32_t)t.r0, y1 = (int32_t)(PHASE == 0 ? t.r0 : t.r0 + 128);
            if (!t.narrow) {
                was_wide = true;
                for (uint32_t kb = 0; kb < KB; ++kb) {
                    if (any_failed()) break;
                    if (kb % kKbPerSc == 0) {
                        const int32_t g0 = (int32_t)(kb / kKbPerSc * 8);
                        if (!wait(sc_empty, sc_use ^ 1)) { give_up(); break; }
                        sc_use ^= 1;
                        const uint32_t dst = smem_base + kWideOffSc;
                        if (!SCT) {
                            copy_scales(std::integral_constant<uint32_t, 4>(), 0, t, (uint32_t)g0, (uint32_t)y0, dst, smem_base + kOffPast, sc_full);
                        } else if (lane == 0) {
                            mbar_expect_tx(sc_full, kWideScBytes);
                            tma_load_3d(dst, &wm->s[0], g0, y0, cell, sc_full);
                            tma_load_3d(dst + kWideScBytes / 4, &wm->s[1], g0, y1, cell, sc_full);
                            tma_load_3d(dst + kWideScBytes / 2, &wm->b[0], g0, y0, cell, sc_full);
                            tma_load_3d(dst + kWideScBytes / 4 * 3, &wm->b[1], g0, y1, cell, sc_full);
                        }
                    }
                    if (kb % kWideKbPerPk == 0) {
                        const int32_t x = (int32_t)(kb / kWideKbPerPk * 64);
                        if (!wait(&pk_empty[slot], ((pk_use >> slot) & 1) ^ 1)) { give_up(); break; }
                        pk_use ^= 1u << slot;
                        if (lane == 0) {
                            mbar_expect_tx(&pk_full[slot], kWidePkBytes);
                            const uint32_t dst = smem_base + kWideOffPk + slot * kWidePkBytes;
                            tma_load_3d(dst, &wm->w[0], x, y0, cell, &pk_full[slot]);
                            tma_load_3d(dst + kWidePkBytes / 2, &wm->w[1], x, y1, cell, &pk_full[slot]);
                        }
                        if (++slot == kWidePk) slot = 0;
                    }
                }
                continue;
            }
            if (in_wide) {
                in_wide = false;
                slot = 0;
                if (was_wide && !wait(wide_over, 0)) { give_up(); break; }
            }
            for (uint32_t kb = 0; kb < KB; kb += kNarrowKbPerPk) {
                if (any_failed()) break;
                if (kb % (2 * kKbPerSc) == 0) {
                    const int32_t g0 = (int32_t)(kb / kKbPerSc * 8);
                    uint64_t* const bar = &nsc_full[ss];
                    if (!wait(&nsc_empty[ss], sc_par ^ 1)) { give_up(); break; }
                    const uint32_t dst = smem_base + kNarrowOffSc + ss * kNarrowScBytes;
                    if (!SCT) {
                        copy_scales(std::integral_constant<uint32_t, 8>(), 0, t, (uint32_t)g0, (uint32_t)y0, dst, smem_base + kOffPast + ss * 2 * kPastBytes, bar);
                    } else if (lane == 0) {
                        mbar_expect_tx(bar, kNarrowScBytes);
                        tma_load_3d(dst, &wm->ns[0], g0, y0, cell, bar);
                        tma_load_3d(dst + kNarrowScBytes / 4, &wm->ns[1], g0, y1, cell, bar);
                        tma_load_3d(dst + kNarrowScBytes / 2, &wm->nb[0], g0, y0, cell, bar);
                        tma_load_3d(dst + kNarrowScBytes / 4 * 3, &wm->nb[1], g0, y1, cell, bar);
                    }
                    if (++ss == kNarrowSc) { ss = 0; sc_par ^= 1; }
                }
                if (!wait(&npk_empty[slot], pk_par ^ 1)) { give_up(); break; }
                if (lane == 0) {
                    mbar_expect_tx(&npk_full[slot], kNarrowPkBytes);
                    const uint32_t dst = smem_base + kNarrowOffPk + slot * kNarrowPkBytes;
                    const int32_t x = (int32_t)(kb / kNarrowKbPerPk * 128);
                    tma_load_3d(dst, &wm->nw[0], x, y0, cell, &npk_full[slot]);
                    tma_load_3d(dst + kNarrowPkBytes / 2, &wm->nw[1], x, y1, cell, &npk_full[slot]);
                }
                if (++slot == kNarrowPk) { slot = 0; pk_par ^= 1; }
            }
        }
    }
    }
    if (failed() && lane == 0 && (warp & ~1u) == kConvWarps + 2) {
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

// One matrix of every cell of a pool chunk: [cells][rows][row_bytes] bytes (packed weights) or [cells][rows][groups] 16-bit
// (scales / biases), in boxes of 128 rows: of 64 bytes, swizzled so, or 8 groups, and twice that for narrow tiles.
static bool make_matrix_map(CUtensorMap* map, const uint8_t* base, bool meta, bool narrow, uint64_t row_elems, uint64_t rows,
                            uint64_t cells, uint64_t cell_stride) {
    const uint64_t esz = meta ? 2 : 1;
    const cuuint64_t dims[3] = {row_elems, rows, cells};
    // a single cell (the shared expert's block) still needs a valid outer pitch
    const cuuint64_t strides[2] = {row_elems * esz, cells > 1 ? cell_stride : row_elems * esz * rows};
    const cuuint32_t box[3] = {(meta ? 8u : 64u) << narrow, 128, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    return encode_tiled_fn()(map, meta ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, (void*)base,
                             dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             meta ? CU_TENSOR_MAP_SWIZZLE_NONE : narrow ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The two tiles of one phase: gate + up (phase 0) or down twice (phase 1: the same maps).
static bool make_weight_maps(WeightMaps* wm, const uint8_t* base, const Offsets3& off, int phase, uint32_t kdim,
                             uint32_t rows, uint32_t bits, uint32_t group, uint64_t cells, uint64_t cell_stride) {
    for (int t = 0; t < (phase == 0 ? 2 : 1); ++t) {
        const int mat = phase == 0 ? t : 2;
        if (!make_matrix_map(&wm->w[t], base + off.w[mat], false, false, (uint64_t)kdim * bits / 8, rows, cells, cell_stride) ||
            !make_matrix_map(&wm->nw[t], base + off.w[mat], false, true, (uint64_t)kdim * bits / 8, rows, cells, cell_stride))
            return false;
        if ((kdim / group) % 8 != 0) continue;   // such scale rows are copied word by word
        for (int n = 0; n < 2; ++n)
            if (!make_matrix_map(n ? &wm->ns[t] : &wm->s[t], base + off.s[mat], true, n, kdim / group, rows, cells, cell_stride) ||
                !make_matrix_map(n ? &wm->nb[t] : &wm->b[t], base + off.b[mat], true, n, kdim / group, rows, cells, cell_stride))
                return false;
    }
    if (phase == 1)
        for (CUtensorMap* both : {wm->w, wm->s, wm->b, wm->nw, wm->ns, wm->nb}) both[1] = both[0];
    return true;
}

// K in whole 64-wide blocks (packed rows are then whole 16-byte units, which the TMA copies need).
bool umma_supported(const shrike_moe_config& c) {
    if (c.d % 64 || c.f % 64) return false;
    if (c.has_shared && c.shared_f % 64) return false;
    return encode_tiled_fn() != nullptr;
}

// A handle's maps: of its activation operands, and of the pool and shared block of its last call with what they were made from.
struct UmmaMapCache {
    CUtensorMap act[4 * kActBoxes];   // operands xs, acts, xh, acts_shared; boxes of 16, 32, 64, 128, 256 rows
    UmmaMaps phase[2];
    PoolView pool;
    Offsets3 routed, shared;
    const uint8_t* shared_block;
    bool valid;
};

// Called once per handle, after the workspace exists: the activation operands' maps.
cudaError_t umma_prepare(shrike_moe* m) {
    const shrike_moe_config& c = m->cfg;
    Workspace& ws = m->ws;
    UmmaMapCache* const cache = (UmmaMapCache*)ws.tensor_maps;
    memset(cache, 0, sizeof *cache);
    if (!ws.xs || !umma_supported(c)) return cudaSuccess;
    CUtensorMap* am = cache->act;
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

// The converters' setmaxnreg.inc waits for registers that the block was launched with: a build with fewer would wait for good.
template <int BITS, int GROUP, int META, int PHASE, bool SCT>
static bool registers_fit() {
    static const bool fits = [] {
        cudaFuncAttributes at;
        return cudaFuncGetAttributes(&at, umma_expert_kernel<BITS, GROUP, META, PHASE, SCT>) == cudaSuccess &&
               (uint32_t)at.numRegs * kUmmaThreads >= kConverters * kConvRegs + (kUmmaThreads - kConverters) * kOtherRegs;
    }();
    return fits;
}

template <int BITS, int GROUP, int META>
static cudaError_t launch_umma_t(const shrike_moe* m, cudaStream_t st, const ExpertArgs& a, const ChunkInstance* inst,
                                 uint32_t* n_inst, uint32_t max_inst, const UmmaMaps& m0, const UmmaMaps& m1) {
    const bool sct0 = (a.d / GROUP & 7u) == 0, sct1 = ((a.f / GROUP | a.f_shared / GROUP) & 7u) == 0;
    auto k0 = sct0 ? umma_expert_kernel<BITS, GROUP, META, 0, true> : umma_expert_kernel<BITS, GROUP, META, 0, false>;
    auto k1 = sct1 ? umma_expert_kernel<BITS, GROUP, META, 1, true> : umma_expert_kernel<BITS, GROUP, META, 1, false>;
    if (!(sct0 ? registers_fit<BITS, GROUP, META, 0, true>() : registers_fit<BITS, GROUP, META, 0, false>()) ||
        !(sct1 ? registers_fit<BITS, GROUP, META, 1, true>() : registers_fit<BITS, GROUP, META, 1, false>()))
        return cudaErrorInvalidConfiguration;
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
size_t umma_tensor_map_bytes() { return (sizeof(UmmaMapCache) + 63) / 64 * 64; }

// The maps of a call's pool and shared block; NULL when one cannot be encoded. They change only when the host changes the pool, the
// offsets or the shared block: encoded on every call, a pool of eight chunks with a shared expert took 216 of them (36 us of host
// work a call of 65 rows, 33 before narrow tiles had boxes of their own; 23 with the maps kept).
static const UmmaMaps* umma_maps_for(const shrike_moe* m, const ExpertArgs& a) {
    const shrike_moe_config& c = m->cfg;
    UmmaMapCache* const cache = (UmmaMapCache*)m->ws.tensor_maps;
    if (cache->valid && memcmp(&cache->pool, &a.pool, sizeof(PoolView)) == 0 && memcmp(&cache->routed, &a.routed, sizeof(Offsets3)) == 0 &&
        memcmp(&cache->shared, &a.shared, sizeof(Offsets3)) == 0 && cache->shared_block == a.shared_block)
        return cache->phase;
    cache->valid = false;
    memset(cache->phase, 0, sizeof cache->phase);
    for (int phase = 0; phase < 2; ++phase) {
        UmmaMaps& mp = cache->phase[phase];
        const uint32_t kdim = phase == 0 ? c.d : c.f, rows = phase == 0 ? c.f : c.d;
        uint32_t left = a.pool.cells;
        for (uint32_t ch = 0; ch < SHRIKE_MAX_POOL_CHUNKS && a.pool.base[ch] && left; ++ch) {
            const uint32_t cells = left < a.pool.cells_per_chunk ? left : a.pool.cells_per_chunk;
            if (!make_weight_maps(&mp.routed[ch], a.pool.base[ch], a.routed, phase, kdim, rows, c.weight_bits,
                                  c.group_size, cells, a.pool.stride))
                return nullptr;
            left -= cells;
        }
        for (int bi = 0; bi < kActBoxes; ++bi) mp.act_routed[bi] = cache->act[phase * kActBoxes + bi];
        if (c.has_shared) {
            const uint32_t kds = phase == 0 ? c.d : c.shared_f, rws = phase == 0 ? c.shared_f : c.d;
            if (!make_weight_maps(&mp.shared, a.shared_block, a.shared, phase, kds, rws, c.weight_bits, c.group_size, 1,
                                  16))
                return nullptr;
            for (int bi = 0; bi < kActBoxes; ++bi) mp.act_shared[bi] = cache->act[(2 + phase) * kActBoxes + bi];
        } else {
            mp.shared = mp.routed[0];
            for (int bi = 0; bi < kActBoxes; ++bi) mp.act_shared[bi] = mp.act_routed[bi];
        }
    }
    cache->pool = a.pool; cache->routed = a.routed; cache->shared = a.shared; cache->shared_block = a.shared_block;
    cache->valid = true;
    return cache->phase;
}

// Gate/up + GLU, then down, for the instances that the prefill plan left in the workspace.
cudaError_t launch_umma_prefill(const shrike_moe* m, cudaStream_t st, const ExpertArgs& a, uint32_t T) {
    const shrike_moe_config& c = m->cfg;
    const Workspace& ws = m->ws;
    if (!ws.tensor_maps || !umma_supported(c)) return cudaErrorNotSupported;
    const UmmaMaps* const maps = umma_maps_for(m, a);
    if (!maps) return cudaErrorInvalidValue;
    const ChunkInstance* const inst = (const ChunkInstance*)ws.chunk_inst;
    const uint32_t max_inst = umma_max_chunk_instances(c, T);
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
