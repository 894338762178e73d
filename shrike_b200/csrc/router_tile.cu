// Router logits of many rows (prefill_router_tiled_body, prefill.metal:446-563): register tiles.
//
// Dozens of activation rows against the same router matrix. A warp that owns one expert row (router.cu) reads every
// activation row again for every expert row and waits for those reads. Here a block owns 8 WR expert rows x 16 WT tokens, both
// operands go to shared memory as they are (cp.async, three stages of 256 columns deep), and a warp accumulates an 8 x 16 register
// tile. Lane l still owns the elements of a row that router_math.cuh gives it and walks them in order, and the 32 lane sums still meet in
// the xor 16..1 butterfly: each logit is the same sequence of roundings as in the warp-per-row kernels. Two tokens share an
// instruction (f32x2: each half rounds as ever). Columns past the end of a row are staged as zeros: adding +0 changes nothing.
//
// What bounds it: fp32 rows, the fused multiply-adds (a lane's slice of K is its own, so a block cannot hold more than 32 x 32 sums
// and reads 393 MB out of L2 for 4096 rows of 256 x 2048); affine rows, five packed instructions per pair of columns and two tokens.
#include "route_args.cuh"
#include "router_math.cuh"
#include "select.cuh"

namespace shrike {

namespace {

constexpr uint32_t kK = 256;                           // columns of a stage
constexpr uint32_t kBufs = 3;

// A warp's tile is RW x TW, a block has WR x WT warps.
template <int BITS, int DT, int RW, int TW, int WR, int WT>
struct TileGeom {
    static constexpr uint32_t kWarpRows = RW, kWarpTokens = TW;
    static constexpr uint32_t kRows = kWarpRows * WR, kTokens = kWarpTokens * WT, kThreads = WR * WT * 32;
    static constexpr uint32_t kWRow = BITS == 0 ? kK * 4 : kK * BITS / 8;      // bytes of a row's stage
    static constexpr uint32_t kXRow = DT == SHRIKE_DTYPE_FP32 ? kK * 4 : kK * 2;
    static constexpr uint32_t kGates = BITS == 0 && DT != SHRIKE_DTYPE_FP32 ? 4 : 1;   // blocks of the gate row, rows of one stage
    static constexpr uint32_t kW = kRows * kWRow, kBuf = kW + kTokens * kXRow;
    static constexpr uint32_t kSb = BITS ? kRows * (kRouterMaxChunks * 2) * 8 : 0;   // {scale, bias} of the block's rows, fp32
    static constexpr uint32_t kSmem = kBufs * kBuf + kSb;
};

__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}

// N neighbouring activations from shared memory, widened.
template <int DT, int N>
__device__ __forceinline__ void load_x(const uint8_t* at, float (&x)[N]) {
    static_assert(N == 2 || N == 4, "elements");
    if constexpr (DT == SHRIKE_DTYPE_FP32) {
        if constexpr (N == 4) {
            const float4 v = *(const float4*)at;
            x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
        } else {
            const float2 v = *(const float2*)at;
            x[0] = v.x; x[1] = v.y;
        }
    } else {
        uint32_t q[N / 2];
        if constexpr (N == 4) {
            const uint2 v = *(const uint2*)at;
            q[0] = v.x; q[1] = v.y;
        } else {
            q[0] = *(const uint32_t*)at;
        }
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            if constexpr (DT == SHRIKE_DTYPE_FP16) {
                x[2 * i] = f16_bits_to_f32(q[i] & 0xffff);
                x[2 * i + 1] = f16_bits_to_f32(q[i] >> 16);
            } else {
                x[2 * i] = __uint_as_float(q[i] << 16);
                x[2 * i + 1] = __uint_as_float(q[i] & 0xffff0000u);
            }
        }
    }
}

// The lane sums of a warp's tile, [token][row], meet in the xor 16..1 order of butterfly_sum, each lane keeping half of the
// values at every step (8 x 16: 124 exchanges instead of 640; an addition does not care which side it is on). Of V values lane l
// ends with V / 32, from V / 32 * l on.
template <uint32_t RW, uint32_t TW>
__device__ __forceinline__ void store_tile(const RouterArgs& a, float (&v)[TW * RW], uint32_t e, uint32_t tok, uint32_t lane) {
    constexpr uint32_t N = TW * RW / 32;
    static_assert(N >= 1 && N * 32 == TW * RW && RW % N == 0, "a lane's values are of one token");
#pragma unroll
    for (uint32_t m = 16; m >= 1; m >>= 1) {
        const bool up = (lane & m) != 0;
#pragma unroll
        for (uint32_t i = 0; i < N * m; ++i) {
            const float keep = up ? v[i + N * m] : v[i], send = up ? v[i] : v[i + N * m];
            v[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, m));
        }
    }
    tok += lane * N / RW;
    e += lane * N % RW;
    if (tok >= a.T) return;
    float* const dst = a.logits + (size_t)tok * a.ne + e;
    if (N == 4 && e + 4 <= a.ne && (a.ne & 3u) == 0) {
        *(float4*)dst = make_float4(v[0], v[N > 1 ? 1 : 0], v[N > 2 ? 2 : 0], v[N > 3 ? 3 : 0]);
    } else {
#pragma unroll
        for (uint32_t i = 0; i < N; ++i)
            if (e + i < a.ne) dst[i] = v[i];
    }
}

}  // namespace

// grid (row tiles, and one or more for the gate row, token tiles)
template <int BITS, int DT, int RW, int TW, int WR, int WT>
__global__ void __launch_bounds__(WR * WT * 32, RW * TW == 128 ? 8 / (WR * WT) : 1) router_tile_kernel(const RouterArgs a) {
    using G = TileGeom<BITS, DT, RW, TW, WR, WT>;
    constexpr uint32_t kWarpRows = RW, kWarpTokens = TW;
    constexpr uint32_t kXB = DT == SHRIKE_DTYPE_FP32 ? 4 : 2;
    pdl_wait();
    pdl_launch_dependents();
    extern __shared__ __align__(16) uint8_t tile_smem[];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t e0 = blockIdx.x * G::kRows, t0 = blockIdx.y * G::kTokens;
    if (e0 >= a.ne) {
        // The shared expert's scalar gate: a warp per token at a time, the gate row in registers. (As a kernel of its own it took
        // 9 us of 4096 rows.)
        const uint32_t chunks = a.d / 4;
        float4 wr[kRouterMaxChunks];
        load_row_f32<kRouterMaxChunks, true>(a.gate_row, chunks, lane, wr);
        uint32_t first = t0, share = G::kTokens;
        if (G::kGates > 1 && a.d <= kK) {
            share /= G::kGates;
            first += (blockIdx.x - (a.ne + G::kRows - 1) / G::kRows) * share;
        }
        for (uint32_t tk = first + warp; tk < min(a.T, first + share); tk += WR * WT) {
            const void* xrow = (const uint8_t*)a.hidden + (size_t)tk * a.stride * kXB;
            const float acc = butterfly_sum(lane_dot_f32<kRouterMaxChunks, true>(wr, chunks, lane, xrow, DT, nullptr));
            if (lane == 0) a.gate_out[tk] = sigmoid_det(acc);
        }
        return;
    }
    const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(tile_smem);
    const uint32_t stages = (a.d + kK - 1) / kK, groups = a.d / 64;
    const uint32_t w_row = BITS == 0 ? a.d * 4 : a.d * BITS / 8, x_row = a.d * kXB;   // bytes

    // Consecutive threads copy consecutive 16-byte units of a row: free of bank conflicts.
    auto fetch = [&](uint32_t s, uint32_t buf) {
        constexpr uint32_t kWU = G::kWRow / 16, kXU = G::kXRow / 16, kWN = G::kRows * kWU, kXN = G::kTokens * kXU;
        const uint32_t to = smem0 + buf * G::kBuf;
#pragma unroll
        for (uint32_t j = 0; j < (kWN + G::kThreads - 1) / G::kThreads; ++j) {
            const uint32_t i = j * G::kThreads + tid, row = i / kWU, u = i % kWU, at = s * G::kWRow + u * 16;
            if (kWN % G::kThreads && i >= kWN) break;
            const uint8_t* src = (const uint8_t*)a.w + (size_t)min(e0 + row, a.ne - 1) * w_row;
            const uint32_t n = at < w_row ? 16u : 0u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + i * 16), "l"(src + (n ? at : 0u)), "r"(n) : "memory");
        }
#pragma unroll
        for (uint32_t j = 0; j < (kXN + G::kThreads - 1) / G::kThreads; ++j) {
            const uint32_t i = j * G::kThreads + tid, row = i / kXU, u = i % kXU, at = s * G::kXRow + u * 16;
            if (kXN % G::kThreads && i >= kXN) break;
            const uint8_t* src = (const uint8_t*)a.hidden + (size_t)min(t0 + row, a.T - 1) * a.stride * kXB;
            const uint32_t n = at < x_row ? 16u : 0u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + G::kW + i * 16), "l"(src + (n ? at : 0u)), "r"(n) : "memory");
        }
        cp_async_commit();
    };

    fetch(0, 0);
    if (stages > 1) fetch(1, 1);
    float2* const sb = (float2*)(tile_smem + kBufs * G::kBuf);
    if constexpr (BITS != 0)
        for (uint32_t j = tid; j < G::kRows * groups; j += G::kThreads) {
            const uint32_t row = j / groups;
            const size_t at = (size_t)min(e0 + row, a.ne - 1) * groups + (j - row * groups);
            sb[j] = make_float2(bf16_bits_to_f32(a.scales[at]), bf16_bits_to_f32(a.biases[at]));
        }

    uint64_t acc[kWarpRows][kWarpTokens / 2];
#pragma unroll
    for (uint32_t r = 0; r < kWarpRows; ++r)
#pragma unroll
        for (uint32_t t = 0; t < kWarpTokens / 2; ++t) acc[r][t] = 0;
    const uint32_t rg = warp % WR, tg = warp / WR;

    for (uint32_t s = 0; s < stages; ++s) {
        const uint32_t buf = s % kBufs;
        if (s + 1 < stages) cp_async_wait<1>();
        else cp_async_wait<0>();
        __syncthreads();   // stage s has landed for every thread, and every warp is done with stage s - 1
        if (s + 2 < stages) fetch(s + 2, (s + 2) % kBufs);
        const uint8_t* const wb = tile_smem + buf * G::kBuf + rg * kWarpRows * G::kWRow;
        const uint8_t* const xb = tile_smem + buf * G::kBuf + G::kW + tg * kWarpTokens * G::kXRow;
        if constexpr (BITS == 0) {
#pragma unroll
            for (uint32_t ii = 0; ii < kK / 128; ++ii) {   // lane l: float4 chunk l of every 32
                const uint32_t c = ii * 32 + lane;
                uint64_t wv[kWarpRows][4];
#pragma unroll
                for (uint32_t r = 0; r < kWarpRows; ++r) {
                    const float4 v = *(const float4*)(wb + r * G::kWRow + c * 16);
                    wv[r][0] = pack2(v.x, v.x); wv[r][1] = pack2(v.y, v.y); wv[r][2] = pack2(v.z, v.z); wv[r][3] = pack2(v.w, v.w);
                }
                uint2 es = make_uint2(0u, 0u);
                if (a.eff_scale && s * (kK / 4) + c < a.d / 4) es = __ldg((const uint2*)a.eff_scale + s * (kK / 4) + c);
#pragma unroll
                for (uint32_t t = 0; t < kWarpTokens / 2; ++t) {
                    float x[2][4];
#pragma unroll
                    for (uint32_t u = 0; u < 2; ++u) load_x<DT>(xb + (2 * t + u) * G::kXRow + c * 4 * kXB, x[u]);
                    if (a.eff_scale) {
#pragma unroll
                        for (uint32_t u = 0; u < 2; ++u) {
                            x[u][0] = __fmul_rn(x[u][0], __uint_as_float(es.x << 16));
                            x[u][1] = __fmul_rn(x[u][1], __uint_as_float(es.x & 0xffff0000u));
                            x[u][2] = __fmul_rn(x[u][2], __uint_as_float(es.y << 16));
                            x[u][3] = __fmul_rn(x[u][3], __uint_as_float(es.y & 0xffff0000u));
                        }
                    }
#pragma unroll
                    for (uint32_t i = 0; i < 4; ++i) {
                        const uint64_t xv = pack2(x[0][i], x[1][i]);
#pragma unroll
                        for (uint32_t r = 0; r < kWarpRows; ++r) acc[r][t] = fma2(wv[r][i], xv, acc[r][t]);
                    }
                }
            }
        } else {
#pragma unroll 1
            for (uint32_t gi = 0; gi < kK / 64; ++gi) {    // lane l: elements 2l, 2l + 1 of every group of 64
                const uint32_t group = s * (kK / 64) + gi;
                if (group >= groups) break;
                uint32_t es = 0;
                if (a.eff_scale) es = __ldg((const uint32_t*)a.eff_scale + group * 32 + lane);
                uint64_t x0[kWarpTokens / 2], x1[kWarpTokens / 2], sum[kWarpTokens / 2];
#pragma unroll
                for (uint32_t t = 0; t < kWarpTokens / 2; ++t) {
                    float x[2][2];
#pragma unroll
                    for (uint32_t u = 0; u < 2; ++u) {
                        load_x<DT>(xb + (2 * t + u) * G::kXRow + (gi * 64 + 2 * lane) * kXB, x[u]);
                        if (a.eff_scale) {
                            x[u][0] = __fmul_rn(x[u][0], __uint_as_float(es << 16));
                            x[u][1] = __fmul_rn(x[u][1], __uint_as_float(es & 0xffff0000u));
                        }
                    }
                    x0[t] = pack2(x[0][0], x[1][0]);
                    x1[t] = pack2(x[0][1], x[1][1]);
                    sum[t] = add2(x0[t], x1[t]);
                }
#pragma unroll
                for (uint32_t r = 0; r < kWarpRows; ++r) {
                    uint32_t q0, q1;
                    if constexpr (BITS == 4) {
                        const uint32_t q = *(wb + r * G::kWRow + gi * 32 + lane);
                        q0 = q & 0xfu;
                        q1 = q >> 4;
                    } else {
                        const uint32_t q = *(const uint16_t*)(wb + r * G::kWRow + gi * 64 + 2 * lane);
                        q0 = q & 0xffu;
                        q1 = q >> 8;
                    }
                    // 2^23 + q, less 2^23: exact, and no conversion instruction
                    const float f0 = __fsub_rn(__uint_as_float(0x4b000000u | q0), 8388608.0f), f1 = __fsub_rn(__uint_as_float(0x4b000000u | q1), 8388608.0f);
                    const float2 m = sb[(rg * kWarpRows + r) * groups + group];
                    const uint64_t w0 = pack2(f0, f0), w1 = pack2(f1, f1), sc = pack2(m.x, m.x), bi = pack2(m.y, m.y);
#pragma unroll
                    for (uint32_t t = 0; t < kWarpTokens / 2; ++t) {
                        acc[r][t] = fma2(sc, add2(mul2(w0, x0[t]), mul2(w1, x1[t])), acc[r][t]);
                        acc[r][t] = fma2(bi, sum[t], acc[r][t]);
                    }
                }
            }
        }
    }

    float sums[kWarpTokens * kWarpRows];
#pragma unroll
    for (uint32_t t = 0; t < kWarpTokens / 2; ++t)
#pragma unroll
        for (uint32_t r = 0; r < kWarpRows; ++r)
            asm("mov.b64 {%0, %1}, %2;" : "=f"(sums[2 * t * kWarpRows + r]), "=f"(sums[(2 * t + 1) * kWarpRows + r]) : "l"(acc[r][t]));
    store_tile<RW, TW>(a, sums, e0 + rg * kWarpRows, t0 + tg * kWarpTokens, lane);
}

namespace {

template <int BITS, int DT, int RW, int TW, int WR, int WT>
cudaError_t launch_tile(const shrike_moe* m, cudaStream_t st, const RouterArgs& a) {
    using G = TileGeom<BITS, DT, RW, TW, WR, WT>;
    static_assert(G::kSmem <= 227 * 1024, "shared memory of a block");
    auto k = router_tile_kernel<BITS, DT, RW, TW, WR, WT>;
    const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::kSmem);
    if (e != cudaSuccess) return e;
    // Blocks of the gate row for a token tile: of rows of one stage a call waits for the block whose warps have eight tokens each (256
    // experts of 256 columns, 512 rows: 10.7 us, with four blocks 8.8; 64 rows 5.9, 4.9; 4096 rows 31.9, 29.8). Longer rows, and those whose
    // tiles take longer, do not wait for it, and four cost them up to a fifth (int8 rows of 256 columns, fp32 activations, 512 rows 10.2, 12.2;
    // 2048 columns, bf16, 20.5, 22.5).
    const uint32_t gates = !a.gate_row ? 0u : a.d <= kK ? G::kGates : 1u;
    return launch_after(m, st, k, dim3((a.ne + G::kRows - 1) / G::kRows + gates, (a.T + G::kTokens - 1) / G::kTokens), G::kThreads,
                        G::kSmem, a);
}

// The tile by the logits of the call: small ones while a warp's way through a row is what a call waits for (its K is serial), large
// ones when the reads of shared memory and L2 per logit are. The whole router of 256 experts of 2048 columns, us, bf16 / fp32 activations; 4 x 8
// by a warp, 8 x 8, 8 x 16 in blocks of 16 x 32 (64 accumulators of two tokens: fp32 activations then wait for shared memory)
// and of 32 x 32. fp32 rows: 200 rows 14.0 / 18.6, 14.4 / 17.5, 15.4 / 21.1, 19.6 / 26.6; 512 rows 24.0 / 34.3, 23.7 / 30.0,
// 21.7 / 38.0, 23.9 / 30.8; 1134 rows 44.0 / 63.0, 44.6 / 58.8, 41.5 / 74.1, 43.4 / 56.9; 4096 rows - , - , 117 / 239, 128 / 176. int8 rows: 200
// rows 20.9 / 26.5, 24.0 / 22.9, 25.3 / 27.3, 35.4 / 38.6; 512 rows 41.2 / 50.2, 43.3 / 41.8, 38.7 / 48.8, 39.3 / 42.4; 1134
// rows 83.5 / 100, 80.4 / 76.0, 77.2 / 98.1, 74.2 / 80.2; 4096 rows - , - , 236 / 323, 237 / 258.
template <int BITS, int DT>
cudaError_t launch_sized(const shrike_moe* m, cudaStream_t st, const RouterArgs& a) {
    const uint64_t logits = (uint64_t)a.ne * a.T;
    if (logits <= 96u * 1024u) return launch_tile<BITS, DT, 4, 8, 2, 2>(m, st, a);
    if constexpr (DT == SHRIKE_DTYPE_FP32) {
        if (logits <= 256u * 1024u) return launch_tile<BITS, DT, 8, 8, 2, 2>(m, st, a);
        return launch_tile<BITS, DT, 8, 16, 4, 2>(m, st, a);
    } else {
        return launch_tile<BITS, DT, 8, 16, 2, 2>(m, st, a);
    }
}

template <int BITS>
cudaError_t launch_typed(const shrike_moe* m, cudaStream_t st, const RouterArgs& a) {
    if (a.dt == SHRIKE_DTYPE_FP32) return launch_sized<BITS, SHRIKE_DTYPE_FP32>(m, st, a);
    if (a.dt == SHRIKE_DTYPE_FP16) return launch_sized<BITS, SHRIKE_DTYPE_FP16>(m, st, a);
    return launch_sized<BITS, SHRIKE_DTYPE_BF16>(m, st, a);
}

}  // namespace

// Rows are copied 16 bytes at a time.
bool router_tiles_take(const RouterArgs& a) {
    const uint32_t esz = a.dt == SHRIKE_DTYPE_FP32 ? 4 : 2, w_row = a.bits ? a.d * a.bits / 8 : a.d * 4;
    return (a.d * esz) % 16 == 0 && ((size_t)a.stride * esz) % 16 == 0 && w_row % 16 == 0 && (a.bits == 0 || a.d % 64 == 0) &&
           a.d <= (uint32_t)kRouterMaxChunks * 128 && (((uintptr_t)a.hidden | (uintptr_t)a.w) & 15u) == 0;
}

cudaError_t launch_router_tiles(const shrike_moe* m, cudaStream_t st, const RouterArgs& a) {
    if (a.bits == 0) return launch_typed<0>(m, st, a);
    if (a.bits == 4) return launch_typed<4>(m, st, a);
    return launch_typed<8>(m, st, a);
}

}  // namespace shrike
