// Packed weight words in shared memory -> operand registers of the skinny tensor-core tiles (mma.sync m16n8k16),
// shared by the kernels that stream whole weight tiles.
#pragma once

#include "internal.h"

namespace shrike {

template <int BITS, int GROUP>
struct FQ {
    static constexpr int kWords = GROUP * BITS / 128;   // u32 per thread, row and group
    static constexpr int kMmas = GROUP / 16;
    static constexpr int kBRegs = GROUP / 8;
    static constexpr uint32_t kGroupBytes = GROUP * BITS / 8;
    // what the tiles multiply is offset + q: 1024 + q for nibbles in bits 0..3 (and for bytes), 64 + q for
    // nibbles in bits 4..7 (the fp16 value 64 has its unit in the last place at bit 4): no shift to unpack
    static constexpr float kOffEven = 1024.0f;
    static constexpr float kOffOdd = BITS == 4 ? 64.0f : 1024.0f;
};

template <int BITS>
__device__ __forceinline__ void unpack2(const uint32_t* w, int m, uint32_t& lo, uint32_t& hi) {
    if constexpr (BITS == 4) {
        const uint32_t v = w[m >> 1] >> ((m & 1) * 8);
        lo = lop3_and_or(v, 0x000F000Fu, 0x64006400u);   // (1024 + n0, 1024 + n4)
        hi = lop3_and_or(v, 0x00F000F0u, 0x54005400u);   // (64 + n1, 64 + n5)
    } else {
        const uint32_t v = w[m];
        lo = prmt(v, 0x64646464u, 0x5140u);
        hi = prmt(v, 0x64646464u, 0x5342u);
    }
}

template <int W>
__device__ __forceinline__ void lds_words(const uint8_t* p, uint32_t (&w)[W]) {
    if constexpr (W == 1) {
        w[0] = *(const uint32_t*)p;
    } else if constexpr (W == 2) {
        const uint2 v = *(const uint2*)p;
        w[0] = v.x; w[1] = v.y;
    } else {
        const uint4 v = *(const uint4*)p;
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    }
}

}  // namespace shrike
