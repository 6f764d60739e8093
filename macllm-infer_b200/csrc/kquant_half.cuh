// Q4_K and Q6_K weights as f16, out of the packed bytes in registers: what the two matmuls that read the blocks in place share.
#pragma once
#include "common.cuh"

namespace mk {

// ---- Q4_K ------------------------------------------------------------------------------------------------------
// Half a row's 256-wide block: groups 4h .. 4h + 3 of 32 weights, whose scales and minima come out of `hdr` (d, dmin, the twelve scale bytes)
// four at a time.  Groups 2J and 2J + 1 of a block share the 32 bytes at 16 + 32 J, low nibbles / high nibbles.
// Four nibbles become (1024 + q) or, where they are, (1024 + 16 q) as f16 by byte permutation; a fma with the scale (a sixteenth of it) and -1024
// (-64) of it gives sc * q exactly (below 1024); then fma(sc * q, d, -dmin * m): the dequantised weight, rounded once.  The scales too stay
// in f16, where whole numbers below 64 and one product's rounding are what they are in f32.
struct Q4Half {
    uint32_t sc4, m4;
    __half2 d, nd;
    __device__ __forceinline__ Q4Half(const uint4& hdr, int h) {
        if (h == 0) {
            sc4 = hdr.y & 0x3F3F3F3Fu;
            m4 = hdr.z & 0x3F3F3F3Fu;
        } else {
            sc4 = (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
            m4 = ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
        }
        const uint32_t dd = __byte_perm(hdr.x, 0, 0x1010), nn = __byte_perm(hdr.x, 0, 0x3232) ^ 0x80008000u;
        d = *reinterpret_cast<const __half2*>(&dd);
        nd = *reinterpret_cast<const __half2*>(&nn);
    }
    // byte i of four as an f16 pair
    static __device__ __forceinline__ __half2 pair(uint32_t four, int i) {
        const uint32_t p = __byte_perm(four, 0x64646464u, 0x4040 + 0x0101 * i);
        return __hadd2(*reinterpret_cast<const __half2*>(&p), __float2half2_rn(-1024.f));
    }
    // group g (0 .. 3 of this half) out of its eight words
    template <int g>
    __device__ __forceinline__ void convert(const uint32_t (&words)[8], uint32_t (&out)[16]) const {
        constexpr bool HIGH = (g & 1) != 0;
        const __half2 sc = pair(sc4, g), nm = __hmul2(nd, pair(m4, g));
        const __half2 s = HIGH ? __hmul2(sc, __float2half2_rn(0.0625f)) : sc, nb = __hmul2(sc, __float2half2_rn(HIGH ? -64.f : -1024.f));
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t bytes = words[i] & (HIGH ? 0xF0F0F0F0u : 0x0F0F0F0Fu);
            const uint32_t p01 = __byte_perm(bytes, 0x64646464u, 0x4140), p23 = __byte_perm(bytes, 0x64646464u, 0x4342);
            const __half2 h01 = __hfma2(__hfma2(*reinterpret_cast<const __half2*>(&p01), s, nb), d, nm);
            const __half2 h23 = __hfma2(__hfma2(*reinterpret_cast<const __half2*>(&p23), s, nb), d, nm);
            out[2 * i] = *reinterpret_cast<const uint32_t*>(&h01);
            out[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&h23);
        }
    }
};
// The block's scales and minima, a byte each, groups 0 .. 7.
__device__ __forceinline__ void q4_scales(const uint4& hdr, uint32_t (&sc)[2], uint32_t (&m)[2]) {
    sc[0] = hdr.y & 0x3F3F3F3Fu;
    m[0] = hdr.z & 0x3F3F3F3Fu;
    sc[1] = (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
    m[1] = ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
}
// Bytes i and j of four as f16.
template <int i, int j>
__device__ __forceinline__ __half2 bytes_to_half2(uint32_t four) {
    const uint32_t p = __byte_perm(four, 0x64646464u, 0x4040 + i + 0x0100 * j);
    return __hadd2(*reinterpret_cast<const __half2*>(&p), __float2half2_rn(-1024.f));
}
// Sixteen weights of one group out of the low (HIGH: high) nibbles of four words, columns (0, 2) and (1, 3) of every word; the group's scale and minimum
// are bytes HIGH of sc4 and m4, nd is -dmin.  Nibbles at bits 0 and 16 turn into 1024 + q by one three-input operation, those at bits 4 and 20 into
// 1024 + 16 q; the arithmetic is Q4Half's.
template <int HIGH>
__device__ __forceinline__ void q4_weights(const uint32_t (&words)[4], uint32_t sc4, uint32_t m4, __half2 d, __half2 nd, uint32_t (&out)[8]) {
    constexpr uint32_t MASK = HIGH ? 0x00F000F0u : 0x000F000Fu;
    const __half2 sc = bytes_to_half2<HIGH, HIGH>(sc4), nm = __hmul2(nd, bytes_to_half2<HIGH, HIGH>(m4));
    const __half2 s = HIGH ? __hmul2(sc, __float2half2_rn(0.0625f)) : sc, nb = __hmul2(sc, __float2half2_rn(HIGH ? -64.f : -1024.f));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t p02 = (words[i] & MASK) | 0x64006400u, p13 = ((words[i] >> 8) & MASK) | 0x64006400u;
        const __half2 h02 = __hfma2(__hfma2(*reinterpret_cast<const __half2*>(&p02), s, nb), d, nm);
        const __half2 h13 = __hfma2(__hfma2(*reinterpret_cast<const __half2*>(&p13), s, nb), d, nm);
        out[2 * i] = *reinterpret_cast<const uint32_t*>(&h02);
        out[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&h13);
    }
}

// ---- Q6_K ------------------------------------------------------------------------------------------------------
// Four 6-bit values, a byte each, -> (q - 32) * s: (0, 1) and (2, 3), or (0, 2) and (1, 3).
template <bool EVEN_ODD = false>
__device__ __forceinline__ void q6_to_weights(uint32_t q, __half2 s, uint32_t& o01, uint32_t& o23) {
    uint32_t p01 = __byte_perm(q, 0x64646464u, EVEN_ODD ? 0x4240 : 0x4140);
    uint32_t p23 = __byte_perm(q, 0x64646464u, EVEN_ODD ? 0x4341 : 0x4342);
    const __half2 bias = __float2half2_rn(-1056.f);  // 1024 + q - 1056 = q - 32, exact
    __half2 h01 = __hmul2(__hadd2(*reinterpret_cast<__half2*>(&p01), bias), s);
    __half2 h23 = __hmul2(__hadd2(*reinterpret_cast<__half2*>(&p23), bias), s);
    o01 = *reinterpret_cast<uint32_t*>(&h01);
    o23 = *reinterpret_cast<uint32_t*>(&h23);
}

// The streamed copy of a matrix: (128-row tile, 256-column block) units one after the other.  A Q4_K unit is 128 raw blocks of 144 bytes.  A Q6_K
// unit: ql plane [128 rows][128 B], qh plane [128][64 B], scales plane [128][16 B], d [128] f16; the 16-byte chunks of a row of the ql and qh
// planes are stored at chunk ^ (row & 7) / chunk ^ (row & 3) so that 32 rows read at once fall into different banks.
constexpr int kUnitRows = 128;
constexpr int kQ4Unit = kUnitRows * 144;                    // 18432
constexpr int kQ6Unit = kUnitRows * (128 + 64 + 16) + 256;  // 26880
constexpr int kQ6Qh = kUnitRows * 128, kQ6Sc = kQ6Qh + kUnitRows * 64, kQ6D = kQ6Sc + kUnitRows * 16;

}  // namespace mk
