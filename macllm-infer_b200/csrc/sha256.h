// SHA-256 (FIPS 180-4), used by the exact-token prefix cache's chained block digests
// (the reference uses the sha2 crate, crates/macllm-kv/src/prefix_cache.rs:556-594).
#pragma once
#include <cstdint>
#include <cstddef>
#include <cstring>
#include <array>
#if defined(__x86_64__) && !defined(__CUDA_ARCH__)
#include <cpuid.h>
#include <immintrin.h>
#define MK_SHA256_EXTENSIONS 1
#endif

namespace mk {

class Sha256 {
public:
    Sha256() { reset(); }
    void reset() {
        static const uint32_t init[8] = {0x6a09e667u, 0xbb67ae85u, 0x3c6ef372u, 0xa54ff53au,
                                         0x510e527fu, 0x9b05688cu, 0x1f83d9abu, 0x5be0cd19u};
        memcpy(h_, init, sizeof init);
        len_ = 0;
        fill_ = 0;
    }
    void update(const void* data, size_t n) {
        const uint8_t* p = static_cast<const uint8_t*>(data);
        len_ += n;
        while (n > 0) {
            size_t take = 64 - fill_ < n ? 64 - fill_ : n;
            memcpy(buf_ + fill_, p, take);
            fill_ += take;
            p += take;
            n -= take;
            if (fill_ == 64) { block(buf_); fill_ = 0; }
        }
    }
    void update_u32le(uint32_t v) {
        uint8_t b[4] = {(uint8_t)v, (uint8_t)(v >> 8), (uint8_t)(v >> 16), (uint8_t)(v >> 24)};
        update(b, 4);
    }
    std::array<uint8_t, 32> finish() {
        uint64_t bits = len_ * 8;
        static const uint8_t pad[64] = {0x80};
        update(pad, fill_ < 56 ? 56 - fill_ : 120 - fill_);
        uint8_t lenb[8];
        for (int i = 0; i < 8; ++i) lenb[i] = (uint8_t)(bits >> (56 - 8 * i));
        update(lenb, 8);
        std::array<uint8_t, 32> out;
        for (int i = 0; i < 8; ++i) {
            out[4 * i] = (uint8_t)(h_[i] >> 24);
            out[4 * i + 1] = (uint8_t)(h_[i] >> 16);
            out[4 * i + 2] = (uint8_t)(h_[i] >> 8);
            out[4 * i + 3] = (uint8_t)h_[i];
        }
        return out;
    }

private:
    static uint32_t rotr(uint32_t x, int n) { return (x >> n) | (x << (32 - n)); }
    void block(const uint8_t* p) {
        alignas(16) static const uint32_t k[64] = {
            0x428a2f98u, 0x71374491u, 0xb5c0fbcfu, 0xe9b5dba5u, 0x3956c25bu, 0x59f111f1u, 0x923f82a4u, 0xab1c5ed5u,
            0xd807aa98u, 0x12835b01u, 0x243185beu, 0x550c7dc3u, 0x72be5d74u, 0x80deb1feu, 0x9bdc06a7u, 0xc19bf174u,
            0xe49b69c1u, 0xefbe4786u, 0x0fc19dc6u, 0x240ca1ccu, 0x2de92c6fu, 0x4a7484aau, 0x5cb0a9dcu, 0x76f988dau,
            0x983e5152u, 0xa831c66du, 0xb00327c8u, 0xbf597fc7u, 0xc6e00bf3u, 0xd5a79147u, 0x06ca6351u, 0x14292967u,
            0x27b70a85u, 0x2e1b2138u, 0x4d2c6dfcu, 0x53380d13u, 0x650a7354u, 0x766a0abbu, 0x81c2c92eu, 0x92722c85u,
            0xa2bfe8a1u, 0xa81a664bu, 0xc24b8b70u, 0xc76c51a3u, 0xd192e819u, 0xd6990624u, 0xf40e3585u, 0x106aa070u,
            0x19a4c116u, 0x1e376c08u, 0x2748774cu, 0x34b0bcb5u, 0x391c0cb3u, 0x4ed8aa4au, 0x5b9cca4fu, 0x682e6ff3u,
            0x748f82eeu, 0x78a5636fu, 0x84c87814u, 0x8cc70208u, 0x90befffau, 0xa4506cebu, 0xbef9a3f7u, 0xc67178f2u};
#ifdef MK_SHA256_EXTENSIONS
        // a 2200-token prompt is 137 chained blocks of three compressions: 130 us in plain code, 15 with the processor's instructions
        static const bool extensions = [] {
            unsigned a, b, c, d;
            return __get_cpuid_count(7, 0, &a, &b, &c, &d) != 0 && (b & (1u << 29)) != 0 && __get_cpuid(1, &a, &b, &c, &d) != 0 && (c & (1u << 19)) != 0;
        }();
        if (extensions) return compress(h_, p, k);
#endif
        uint32_t w[64];
        for (int i = 0; i < 16; ++i)
            w[i] = ((uint32_t)p[4 * i] << 24) | ((uint32_t)p[4 * i + 1] << 16) | ((uint32_t)p[4 * i + 2] << 8) | p[4 * i + 3];
        for (int i = 16; i < 64; ++i) {
            uint32_t s0 = rotr(w[i - 15], 7) ^ rotr(w[i - 15], 18) ^ (w[i - 15] >> 3);
            uint32_t s1 = rotr(w[i - 2], 17) ^ rotr(w[i - 2], 19) ^ (w[i - 2] >> 10);
            w[i] = w[i - 16] + s0 + w[i - 7] + s1;
        }
        uint32_t a = h_[0], b = h_[1], c = h_[2], d = h_[3], e = h_[4], f = h_[5], g = h_[6], h = h_[7];
        for (int i = 0; i < 64; ++i) {
            uint32_t S1 = rotr(e, 6) ^ rotr(e, 11) ^ rotr(e, 25);
            uint32_t ch = (e & f) ^ (~e & g);
            uint32_t t1 = h + S1 + ch + k[i] + w[i];
            uint32_t S0 = rotr(a, 2) ^ rotr(a, 13) ^ rotr(a, 22);
            uint32_t mj = (a & b) ^ (a & c) ^ (b & c);
            uint32_t t2 = S0 + mj;
            h = g; g = f; f = e; e = d + t1; d = c; c = b; b = a; a = t1 + t2;
        }
        h_[0] += a; h_[1] += b; h_[2] += c; h_[3] += d; h_[4] += e; h_[5] += f; h_[6] += g; h_[7] += h;
    }
#ifdef MK_SHA256_EXTENSIONS
    // The same rounds, four at a time, on the SHA instructions of x86: they keep the state as (a, b, e, f) and (c, d, g, h), highest lane first.
    __attribute__((target("sha,sse4.1,ssse3"))) static void compress(uint32_t* h, const uint8_t* p, const uint32_t* k) {
        const __m128i abcd = _mm_loadu_si128(reinterpret_cast<const __m128i*>(h)), efgh = _mm_loadu_si128(reinterpret_cast<const __m128i*>(h + 4));
        const __m128i badc = _mm_shuffle_epi32(abcd, 0xB1), hgfe = _mm_shuffle_epi32(efgh, 0x1B);
        const __m128i abef0 = _mm_alignr_epi8(badc, hgfe, 8), cdgh0 = _mm_blend_epi16(hgfe, badc, 0xF0);
        const __m128i big_endian = _mm_set_epi8(12, 13, 14, 15, 8, 9, 10, 11, 4, 5, 6, 7, 0, 1, 2, 3);
        __m128i abef = abef0, cdgh = cdgh0, w[4];
        for (int i = 0; i < 16; ++i) {
            __m128i& now = w[i & 3];
            if (i < 4) {
                now = _mm_shuffle_epi8(_mm_loadu_si128(reinterpret_cast<const __m128i*>(p + 16 * i)), big_endian);
            } else {
                const __m128i last = w[(i + 3) & 3];
                now = _mm_sha256msg2_epu32(_mm_add_epi32(_mm_sha256msg1_epu32(now, w[(i + 1) & 3]), _mm_alignr_epi8(last, w[(i + 2) & 3], 4)), last);
            }
            const __m128i wk = _mm_add_epi32(now, _mm_load_si128(reinterpret_cast<const __m128i*>(k + 4 * i)));
            cdgh = _mm_sha256rnds2_epu32(cdgh, abef, wk);
            abef = _mm_sha256rnds2_epu32(abef, cdgh, _mm_shuffle_epi32(wk, 0x0E));
        }
        abef = _mm_add_epi32(abef, abef0);
        cdgh = _mm_add_epi32(cdgh, cdgh0);
        const __m128i feba = _mm_shuffle_epi32(abef, 0x1B), dchg = _mm_shuffle_epi32(cdgh, 0xB1);
        _mm_storeu_si128(reinterpret_cast<__m128i*>(h), _mm_blend_epi16(feba, dchg, 0xF0));
        _mm_storeu_si128(reinterpret_cast<__m128i*>(h + 4), _mm_alignr_epi8(dchg, feba, 8));
    }
#endif
    uint32_t h_[8];
    uint64_t len_;
    uint8_t buf_[64];
    size_t fill_;
};

}  // namespace mk
