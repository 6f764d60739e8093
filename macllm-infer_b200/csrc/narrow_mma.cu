// Matmul of the narrowest ticks, y[t][n] = sum_k x[t][k] W[n][k] for up to 16 rows (8 of Q4_K / Q6_K weights): a few lanes decoding.
//
// At this width a matmul is bound by what stands around its weight stream: the tcgen05 kernels hand every tile from a loader to (converters to) an
// issuer to an epilogue, and a 2048 x 2048 matrix at one row spends more on those hand-overs than on its 2 - 8 MB.  Here nothing is handed over.  A
// warp copies its own weights into a ring, turns them into A fragments of mma.sync.m16n8k16 in registers and adds up; warps meet once per row tile, to
// add their K slices.  The tensor rate of mma.sync does not count: 16 rows x 16 columns of weights take one or two instructions, against some 20 to
// unpack Q4_K.
//
// K is permuted so that every operand is read in runs of 16 bytes: lane (g, t) of a warp supplies rows g and g + 8 of A and row g (token) of B, and
// which four columns it calls its k = 2t, 2t+1, 2t+8, 2t+9 does not matter as long as A and B agree.  For an image they are neighbours of a 16-byte run;
// for Q4_K / Q6_K a lane's 16 bytes of nibbles are 16 columns of one group (low) and 16 of another (high), and the activations are put into
// shared memory in that order, 16 bytes per lane, once per CTA.
//
// The weights depend on no predecessor, so a CTA fills its ring before it waits for one; with 8 warps and at most half an SM's shared memory, the next
// matmul's CTAs do that while this one's compute.  Shares of K over CTAs (partial sums that the consumer adds in order) are used
// where there are fewer row tiles than SMs need, or where the activations would not fit.
#include "narrow_mma.h"
#include "kernels.h"
#include "kquant_half.cuh"
#include "narrow_ring.h"
#include <cuda_bf16.h>

namespace mk {

namespace {

constexpr int NM_WARPS = 8;
constexpr int NM_THREADS = NM_WARPS * 32;
constexpr uint32_t NM_SPIN_LIMIT = 1u << 22;
constexpr int NM_RED_PITCH = 20;                 // floats between the tokens of a 16-row tile's sums: lanes of a fragment hit all banks

// A step is what a warp copies and multiplies at a time: 16 rows x 64 columns of an image, or 16 rows of a 256-wide block.
constexpr int nm_step_cols(bool blocks) { return blocks ? 256 : 64; }
constexpr int NM_IMAGE_STEP = 16 * 64 * 2;                    // [chunk][lane][16 bytes]
constexpr int NM_Q4_STEP = 16 * 144;                          // raw blocks
constexpr int NM_Q6_STEP = 16 * (128 + 64 + 16) + 32;         // ql, qh, scales, d of 16 rows
constexpr int NM_IMAGE_STAGES = 6, NM_Q4_STAGES = 4, NM_Q6_STAGES = 3;

struct NmParams {
    int T, rows, cols;
    int n_steps;                   // of the whole K
    int shares, per_share_ctas;
    int groups;                    // row groups of RG tiles
    int rg_shift;                  // RG = 1 << rg_shift
    int tiles_first;               // 16-row tiles of the first matrix
    int q6, q6_2, stage_bytes, n_stages;
    int share_cols;                // most columns of a share: rows of X in shared memory are this wide
    const uint8_t *w, *w2;
    const __half* x;
    int n_inputs, input_tiles, input_end[kMaxRowGroups];
    float* y;
    int ldy;
    float out_scale, softcap;
    float* partial;
    int32_t* status;
    int gated;                     // 0 off, otherwise 1 + GatedAct::Kind
    float act_limit;
    const float *act_pre, *act_post;
    __half* yh;
    int ldyh, yh_bf16;
    int scattered;
    MatmulScatter scatter;
};

__device__ __forceinline__ uint32_t nm_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void nm_copy16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void nm_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void nm_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint4 nm_lds(const uint8_t* p) { return *reinterpret_cast<const uint4*>(p); }
template <bool BF16>
__device__ __forceinline__ void nm_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (BF16)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void nm_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void nm_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ bool nm_wait_full(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i <= NM_SPIN_LIMIT; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// NT tiles of 8 tokens.
template <NarrowFormat FORMAT, int NT>
__global__ void __launch_bounds__(NM_THREADS, 2)
narrow_mma_kernel(const __grid_constant__ NmParams p) {
    constexpr bool BLOCKS = FORMAT == NarrowFormat::Blocks, BF16 = FORMAT == NarrowFormat::BF16;
    constexpr int COLS = BLOCKS ? 256 : 64;
    constexpr int CHAINS = NT == 1 ? 4 : 2;   // sums side by side: an mma waits for the one before it on the same sum
    extern __shared__ __align__(128) uint8_t nm_shared[];
    __shared__ uint64_t full[BLOCKS ? NM_WARPS : 1][BLOCKS ? NM_Q4_STAGES : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int rg_shift = p.rg_shift, KW = NM_WARPS >> rg_shift, kw = warp & (KW - 1), sub_tile = warp / KW;
    // rows of a tile that this lane's fragments stand for: r and r + 8.  Raw blocks lie 144 bytes apart: rows 4 apart for neighbouring g hit all banks.
    const int r = BLOCKS ? (g >> 1) + 4 * (g & 1) : g;
    const int pitch = p.share_cols * 2 + 64;                     // bytes between tokens: 64 modulo 128
    const int stage_bytes = p.stage_bytes, n_stages = p.n_stages;
    uint8_t* const ring = nm_shared + warp * n_stages * stage_bytes;
    float* const red = reinterpret_cast<float*>(nm_shared + NM_WARPS * n_stages * stage_bytes);   // [2][warp][8 NT][NM_RED_PITCH]
    constexpr int RED_WARP = 8 * NT * NM_RED_PITCH, RED = NM_WARPS * RED_WARP;
    uint8_t* const xs = reinterpret_cast<uint8_t*>(red + 2 * RED);

    const int share = (int)blockIdx.x % p.shares, cta = (int)blockIdx.x / p.shares;
    const int i0 = (int)((int64_t)cta * p.groups / p.per_share_ctas), i1 = (int)((int64_t)(cta + 1) * p.groups / p.per_share_ctas);
    const int s0 = (int)((int64_t)share * p.n_steps / p.shares), s1 = (int)((int64_t)(share + 1) * p.n_steps / p.shares);
    const int a0 = s0 + kw * (s1 - s0) / KW, a1 = s0 + (kw + 1) * (s1 - s0) / KW;   // this warp's steps
    // a row group may reach past the matrix: an image's last row is copied again, a block format's 128-row tile is filled up with zeros that stay where they are
    const int live_groups = BLOCKS ? narrow_live_groups(i0, i1, rg_shift, sub_tile, (p.rows + 15) / 16) : i1 - i0;
    NarrowRing copies(n_stages, live_groups * (a1 - a0));
    pdl_trigger();

    if constexpr (BLOCKS) {
        if (lane == 0) {
            for (int i = 0; i < n_stages; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(nm_smem(&full[warp][i])));
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
    }

    // ---- the warp's copies, in the order in which it uses them: step load_st of row group load_i
    int load_i = i0, load_st = a0;
    const uint8_t *src0 = nullptr, *src1 = nullptr;   // image: this lane's 16 bytes of rows r and r + 8
    auto copy_step = [&] {
        if (!copies.more()) return;
        const uint32_t dst = nm_smem(ring + copies.load_stage * stage_bytes);
        if constexpr (BLOCKS) {
            if (lane == 0) {
                const int tile = (load_i << rg_shift) + sub_tile;
                const bool second = tile >= p.tiles_first;
                const int rt = second ? tile - p.tiles_first : tile, r0 = (rt & 7) * 16;
                const bool q6 = (second ? p.q6_2 : p.q6) != 0;
                const uint8_t* unit = (second ? p.w2 : p.w) + ((int64_t)(rt >> 3) * p.n_steps + load_st) * (q6 ? kQ6Unit : kQ4Unit);
                const uint32_t bar = nm_smem(&full[warp][copies.load_stage]);
                nm_expect(bar, q6 ? NM_Q6_STEP : NM_Q4_STEP);
                if (!q6) {
                    nm_bulk(dst, unit + r0 * 144, NM_Q4_STEP, bar);
                } else {
                    nm_bulk(dst, unit + r0 * 128, 2048, bar);
                    nm_bulk(dst + 2048, unit + kQ6Qh + r0 * 64, 1024, bar);
                    nm_bulk(dst + 3072, unit + kQ6Sc + r0 * 16, 256, bar);
                    nm_bulk(dst + 3328, unit + kQ6D + r0 * 2, 32, bar);
                }
            }
        } else {
            if (load_st == a0) {
                const int row = ((load_i << rg_shift) + sub_tile) * 16 + r;
                const int64_t at = (int64_t)a0 * (COLS * 2) + t * 16, ld = (int64_t)p.cols * 2;
                src0 = p.w + min(row, p.rows - 1) * ld + at;
                src1 = p.w + min(row + 8, p.rows - 1) * ld + at;
            }
            nm_copy16(dst + lane * 16, src0);
            nm_copy16(dst + 512 + lane * 16, src0 + 64);
            nm_copy16(dst + 1024 + lane * 16, src1);
            nm_copy16(dst + 1536 + lane * 16, src1 + 64);
            src0 += COLS * 2;
            src1 += COLS * 2;
        }
        if (++load_st == a1) {
            load_st = a0;
            ++load_i;
        }
        copies.loaded();
    };
    for (int i = 0; i < n_stages - 1; ++i) {
        copy_step();
        if constexpr (!BLOCKS) nm_commit();
    }
    pdl_wait();

    // ---- the activations of the share's columns, in the order in which lanes read them
    int input = -1;
    auto input_of = [&](int group) {
        const int tile128 = (group << rg_shift) >> 3;
        if (p.input_tiles > 0) return tile128 / p.input_tiles;
        int k = 0;
        while (k < p.n_inputs - 1 && tile128 >= p.input_end[k]) ++k;
        return k;
    };
    auto stage_x = [&] {
        const int chunks = (s1 - s0) * (COLS / 8);   // 16-byte chunks per token
        const __half* x = p.x + (int64_t)input * p.T * p.cols + s0 * COLS;
        if constexpr (!BLOCKS) {
            // all on their way at once, behind the weights that are
            for (int c = threadIdx.x; c < chunks; c += NM_THREADS)
                for (int tok = 0; tok < p.T; ++tok) nm_copy16(nm_smem(xs + tok * pitch + c * 16), reinterpret_cast<const uint4*>(x + (int64_t)tok * p.cols) + c);
            nm_commit();
            nm_wait<0>();
        } else {
            for (int c = threadIdx.x; c < chunks; c += NM_THREADS) {
                // bits of a chunk's number inside its block: half, 64-wide run, low / high nibbles (the last two the other way round in Q6_K), half of
                // 32, eight columns; a lane's chunk t is (run, half of 32)
                const int half = (c >> 4) & 1, b3 = (c >> 3) & 1, b2 = (c >> 2) & 1, sub = c & 1;
                const int run = p.q6 ? b2 : b3, high = p.q6 ? b3 : b2;
                const int at = (c & ~31) + ((half * 2 + high) * 2 + sub) * 4 + ((run << 1) | ((c >> 1) & 1));
#pragma unroll 4
                for (int tok = 0; tok < p.T; ++tok) {   // no more at a time: the instructions are fetched anew by every launch
                    // columns (0, 2), (1, 3) of every four, as the nibbles of a word come apart
                    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(x + (int64_t)tok * p.cols) + c);
                    *reinterpret_cast<uint4*>(xs + tok * pitch + at * 16) =
                        make_uint4(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.x, v.y, 0x7632), __byte_perm(v.z, v.w, 0x5410), __byte_perm(v.z, v.w, 0x7632));
                }
            }
        }
    };
    const uint8_t* x_tok[NT];   // this lane's token rows (tokens past the last one repeat it; their columns are not stored)
#pragma unroll
    for (int j = 0; j < NT; ++j) x_tok[j] = xs + min(8 * j + g, p.T - 1) * pitch;

    int buffer = 0;
    uint32_t given_up = 0;
    for (int i = i0; i < i1; ++i) {
        if (const int next = p.n_inputs > 1 ? input_of(i) : 0; next != input) {
            input = next;   // the old input's readers met at the sums of the group before
            stage_x();
            __syncthreads();
        }
        float acc[CHAINS][NT][4];
#pragma unroll
        for (int c = 0; c < CHAINS; ++c)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[c][j][e] = 0.f;
        const int tile = (i << rg_shift) + sub_tile;
        const bool live = !BLOCKS || tile * 16 < p.rows;
        const bool q6 = BLOCKS && (tile >= p.tiles_first ? p.q6_2 : p.q6) != 0;
        int x_off = (a0 - s0) * COLS * 2;
        for (int st = a0; st < a1; ++st, x_off += COLS * 2) {
            copy_step();
            const uint8_t* src = ring + copies.stage * stage_bytes;
            if constexpr (!BLOCKS) {
                nm_commit();
                nm_wait<NM_IMAGE_STAGES - 1>();   // each lane reads what it copied itself
                const uint4 v00 = nm_lds(src + lane * 16), v01 = nm_lds(src + 512 + lane * 16), v10 = nm_lds(src + 1024 + lane * 16), v11 = nm_lds(src + 1536 + lane * 16);
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const uint4 b = nm_lds(x_tok[j] + x_off + t * 16);
                    nm_mma<BF16>(acc[0][j], v00.x, v10.x, v00.y, v10.y, b.x, b.y);
                    nm_mma<BF16>(acc[1][j], v00.z, v10.z, v00.w, v10.w, b.z, b.w);
                }
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const uint4 b = nm_lds(x_tok[j] + x_off + 64 + t * 16);
                    nm_mma<BF16>(acc[2 % CHAINS][j], v01.x, v11.x, v01.y, v11.y, b.x, b.y);
                    nm_mma<BF16>(acc[3 % CHAINS][j], v01.z, v11.z, v01.w, v11.w, b.z, b.w);
                }
            } else if (live) {
                if (given_up == 0 && !nm_wait_full(nm_smem(&full[warp][copies.stage]), copies.phase)) {
                    given_up = copies.give_up((i0 + live_groups - i) * (a1 - a0) - (st - a0));
                    atomicExch(p.status, 34);
                }
                // where the lanes' chunks lie for this matrix's format: 16 bytes apart in its own order, else in two runs
                const bool own = q6 == (p.q6 != 0);
                const int x_lane = x_off + (own ? 16 * t : (t >> 1) * 128 + (t & 1) * 16), x_high = own ? 128 : 32;
                auto multiply = [&](const uint32_t (&lo)[8], const uint32_t (&hi)[8], int half, int high) {
#pragma unroll
                    for (int sub = 0; sub < 2; ++sub)
#pragma unroll
                        for (int j = 0; j < NT; ++j) {
                            const uint4 b = nm_lds(x_tok[j] + x_lane + half * 256 + high * x_high + sub * 64);
                            nm_mma<false>(acc[2 * sub % CHAINS][j], lo[4 * sub], hi[4 * sub], lo[4 * sub + 1], hi[4 * sub + 1], b.x, b.y);
                            nm_mma<false>(acc[(2 * sub + 1) % CHAINS][j], lo[4 * sub + 2], hi[4 * sub + 2], lo[4 * sub + 3], hi[4 * sub + 3], b.z, b.w);
                        }
                };
                if (!q6) {
                    const uint8_t *b0 = src + r * 144, *b1 = b0 + 8 * 144;
                    const uint4 h0 = nm_lds(b0), h1 = nm_lds(b1);
                    uint32_t sc0[2], sc1[2], m0[2], m1[2];
                    q4_scales(h0, sc0, m0);
                    q4_scales(h1, sc1, m1);
                    const uint32_t dn0 = h0.x ^ 0x80000000u, dn1 = h1.x ^ 0x80000000u;   // d, -dmin
                    const __half2 d0 = __low2half2(*reinterpret_cast<const __half2*>(&dn0)), n0 = __high2half2(*reinterpret_cast<const __half2*>(&dn0));
                    const __half2 d1 = __low2half2(*reinterpret_cast<const __half2*>(&dn1)), n1 = __high2half2(*reinterpret_cast<const __half2*>(&dn1));
                    const int mine = 16 * (t >> 1);   // this lane's two groups of a half's four
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        const uint4 v0 = nm_lds(b0 + 16 + half * 64 + t * 16), v1 = nm_lds(b1 + 16 + half * 64 + t * 16);
                        const uint32_t w0[4] = {v0.x, v0.y, v0.z, v0.w}, w1[4] = {v1.x, v1.y, v1.z, v1.w};
                        uint32_t f0[8], f1[8];
                        q4_weights<0>(w0, sc0[half] >> mine, m0[half] >> mine, d0, n0, f0);
                        q4_weights<0>(w1, sc1[half] >> mine, m1[half] >> mine, d1, n1, f1);
                        multiply(f0, f1, half, 0);
                        q4_weights<1>(w0, sc0[half] >> mine, m0[half] >> mine, d0, n0, f0);
                        q4_weights<1>(w1, sc1[half] >> mine, m1[half] >> mine, d1, n1, f1);
                        multiply(f0, f1, half, 1);
                    }
                } else {
                    float d[2];
#pragma unroll
                    for (int q = 0; q < 2; ++q) d[q] = __half2float(*reinterpret_cast<const __half*>(src + 3328 + (r + 8 * q) * 2));
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        uint4 l[2], h[2];
                        uint2 sc[2];  // the half's eight scales
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            const int row = r + 8 * q;
                            l[q] = nm_lds(src + row * 128 + (((4 * half + t) ^ (row & 7)) << 4));
                            h[q] = nm_lds(src + 2048 + row * 64 + (((2 * half + (t & 1)) ^ (row & 3)) << 4));
                            sc[q] = *reinterpret_cast<const uint2*>(src + 3072 + row * 16 + half * 8);
                        }
#pragma unroll
                        for (int high = 0; high < 2; ++high) {
                            // quarter 2 high + (t >> 1) of the half, its 16 columns t & 1: scale 4 high + 2 (t >> 1) + (t & 1)
                            uint32_t f[2][8];
                            const int up = 2 * (2 * high + (t >> 1));   // where the quarter's two high bits lie
#pragma unroll
                            for (int q = 0; q < 2; ++q) {
                                const int scale = (int)(int8_t)((high ? sc[q].y : sc[q].x) >> (8 * t));
                                const __half2 s = __float2half2_rn(d[q] * (float)scale);
                                const uint32_t lw[4] = {l[q].x, l[q].y, l[q].z, l[q].w}, hw[4] = {h[q].x, h[q].y, h[q].z, h[q].w};
#pragma unroll
                                for (int i4 = 0; i4 < 4; ++i4)
                                    q6_to_weights<true>(((lw[i4] >> (4 * high)) & 0x0F0F0F0Fu) | (((hw[i4] >> up) & 0x03030303u) << 4), s, f[q][2 * i4], f[q][2 * i4 + 1]);
                            }
                            multiply(f[0], f[1], half, high);
                        }
                    }
                }
                __syncwarp();   // the stage is refilled next
            }
            copies.used();
        }

        // ---- the warps' slices of K meet
        float* mine = red + buffer * RED + warp * RED_WARP + r;
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float v = acc[0][j][e] + acc[1][j][e];
                if constexpr (CHAINS == 4) v += acc[2][j][e] + acc[3][j][e];
                const int tok = 8 * j + 2 * t + (e & 1);
                if (tok < p.T) mine[tok * NM_RED_PITCH + (e >> 1) * 8] = v;
            }
        __syncthreads();
        const float* sums = red + buffer * RED;
        buffer ^= 1;
        auto sum_at = [&](int row, int tok) {  // row: inside the group
            const float* q = sums + (row >> 4) * KW * RED_WARP + tok * NM_RED_PITCH + (row & 15);
            float v[NM_WARPS];
#pragma unroll
            for (int k = 0; k < NM_WARPS; ++k) v[k] = k < KW ? q[k * RED_WARP] : 0.f;
#pragma unroll
            for (int k = 1; k < NM_WARPS; ++k) v[0] += v[k];
            return v[0];
        };
        const int row0 = (i << rg_shift) * 16, n_rows = 16 << rg_shift;
        if (p.gated != 0) {
            const int n_features = n_rows >> 1, shift = 3 + rg_shift;
            for (int o = threadIdx.x; o < n_features * p.T; o += NM_THREADS) {
                const int f = o & (n_features - 1), tok = o >> shift, row = row0 + 2 * f;
                if (row >= p.rows) continue;
                const float gate = sum_at(2 * f, tok), up = sum_at(2 * f + 1, tok);
                float v;
                if (p.gated == 1 + GatedAct::Silu) v = silu_f(gate) * up;
                else if (p.gated == 1 + GatedAct::GeluTanh) v = gelu_tanh_f(gate) * up;
                else {
                    const float pre = p.act_pre != nullptr ? p.act_pre[tok] : 1.f, post = p.act_post != nullptr ? p.act_post[tok] : 1.f;
                    v = clamped_gate_f(pre * gate, pre * up, p.act_limit) * post;
                }
                const int64_t at = (int64_t)tok * p.ldyh + (row >> 1);
                if (p.yh_bf16) reinterpret_cast<__nv_bfloat16*>(p.yh)[at] = __float2bfloat16_rn(v);
                else p.yh[at] = __float2half_rn(v);
            }
        } else {
            for (int o = threadIdx.x; o < n_rows * p.T; o += NM_THREADS) {
                const int f = o & (n_rows - 1), tok = o >> (4 + rg_shift), row = row0 + f;
                if (row >= p.rows) continue;
                float v = sum_at(f, tok);
                if (p.shares > 1) {
                    p.partial[((int64_t)share * p.T + tok) * p.rows + row] = v;
                } else if (p.scattered == 0) {
                    v *= p.out_scale;
                    if (p.softcap != 0.f) v = tanhf(v * (1.0f / p.softcap)) * p.softcap;
                    p.y[(int64_t)tok * p.ldy + row] = v;
                } else if (p.scatter.rest != nullptr && row >= p.scatter.rest_from) {
                    p.scatter.rest[(int64_t)tok * p.scatter.ld_rest + row - p.scatter.rest_from] = v;
                } else {
                    const int64_t col = p.scatter.column(row);
                    if (col < 0) continue;
                    if (p.scatter.gate != nullptr) v *= sigmoid_f(p.scatter.gate_sum(tok, row));
                    p.scatter.put(p.scatter.row(tok) + col, v);
                }
            }
        }
    }
    if constexpr (BLOCKS)
        if (given_up != 0 && lane == 0)   // what is under way lands before the CTA is gone (lane 0 asks for all copies)
            NarrowRing::drain(n_stages, given_up, [&](int at, uint32_t parity) { nm_wait_full(nm_smem(&full[warp][at]), parity); });
}

size_t nm_smem_bytes(NarrowFormat format, bool q6, int T, int64_t share_cols) {
    const int nt = T <= 8 ? 1 : 2;
    const int ring = format != NarrowFormat::Blocks ? NM_IMAGE_STAGES * NM_IMAGE_STEP : (q6 ? NM_Q6_STAGES * NM_Q6_STEP : NM_Q4_STAGES * NM_Q4_STEP);
    return (size_t)NM_WARPS * ring + 2 * (size_t)NM_WARPS * 8 * nt * NM_RED_PITCH * 4 +
           (size_t)T * (share_cols * 2 + 64);
}

template <NarrowFormat FORMAT>
void launch_nm(const NmParams& p, const NarrowPlan& plan, cudaStream_t s) {
    auto* kernel = narrow_mma_kernel<FORMAT, 1>;
    if constexpr (FORMAT != NarrowFormat::Blocks)
        if (p.T > 8) kernel = narrow_mma_kernel<FORMAT, 2>;
    ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), plan.smem);
    launch_pdl(kernel, dim3(plan.ctas), dim3(NM_THREADS), plan.smem, s, p);
    MK_LAUNCH_CHECK();
}

}  // namespace

// Where the tcgen05 kernels take over (us here / there).
// Images: nowhere up to 16 tokens.  With the L2 flushed they are level - 2048 x 2048 10.3 / 12.2 at 9 to 16 tokens, 22016 x 2048 30.3 / 30.7, 24576 x 4096
// 53.2 / 51.2 at 16 - but a tick's chain of launches is not: bf16 models of 2048 wide at 9 lanes 608 / 730, 462 / 530, 549 / 574, 717 / 844 a tick, at
// 16 628 / 764, 481 / 533, 599 / 622, 749 / 857, and with a head of 131072 rows at 16 still 693 / 703, 549 / 557, 670 / 680, 809 / 819.  32 tokens: 43 / 31.
// Blocks: unpacking is a warp's own work here and sets the pace of long streams.  In ticks with the line at 20 M, 32 M and 64 M weights, one lane: 2048 wide
// 403, 386 and 386, 4096 wide 690, 659 and 691, 3584 wide 678, 649 and 685; four lanes level.
// Gated blocks (Q4_K: no other format is interleaved): the kernel there leaves whole row tiles to its CTAs, so how much of the chip it uses follows from their number: 88 and 172 tiles keep
// 59 % of the SMs busy on average, 192 keep 65, 224 keep 76.  Ticks of Q4_K models with these: 339 / 351, 386 / 402, 650 / 659, 685 / 653 at one
// lane; 337 / 347, 395 / 410, 712 / 703, 715 / 694 at four; 364 / 362, 416 / 424, 744 / 716, 795 / 711 at eight.
static bool narrow_preferred(NarrowFormat format, int64_t rows, int64_t cols, int T, bool gated, int sms) {
    if (format != NarrowFormat::Blocks) return T <= kNarrowImageRows;
    if (T > kNarrowBlockRows) return false;
    if (!gated) return rows * cols <= (int64_t)32 << 20;
    const int64_t tiles = (rows + 127) / 128, most = (tiles + sms - 1) / sms, busy = 100 * tiles / (most * sms);
    return busy <= (T <= 2 ? 70 : 62);
}

NarrowPlan narrow_plan(NarrowFormat format, bool q6, int64_t rows, int64_t cols, int T, bool gated, int max_shares, size_t scratch_floats, int n_inputs, int sms) {
    NarrowPlan best;
    const bool blocks = format == NarrowFormat::Blocks;
    if (T <= 0 || cols % nm_step_cols(blocks) != 0 || !narrow_preferred(format, rows, cols, T, gated, sms)) return best;
    if (gated) max_shares = 1;   // its pairs of rows are finished by the CTA that has their sums
    const int64_t steps = cols / nm_step_cols(blocks), tiles = (rows + 15) / 16;
    // Microseconds of a step on one CTA of an SM (half as long again with two), of a meeting of the warps, of staging the activations and of adding
    // shares: fitted to launches of 2048 ... 75776 rows at K = 2048 and 11008, 1 to 16 tokens.
    const double step_us = blocks ? (q6 ? 0.55 : 0.42) : (T <= 8 ? 0.38 : 0.41);
    for (int shift = 0; shift <= 3; ++shift) {
        const int RG = 1 << shift, KW = NM_WARPS >> shift;
        const int64_t groups = (tiles + RG - 1) / RG;
        for (int S = 1; S <= std::max(1, std::min(max_shares, 8)); ++S) {
            if (S > steps || (S > 1 && (size_t)S * T * rows > scratch_floats)) break;
            const int64_t share_steps = (steps + S - 1) / S, share_cols = share_steps * nm_step_cols(blocks);
            const size_t smem = nm_smem_bytes(format, q6, T, share_cols);
            if (smem > (size_t)200 * 1024) continue;
            const int per_sm = smem <= (size_t)112 * 1024 ? 2 : 1;
            const int64_t per_share = std::min<int64_t>(groups, std::max(1, per_sm * sms / S));
            const int64_t rounds = (groups + per_share - 1) / per_share, slice = (share_steps + KW - 1) / KW;
            const double us = (double)rounds * ((double)slice * step_us * (per_share * S > sms ? 1.5 : 1.0) + 0.25) + (double)T * share_cols * 2 / 90e3 * (n_inputs > 1 && rounds > 1 ? 2 : 1) +
                              (S > 1 ? 0.2 * S : 0.0);
            if (!best.ok || us < best.us - 1e-9) {
                best.ok = true;
                best.us = us;
                best.RG = RG;
                best.shares = S;
                best.ctas = (int)per_share * S;
                best.smem = smem;
                best.partial_floats = S > 1 ? (size_t)S * T * rows : 0;
            }
        }
    }
    return best;
}

void launch_narrow_mma(const NarrowCall& c, const NarrowPlan& plan, cudaStream_t s) {
    const bool blocks = c.format == NarrowFormat::Blocks;
    NmParams p{};
    p.T = c.T;
    p.rows = (int)c.rows;
    p.cols = (int)c.cols;
    p.n_steps = (int)(c.cols / nm_step_cols(blocks));
    p.shares = plan.shares;
    p.per_share_ctas = plan.ctas / plan.shares;
    p.rg_shift = plan.RG == 8 ? 3 : (plan.RG == 4 ? 2 : plan.RG - 1);
    p.groups = (int)(((c.rows + 15) / 16 + plan.RG - 1) / plan.RG);
    p.tiles_first = c.w2 != nullptr ? (int)(c.rows_first / 16) : INT32_MAX;
    p.q6 = c.q6;
    p.q6_2 = c.q6_2;
    const bool any_q6 = c.q6 || (c.w2 != nullptr && c.q6_2);
    p.stage_bytes = !blocks ? NM_IMAGE_STEP : (any_q6 ? NM_Q6_STEP : NM_Q4_STEP);
    p.n_stages = !blocks ? NM_IMAGE_STAGES : (any_q6 ? NM_Q6_STAGES : NM_Q4_STAGES);
    p.share_cols = (int)((p.n_steps + plan.shares - 1) / plan.shares * nm_step_cols(blocks));
    p.w = static_cast<const uint8_t*>(c.w);
    p.w2 = static_cast<const uint8_t*>(c.w2);
    p.x = c.x;
    p.n_inputs = c.n_inputs;
    p.input_tiles = c.input_tiles;
    for (int g = 0; g < kMaxRowGroups; ++g) p.input_end[g] = c.input_end[g];
    p.y = c.y;
    p.ldy = c.ldy;
    p.out_scale = c.out_scale;
    p.softcap = c.softcap;
    p.partial = c.partial;
    p.status = c.status;
    if (c.act != nullptr) {
        p.gated = 1 + c.act->kind;
        p.act_limit = c.act->limit;
        p.act_pre = c.act->pre;
        p.act_post = c.act->post;
    }
    p.yh = c.yh;
    p.ldyh = c.ldyh;
    p.yh_bf16 = c.format == NarrowFormat::BF16;
    if (c.scatter != nullptr) {
        p.scattered = 1;
        p.scatter = *c.scatter;
    }
    if (c.format == NarrowFormat::F16) launch_nm<NarrowFormat::F16>(p, plan, s);
    else if (c.format == NarrowFormat::BF16) launch_nm<NarrowFormat::BF16>(p, plan, s);
    else launch_nm<NarrowFormat::Blocks>(p, plan, s);
}

}  // namespace mk
