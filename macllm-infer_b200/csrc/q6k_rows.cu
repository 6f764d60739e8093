// Q6_K matrices of many rows (output heads) times two to eight activation rows: the integer sums of qgemv_q6k_kernel on tensor cores.
//
// The bytes should bound it - 32000 x 2048 holds 54 MB, 8.2 us at 6.6 TB/s - but what a byte costs in instructions still does.  On dp4a every
// product is issued four at a time and the activations are read from L1 once per pair of output rows: in a tick 15 us at one activation row, 35 at
// four, 61 at eight.  Here a scale's sixteen weights of sixteen output rows meet eight activation rows in one mma.m16n8k16 on bytes, whose
// sums stay integers: 15.1 us at four and 15.8 at eight (14.6 at one, but a one-lane decode as a whole 0.6 % longer: one row stays there).  (128256 x 2048, 216 MB: 54 us, instructions issued in 53 % of the cycles, 4.0 TB/s.)  Scales, block factors and
// the order within a block are those of the other kernel, so a block's value has the same bits; blocks are added in f32, a quarter of them per warp.
// A weight is taken as 4 (q - 32), which is its six bits at the top of a byte with the highest turned over: no subtraction byte by byte.
//
// A CTA of four warps walks tiles of sixteen output rows; a step is eight blocks (2048 columns), staged by cp.async in rows 16 bytes apart from a
// multiple of 128, so that a fragment's 8 rows x 4 lanes hit all banks.  Two stages and three CTAs per SM: 54 us where three stages and two CTAs took 61, and
// as many warps in CTAs of eight 57 to 65.  A block's factors are asked for a step ahead; asked for in the step they cost 8 %.
#include "kernels.h"
#include "device_util.h"

namespace mk {

namespace {

constexpr int Q6R_WARPS = 4, Q6R_THREADS = Q6R_WARPS * 32, Q6R_TILE = 16, Q6R_BLOCKS = 8;
constexpr int Q6R_LOW = Q6R_BLOCKS * 128 + 16, Q6R_HIGH = Q6R_BLOCKS * 64 + 16, Q6R_SCALE = Q6R_BLOCKS * 16 + 16;   // bytes between rows
constexpr int Q6R_HIGH_AT = Q6R_TILE * Q6R_LOW, Q6R_SCALE_AT = Q6R_HIGH_AT + Q6R_TILE * Q6R_HIGH, Q6R_STAGE = Q6R_SCALE_AT + Q6R_TILE * Q6R_SCALE;
constexpr int Q6R_STAGES = 2;
constexpr size_t Q6R_SMEM = (size_t)112 * 1024;   // of a CTA: two fit an SM, or three

struct Q6RowsArgs {
    const uint8_t *low, *high;
    const int8_t* scale;
    const __half* d;
    int nb, rows, tiles, T;
    const int8_t* xq;
    const float* xd;
    float* y;
    int ldy;
    float out_scale, softcap;
};

__device__ __forceinline__ void q6r_copy16(uint32_t dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void q6r_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void q6r_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// C[16 rows][8 tokens] of sixteen bytes per row.
__device__ __forceinline__ void q6r_mma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b) {
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(b), "r"(0));
}

// Four weights of group i (see qgemv_q6k_kernel) as 4 (q - 32); `high` has its fields' upper bits turned over.
template <int I>
__device__ __forceinline__ uint32_t q6r_weights(uint32_t low, uint32_t high) {
    const uint32_t l = I < 2 ? low << 2 : low >> 2;
    const uint32_t h = I == 0 ? high << 6 : I == 1 ? high << 4 : I == 2 ? high << 2 : high;
    return (l & 0x3C3C3C3Cu) | (h & 0xC0C0C0C0u);
}

template <int Q>
__device__ __forceinline__ int q6r_byte(const uint4& v) {
    const uint32_t w = Q < 4 ? v.x : Q < 8 ? v.y : Q < 12 ? v.z : v.w;
    int r;
    asm("prmt.b32 %0, %1, %1, %2;" : "=r"(r) : "r"(w), "n"((Q & 3) * 0x1111 + 0x8880));   // a byte and three times its sign
    return r;
}

struct Q6Block {
    const uint8_t *low, *high;   // of row g, this lane's bytes; row g + 8 is 8 pitches on
    uint4 sc0, sc1;              // scales of rows g, g + 8
    int sum[4] = {0, 0, 0, 0};   // row g: tokens 2t, 2t + 1; row g + 8

    template <int HALF, int S, int I>
    __device__ __forceinline__ void group(uint32_t l0, uint32_t l1, uint32_t h0, uint32_t h1, const uint4& x) {
        constexpr int W = 2 * (I & 1) + S, Q = HALF * 8 + 2 * I + S;
        int c[4];
        q6r_mma(c, q6r_weights<I>(l0, h0), q6r_weights<I>(l1, h1), W == 0 ? x.x : W == 1 ? x.y : W == 2 ? x.z : x.w);
        const int s0 = q6r_byte<Q>(sc0), s1 = q6r_byte<Q>(sc1);
        sum[0] += s0 * c[0];
        sum[1] += s0 * c[1];
        sum[2] += s1 * c[2];
        sum[3] += s1 * c[3];
    }
    template <int HALF, int S>
    __device__ __forceinline__ void run(const uint4& xa, const uint4& xb) {
        const uint8_t *l = low + HALF * 64 + S * 16, *h = high + HALF * 32 + S * 16;
        const uint32_t a0 = *reinterpret_cast<const uint32_t*>(l), a1 = *reinterpret_cast<const uint32_t*>(l + 8 * Q6R_LOW);
        const uint32_t b0 = *reinterpret_cast<const uint32_t*>(l + 32), b1 = *reinterpret_cast<const uint32_t*>(l + 32 + 8 * Q6R_LOW);
        const uint32_t h0 = *reinterpret_cast<const uint32_t*>(h) ^ 0xAAAAAAAAu, h1 = *reinterpret_cast<const uint32_t*>(h + 8 * Q6R_HIGH) ^ 0xAAAAAAAAu;
        group<HALF, S, 0>(a0, a1, h0, h1, xa);
        group<HALF, S, 1>(b0, b1, h0, h1, xa);
        group<HALF, S, 2>(a0, a1, h0, h1, xb);
        group<HALF, S, 3>(b0, b1, h0, h1, xb);
    }
};

// Shared memory: the stages, the activations [T][nb][4 quarters of groups][4 lanes][4 groups] words in rows of K + 64 bytes, their block
// factors [nb][8], two sets of the warps' sums [4][16][8].
__global__ void __launch_bounds__(Q6R_THREADS) q6k_rows_kernel(const __grid_constant__ Q6RowsArgs a) {
    extern __shared__ __align__(128) uint8_t q6r_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int K = a.nb * 256, pitch = K + 64, steps = (a.nb + Q6R_BLOCKS - 1) / Q6R_BLOCKS;
    uint8_t* xs = q6r_smem + Q6R_STAGES * Q6R_STAGE;
    float* dx = reinterpret_cast<float*>(xs + a.T * pitch);
    float* red = dx + a.nb * 8;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(q6r_smem);
    const int mine = a.tiles > (int)blockIdx.x ? (a.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0, work = mine * steps;

    // A thread's share of a step: the same chunk of some of the rows, of each plane.
    const int lr = threadIdx.x >> 6, lc = threadIdx.x & 63, hr = threadIdx.x >> 5, hc = threadIdx.x & 31, sr = threadIdx.x >> 3, sc = threadIdx.x & 7;
    const uint32_t to_low = base + lr * Q6R_LOW + lc * 16, to_high = base + Q6R_HIGH_AT + hr * Q6R_HIGH + hc * 16, to_scale = base + Q6R_SCALE_AT + sr * Q6R_SCALE + sc * 16;
    auto fetch = [&](int n) {
        if (n < work) {
            const int tile = n / steps, row0 = ((int)blockIdx.x + tile * (int)gridDim.x) * Q6R_TILE, b0 = (n - tile * steps) * Q6R_BLOCKS, m = min(Q6R_BLOCKS, a.nb - b0);
            const uint32_t at = n % Q6R_STAGES * Q6R_STAGE;
            const int64_t first = (int64_t)row0 * a.nb + b0;
            const int last = min(Q6R_TILE, a.rows - row0) - 1;   // a row behind the last one reads the last one and is not stored
            const uint8_t *low = a.low + first * 128 + lc * 16, *high = a.high + first * 64 + hc * 16;
            if (lc < m * 8) {
#pragma unroll
                for (int i = 0; i < Q6R_TILE; i += Q6R_THREADS / 64) q6r_copy16(to_low + at + i * Q6R_LOW, low + (uint32_t)(min(lr + i, last) * a.nb) * 128);
            }
            if (hc < m * 4) {
#pragma unroll
                for (int i = 0; i < Q6R_TILE; i += Q6R_THREADS / 32) q6r_copy16(to_high + at + i * Q6R_HIGH, high + (uint32_t)(min(hr + i, last) * a.nb) * 64);
            }
            if (sr < Q6R_TILE && sc < m) q6r_copy16(to_scale + at, a.scale + first * 16 + (uint32_t)(min(sr, last) * a.nb) * 16 + sc * 16);
        }
        q6r_commit();
    };
    static_assert((Q6R_THREADS == 128 || Q6R_THREADS == 256) && Q6R_BLOCKS == 8 && Q6R_TILE == 16);

    pdl_trigger();
    for (int n = 0; n < Q6R_STAGES - 1; ++n) fetch(n);   // the weights do not wait for the predecessor
    pdl_wait();
    for (int i = threadIdx.x; i < a.T * (K / 16); i += Q6R_THREADS) {
        const int tok = i / (K / 16), c = i - tok * (K / 16);
        const int half = c >> 3 & 1, in = c & 7, q = half * 8 + in;   // sixteen bytes: a group
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(a.xq + (int64_t)tok * K) + c);
        uint32_t* to = reinterpret_cast<uint32_t*>(xs + tok * pitch + (c >> 4) * 256 + (q >> 2) * 64) + (q & 3);
        to[0] = v.x; to[4] = v.y; to[8] = v.z; to[12] = v.w;
    }
    for (int i = threadIdx.x; i < a.nb * 8; i += Q6R_THREADS) dx[i] = (i & 7) < a.T ? __ldcg(a.xd + (int64_t)(i & 7) * a.nb + (i >> 3)) : 0.f;

    const uint8_t* xrow = xs + (g < a.T ? g : 0) * pitch + t * 16;   // columns behind the last activation row are not stored
    // block factors of this lane's rows: of a step's blocks, asked for a step ahead
    constexpr int MINE = Q6R_BLOCKS / Q6R_WARPS;
    __half d0[MINE], d1[MINE];
    auto factors = [&](int n) {
        const int row0 = ((int)blockIdx.x + n / steps * (int)gridDim.x) * Q6R_TILE, b0 = n % steps * Q6R_BLOCKS;
        const int64_t r0 = min(row0 + g, a.rows - 1), r1 = min(row0 + g + 8, a.rows - 1);
#pragma unroll
        for (int j = 0; j < MINE; ++j) {
            const int b = min(b0 + warp + j * Q6R_WARPS, a.nb - 1);
            d0[j] = a.d[r0 * a.nb + b];
            d1[j] = a.d[r1 * a.nb + b];
        }
    };
    if (work > 0) factors(0);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int n = 0; n < work; ++n) {
        const int row0 = ((int)blockIdx.x + n / steps * (int)gridDim.x) * Q6R_TILE, step = n % steps, b0 = step * Q6R_BLOCKS;
        q6r_wait<Q6R_STAGES - 2>();
        __syncthreads();   // step n is here for everyone, and everyone is done with the one whose place the next takes
        fetch(n + Q6R_STAGES - 1);
        float e0[MINE], e1[MINE];
#pragma unroll
        for (int j = 0; j < MINE; ++j) {
            e0[j] = __half2float(d0[j]) * 0.25f;
            e1[j] = __half2float(d1[j]) * 0.25f;
        }
        if (n + 1 < work) factors(n + 1);
        const uint8_t* st = q6r_smem + n % Q6R_STAGES * Q6R_STAGE;
#pragma unroll
        for (int j = 0; j < Q6R_BLOCKS / Q6R_WARPS; ++j) {
            const int bl = warp + j * Q6R_WARPS, b = b0 + bl;
            if (b >= a.nb) break;
            Q6Block blk;
            blk.low = st + g * Q6R_LOW + bl * 128 + 4 * t;
            blk.high = st + Q6R_HIGH_AT + g * Q6R_HIGH + bl * 64 + 4 * t;
            blk.sc0 = *reinterpret_cast<const uint4*>(st + Q6R_SCALE_AT + g * Q6R_SCALE + bl * 16);
            blk.sc1 = *reinterpret_cast<const uint4*>(st + Q6R_SCALE_AT + (g + 8) * Q6R_SCALE + bl * 16);
            uint4 x[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) x[q] = *reinterpret_cast<const uint4*>(xrow + b * 256 + q * 64);
            blk.run<0, 0>(x[0], x[1]);
            blk.run<0, 1>(x[0], x[1]);
            blk.run<1, 0>(x[2], x[3]);
            blk.run<1, 1>(x[2], x[3]);
            const float2 f = *reinterpret_cast<const float2*>(dx + b * 8 + 2 * t);
            acc[0] += f.x * (e0[j] * (float)blk.sum[0]);
            acc[1] += f.y * (e0[j] * (float)blk.sum[1]);
            acc[2] += f.x * (e1[j] * (float)blk.sum[2]);
            acc[3] += f.y * (e1[j] * (float)blk.sum[3]);
        }
        if (step + 1 < steps) continue;
        float* sums = red + (n / steps & 1) * Q6R_WARPS * 128;   // two sets: the barrier above lies between a set's readers and its next writers
        *reinterpret_cast<float2*>(sums + warp * 128 + g * 8 + 2 * t) = make_float2(acc[0], acc[1]);
        *reinterpret_cast<float2*>(sums + warp * 128 + (g + 8) * 8 + 2 * t) = make_float2(acc[2], acc[3]);
        acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
        __syncthreads();
        const int tok = threadIdx.x >> 4, row = threadIdx.x & 15;
        if (tok < a.T && row0 + row < a.rows) {
            const float* s = sums + row * 8 + tok;
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < Q6R_WARPS; ++w) v += s[w * 128];
            v *= a.out_scale;
            if (a.softcap != 0.f) v = tanhf(v * (1.0f / a.softcap)) * a.softcap;
            a.y[(int64_t)tok * a.ldy + row0 + row] = v;
        }
    }
}

size_t q6r_bytes(int nb, int T) { return (size_t)Q6R_STAGES * Q6R_STAGE + (size_t)T * (nb * 256 + 64) + (size_t)nb * 32 + 2 * Q6R_WARPS * 128 * 4; }

}  // namespace

bool q6k_rows_cover(const QWeight& W, const ActQ& x, int T) {
    if (W.type != QT_Q6_K || W.cols % 256 != 0 || T < 2 || T > 8 || W.rows > (int64_t)1 << 30) return false;
    const uintptr_t at = reinterpret_cast<uintptr_t>(W.p0) | reinterpret_cast<uintptr_t>(W.p1) | reinterpret_cast<uintptr_t>(W.p2) | reinterpret_cast<uintptr_t>(x.qs);
    return (at & 15) == 0 && q6r_bytes((int)(W.cols / 256), T) <= Q6R_SMEM;
}

void launch_q6k_rows(const QWeight& W, const ActQ& x, int T, float* y, int ldy, float out_scale, float softcap, cudaStream_t s) {
    Q6RowsArgs a;
    a.low = (const uint8_t*)W.p0;
    a.high = (const uint8_t*)W.p1;
    a.scale = (const int8_t*)W.p2;
    a.d = (const __half*)W.p3;
    a.nb = (int)(W.cols / 256);
    a.rows = (int)W.rows;
    a.tiles = (a.rows + Q6R_TILE - 1) / Q6R_TILE;
    a.T = T;
    a.xq = x.qs;
    a.xd = x.d;
    a.y = y;
    a.ldy = ldy;
    a.out_scale = out_scale;
    a.softcap = softcap;
    const size_t smem = q6r_bytes(a.nb, T);
    const int per_sm = smem <= (size_t)75 * 1024 ? 3 : 2;
    ensure_dynamic_smem(reinterpret_cast<const void*>(&q6k_rows_kernel), smem);
    launch_pdl(q6k_rows_kernel, dim3((unsigned)std::min(a.tiles, per_sm * device_sm_count())), dim3(Q6R_THREADS), smem, s, a);
    MK_LAUNCH_CHECK();
}

}  // namespace mk
