// Fused per-head QK RMSNorm + half-split RoPE + paged-KV scatter.
//
// Replaces, per layer, SelfAttention::project_packed_qkv's per-head norms (src/decoder.rs:1137-1154,
// applied BEFORE the rotation), RotaryEmbedding::apply (src/decoder.rs:203-257, half-split layout on
// the first rotary_dim dims) and PagedKvBatchReservation::write_layer
// (crates/macllm-kv/src/cache.rs:2543-2643): K is stored after the rotation, V unmodified, both at
// KV-head cardinality, token at slot block*block_tokens + row.
// One warp per (token, head), the head vector staged in shared memory so any head_dim works; the usual widths a few heads per warp in registers.
#include "kernels.h"
#include "rope_head.cuh"
#include <algorithm>

namespace mk {

namespace {

constexpr int RK_WARPS = 4;

template <typename KV>
__device__ __forceinline__ KV to_kv(float v);
template <>
__device__ __forceinline__ float to_kv<float>(float v) { return v; }
template <>
__device__ __forceinline__ __half to_kv<__half>(float v) { return __float2half_rn(v); }

template <typename KV>
__global__ void __launch_bounds__(RK_WARPS * 32) rope_kv_kernel(RopeKvArgs a) {
    __shared__ __align__(16) float buf[RK_WARPS][RK_MAX_D];  // rows are filled in pieces of up to 16 bytes
    pdl_trigger();
    pdl_wait();
    int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int heads_total = a.q_heads + 2 * a.kv_heads;
    int head = blockIdx.y * RK_WARPS + warp;
    int t = blockIdx.x;
    if (head >= heads_total) return;
    const int d = rope_row_width(a);
    float* x = buf[warp];

    int kind, hh;  // 0 = q, 1 = k, 2 = v
    if (head < a.q_heads) { kind = 0; hh = head; }
    else if (head < a.q_heads + a.kv_heads) { kind = 1; hh = head - a.q_heads; }
    else { kind = 2; hh = head - a.q_heads - a.kv_heads; }
    rope_head_prepare(a, kind, hh, t, kind != 2 && a.cos_t != nullptr ? a.positions[t] : 0, x, lane);
    if (kind == 0) {
        float* dst = a.q_out != nullptr ? a.q_out + (int64_t)t * a.ldq_out + hh * d : a.q + (int64_t)t * a.ldq + hh * d;
        for (int i = lane; i < d; i += 32) dst[i] = x[i];
    } else {
        int64_t slot = a.slots[t];
        int64_t blk = slot / a.block_tokens, row = slot % a.block_tokens;
        int64_t base = ((kv_page_index(blk, a.layer, a.layers, a.pool_blocks) * a.kv_heads + hh) * a.block_tokens + row) * (int64_t)d;
        KV* pool = reinterpret_cast<KV*>(kind == 1 ? a.k_pool : a.v_pool);
        for (int i = lane; i < d; i += 32) pool[base + i] = to_kv<KV>(x[i]);
    }
}

// Heads of 32 J dimensions that turn whole (or not at all), from whole projections: a warp takes U heads of a token, lane l the dimensions
// l + 32 j.  Both halves of a half-split pair are then the lane's own, the angles serve all U heads, and nothing passes through shared memory.
// The sums run as in rope_head.cuh, so both give the same bits.  Bound by HBM; with a warp per head, each waiting for its own load,
// position, slot and angles in turn, 1420 rows of 40 heads took 34 us, this 19.
template <typename KV, int J, int U>
__global__ void __launch_bounds__(RK_WARPS * 32) rope_kv_whole_kernel(RopeKvArgs a) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31, heads_total = a.q_heads + 2 * a.kv_heads, runs = (heads_total + U - 1) / U;
    const int64_t item = (int64_t)blockIdx.x * RK_WARPS + (threadIdx.x >> 5);
    const int t = (int)(item / runs), h0 = (int)(item - (int64_t)t * runs) * U;
    if (t >= a.T) return;
    constexpr int D = 32 * J;
    float x[U][J];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int h = min(h0 + u, heads_total - 1), k = h - a.q_heads, v = k - a.kv_heads;
        const float* src = k < 0 ? a.q + (int64_t)t * a.ldq + h * D : (v < 0 ? a.k + (int64_t)t * a.ldk + k * D : a.v + (int64_t)t * a.ldv + v * D);
#pragma unroll
        for (int j = 0; j < J; ++j) x[u][j] = src[lane + 32 * j];
    }
    const bool turns = a.cos_t != nullptr;
    float c[J], s[J];  // half-split: the first J / 2 count
    if (turns) {
        const int64_t at = (int64_t)a.positions[t] * (D / 2);
#pragma unroll
        for (int j = 0; j < J; ++j) {
            if (!a.interleaved && j >= J / 2) break;
            const int i = a.interleaved ? (lane >> 1) + 16 * j : lane + 32 * j;
            c[j] = a.cos_t[at + i];
            s[j] = a.sin_t[at + i];
        }
    }
    const int64_t slot = a.slots[t], blk = slot / a.block_tokens, row = slot - blk * a.block_tokens;
    const int64_t page = kv_page_index(blk, a.layer, a.layers, a.pool_blocks) * a.kv_heads;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int h = h0 + u, k = h - a.q_heads, v = k - a.kv_heads;
        if (h >= heads_total) break;
        const float* bias = k < 0 ? a.q_bias : (v < 0 ? a.k_bias : a.v_bias);
        if (bias != nullptr) {
            bias += (k < 0 ? h : (v < 0 ? k : v)) * D;
#pragma unroll
            for (int j = 0; j < J; ++j) x[u][j] += bias[lane + 32 * j];
        }
        const float* nw = k < 0 ? a.q_norm_w : (v < 0 ? a.k_norm_w : nullptr);
        if (nw != nullptr) {
            float ss = 0.f;
#pragma unroll
            for (int j = 0; j < J; ++j) ss += x[u][j] * x[u][j];
            ss = warp_sum(ss);
            const float m = sqrtf(ss / (float)D + a.norm_eps);
#pragma unroll
            for (int j = 0; j < J; ++j) x[u][j] = x[u][j] / m * nw[lane + 32 * j];
        }
        if (v < 0 && turns) {
            if (a.interleaved) {
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    const float other = __shfl_xor_sync(0xffffffffu, x[u][j], 1);
                    x[u][j] = (lane & 1) ? __fadd_rn(__fmul_rn(other, s[j]), __fmul_rn(x[u][j], c[j])) : __fsub_rn(__fmul_rn(x[u][j], c[j]), __fmul_rn(other, s[j]));
                }
            } else {
#pragma unroll
                for (int j = 0; j < J / 2; ++j) {
                    const float x1 = x[u][j], x2 = x[u][j + J / 2];
                    x[u][j] = __fsub_rn(__fmul_rn(x1, c[j]), __fmul_rn(x2, s[j]));
                    x[u][j + J / 2] = __fadd_rn(__fmul_rn(x1, s[j]), __fmul_rn(x2, c[j]));
                }
            }
        }
        if (k < 0) {
            float* dst = a.q_out != nullptr ? a.q_out + (int64_t)t * a.ldq_out + h * D : a.q + (int64_t)t * a.ldq + h * D;
#pragma unroll
            for (int j = 0; j < J; ++j) dst[lane + 32 * j] = x[u][j];
        } else {
            KV* pool = reinterpret_cast<KV*>(v < 0 ? a.k_pool : a.v_pool) + ((page + (v < 0 ? k : v)) * a.block_tokens + row) * D;
#pragma unroll
            for (int j = 0; j < J; ++j) pool[lane + 32 * j] = to_kv<KV>(x[u][j]);
        }
    }
}

template <typename KV>
bool launch_rope_whole(const RopeKvArgs& a, cudaStream_t s) {
    const int row = rope_row_width(a);
    if (a.qk_splits > 1 || a.v_splits > 1 || row != a.d || (a.dv > 0 && a.dv != a.d) || (a.cos_t != nullptr && a.rotary_dim != a.d)) return false;
    constexpr int U = 4;
    auto launch = [&](auto* kernel, int per) {
        const int64_t warps = (int64_t)a.T * ((a.q_heads + 2 * a.kv_heads + per - 1) / per);
        launch_pdl(kernel, dim3((unsigned)((warps + RK_WARPS - 1) / RK_WARPS)), dim3(RK_WARPS * 32), 0, s, a);
    };
    switch (a.d) {
        case 64: launch(rope_kv_whole_kernel<KV, 2, U>, U); return true;
        case 128: launch(rope_kv_whole_kernel<KV, 4, U>, U); return true;
        case 256: launch(rope_kv_whole_kernel<KV, 8, U / 2>, U / 2); return true;
        default: return false;
    }
}

// One CTA per token: all heads of the token in shared memory ((q_heads + kv_heads) * d + kv_heads * dv floats).
// vec: every row starts on 16 bytes and head widths are multiples of four.
template <typename KV, int THREADS>
__global__ void __launch_bounds__(THREADS) rope_kv_rows_kernel(RopeKvArgs a, int vec) {
    extern __shared__ __align__(16) float rr_row[];
    __shared__ float red[2][32];
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x, dv = a.dv > 0 ? a.dv : a.d, D = rope_row_width(a);
    const int qw = a.q_heads * a.d, kw = a.kv_heads * a.d, vw = a.kv_heads * dv;
    float *xq = rr_row, *xk = xq + qw, *xv = xk + kw;
    // a projection's row: the shares' sum and the bias; returns the thread's sum of squares
    auto load = [&](float* dst, const float* src, int n, int parts, int64_t stride, const float* bias) {
        float ss = 0.f;
        if (vec) {
            for (int c = threadIdx.x * 4; c < n; c += THREADS * 4) {
                float4 v = *reinterpret_cast<const float4*>(src + c);
#pragma unroll 8
                for (int p = 1; p < parts; ++p) {
                    const float4 w = *reinterpret_cast<const float4*>(src + (int64_t)p * stride + c);
                    v = make_float4(v.x + w.x, v.y + w.y, v.z + w.z, v.w + w.w);
                }
                if (bias != nullptr) {
                    const float4 b = *reinterpret_cast<const float4*>(bias + c);
                    v = make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w);
                }
                *reinterpret_cast<float4*>(dst + c) = v;
                ss = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ss))));
            }
            return ss;
        }
        for (int c = threadIdx.x; c < n; c += THREADS) {
            float v = src[c];
            for (int p = 1; p < parts; ++p) v += src[(int64_t)p * stride + c];
            if (bias != nullptr) v += bias[c];
            dst[c] = v;
            ss = fmaf(v, v, ss);
        }
        return ss;
    };
    float sq = load(xq, a.q + (int64_t)t * a.ldq, qw, a.qk_splits, a.qk_split_stride, a.q_bias);
    float sk = load(xk, a.k + (int64_t)t * a.ldk, kw, a.qk_splits, a.qk_split_stride, a.k_bias);
    load(xv, a.v + (int64_t)t * a.ldv, vw, a.v_splits, a.v_split_stride, a.v_bias);
    sq = warp_sum(sq);
    sk = warp_sum(sk);
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = sq;
        red[1][threadIdx.x >> 5] = sk;
    }
    __syncthreads();
    sq = sk = 0.f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) {
        sq += red[0][w];
        sk += red[1][w];
    }
    const float rq = sqrtf(sq / (float)qw + a.norm_eps), rk = sqrtf(sk / (float)kw + a.norm_eps);
    const int rd = a.cos_t != nullptr ? a.rotary_dim : 0, half = rd / 2;
    const float* cs = a.cos_t + (rd > 0 ? (int64_t)a.positions[t] * half : 0);
    const float* sn = a.sin_t + (rd > 0 ? (int64_t)a.positions[t] * half : 0);
    // value c of the head at x (norm weights at w): normed, then turned with its partner
    auto turned = [&](const float* x, const float* w, float root, int c) {
        const float own = x[c] / root * w[c];
        if (c >= rd) return own;
        const int i = a.interleaved ? c >> 1 : (c < half ? c : c - half);
        const bool first = a.interleaved ? (c & 1) == 0 : c < half;
        const int p = a.interleaved ? c ^ 1 : (first ? c + half : c - half);
        const float other = x[p] / root * w[p];
        return first ? own * cs[i] - other * sn[i] : own * cs[i] + other * sn[i];
    };
    float* q_out = a.q_out + (int64_t)t * a.ldq_out;
#pragma unroll 4
    for (int i = threadIdx.x; i < a.q_heads * D; i += THREADS) {
        const int h = i / D, c = i - h * D;
        q_out[i] = c < a.d ? turned(xq + h * a.d, a.q_norm_w + h * a.d, rq, c) : 0.f;
    }
    const int64_t slot = a.slots[t], blk = slot / a.block_tokens, row = slot % a.block_tokens;
    KV *kp = reinterpret_cast<KV*>(a.k_pool), *vp = reinterpret_cast<KV*>(a.v_pool);
    const int64_t page = kv_page_index(blk, a.layer, a.layers, a.pool_blocks) * a.kv_heads;
#pragma unroll 2
    for (int i = threadIdx.x; i < a.kv_heads * D; i += THREADS) {
        const int h = i / D, c = i - h * D;
        const int64_t at = ((page + h) * a.block_tokens + row) * (int64_t)D + c;
        kp[at] = to_kv<KV>(c < a.d ? turned(xk + h * a.d, a.k_norm_w + h * a.d, rk, c) : 0.f);
        vp[at] = to_kv<KV>(c < dv ? xv[h * dv + c] : 0.f);
    }
}

template <typename KV, int THREADS>
void launch_rope_rows(const RopeKvArgs& a, size_t smem, int vec, cudaStream_t s) {
    auto* kernel = rope_kv_rows_kernel<KV, THREADS>;
    ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    launch_pdl(kernel, dim3((unsigned)a.T), dim3(THREADS), smem, s, a, vec);
}

// All copies of a tick in one launch, a CTA per (copy, layer, head): one launch per copy cost 9 to 18 us each, whatever it moved.  PIECE: what
// a thread moves at a time; a row is a whole number of them.
template <typename PIECE>
__global__ void __launch_bounds__(128) cow_copy_kernel(PIECE* k_pool, PIECE* v_pool, const CowCopy* copies, int layers, int64_t pool_blocks, int kv_heads, int block_tokens,
                                                       int row_pieces) {
    const int per = layers * kv_heads, copy = blockIdx.x / per, layer = blockIdx.x % per / kv_heads, h = blockIdx.x % kv_heads;
    const CowCopy c = copies[copy];
    const int64_t page = (int64_t)block_tokens * row_pieces;
    const int64_t s = (kv_page_index(c.src, layer, layers, pool_blocks) * kv_heads + h) * page;
    const int64_t t = (kv_page_index(c.dst, layer, layers, pool_blocks) * kv_heads + h) * page;
    for (int i = threadIdx.x; i < c.rows * row_pieces; i += blockDim.x) {
        const PIECE k = k_pool[s + i], v = v_pool[s + i];
        k_pool[t + i] = k;
        v_pool[t + i] = v;
    }
}

}  // namespace

void launch_rope_kv(const RopeKvArgs& a, cudaStream_t s) {
    if (a.T <= 0) return;
    if (std::max({a.d, a.dv, a.d_row}) > RK_MAX_D) throw std::runtime_error("launch_rope_kv: head_dim above 256 is not supported");
    if (a.d_row > 0 && (a.d_row < a.d || a.d_row < a.dv || a.q_out == nullptr))
        throw std::runtime_error("launch_rope_kv: padded heads need a separate query output at least as wide as the heads");
    int heads_total = a.q_heads + 2 * a.kv_heads;
    if (a.kv_f16 ? launch_rope_whole<__half>(a, s) : launch_rope_whole<float>(a, s)) {
        MK_LAUNCH_CHECK();
        return;
    }
    dim3 grid((unsigned)a.T, (unsigned)((heads_total + RK_WARPS - 1) / RK_WARPS));
    if (a.kv_f16)
        launch_pdl(rope_kv_kernel<__half>, grid, dim3(RK_WARPS * 32), 0, s, a);
    else
        launch_pdl(rope_kv_kernel<float>, grid, dim3(RK_WARPS * 32), 0, s, a);
    MK_LAUNCH_CHECK();
}

void launch_rope_kv_rows(const RopeKvArgs& a, cudaStream_t s) {
    if (a.T <= 0) return;
    if (a.q_out == nullptr || a.q_norm_w == nullptr || a.k_norm_w == nullptr) throw std::runtime_error("launch_rope_kv_rows: needs norm weights and a query output");
    const size_t smem = ((size_t)a.q_heads * a.d + (size_t)a.kv_heads * (a.d + (a.dv > 0 ? a.dv : a.d))) * 4;
    if (smem > (size_t)200 * 1024) throw std::runtime_error("launch_rope_kv_rows: the projections are too wide");
    const int dv = a.dv > 0 ? a.dv : a.d;
    auto on16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    const int vec = a.d % 4 == 0 && dv % 4 == 0 && a.ldq % 4 == 0 && a.ldk % 4 == 0 && a.ldv % 4 == 0 && a.qk_split_stride % 4 == 0 && a.v_split_stride % 4 == 0 &&
                    on16(a.q) && on16(a.k) && on16(a.v) && on16(a.q_bias) && on16(a.k_bias) && on16(a.v_bias) ? 1 : 0;
    // ticks of a few rows: a row's latency counts, so many threads share it
    if (a.T <= 148) {
        if (a.kv_f16) launch_rope_rows<__half, 1024>(a, smem, vec, s);
        else launch_rope_rows<float, 1024>(a, smem, vec, s);
    } else {
        if (a.kv_f16) launch_rope_rows<__half, 256>(a, smem, vec, s);
        else launch_rope_rows<float, 256>(a, smem, vec, s);
    }
    MK_LAUNCH_CHECK();
}

void launch_cow_copies(void* k_pool, void* v_pool, int kv_f16, const CowCopy* copies, int n_copies, int layers, int64_t pool_blocks, int kv_heads, int block_tokens, int d,
                       cudaStream_t s) {
    if (n_copies <= 0) return;
    const unsigned grid = (unsigned)(n_copies * layers * kv_heads);
    const int row_bytes = d * (kv_f16 ? 2 : 4);
    // pages begin a multiple of their rows' bytes from the pool's base
    const bool wide = row_bytes % 16 == 0 && ((reinterpret_cast<uintptr_t>(k_pool) | reinterpret_cast<uintptr_t>(v_pool)) & 15) == 0;
    if (wide) cow_copy_kernel<uint4><<<grid, 128, 0, s>>>((uint4*)k_pool, (uint4*)v_pool, copies, layers, pool_blocks, kv_heads, block_tokens, row_bytes / 16);
    else cow_copy_kernel<uint16_t><<<grid, 128, 0, s>>>((uint16_t*)k_pool, (uint16_t*)v_pool, copies, layers, pool_blocks, kv_heads, block_tokens, row_bytes / 2);
    MK_LAUNCH_CHECK();
}

}  // namespace mk
