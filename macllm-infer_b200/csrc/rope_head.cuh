// One head vector of one token on its way from the projection to the attention: summation of split-K shares, an optional bias, the
// optional per-head RMSNorm (SelfAttention::project_packed_qkv, src/decoder.rs:1137-1154, applied BEFORE the rotation)
// and the half-split rotation (RotaryEmbedding::apply, src/decoder.rs:203-257).  Shared by the stand-alone
// RoPE + KV-scatter kernel and by the decode attention kernel that prepares its own rows, so that both produce the
// same bits.
#pragma once
#include "kernels.h"

namespace mk {

constexpr int RK_MAX_D = 256;

// Width of a head's row in q_out and in the pools.
__host__ __device__ __forceinline__ int rope_row_width(const RopeKvArgs& a) { return a.d_row > 0 ? a.d_row : a.d; }

__device__ __forceinline__ void rope_add(float& a, float b) { a += b; }
__device__ __forceinline__ void rope_add(float2& a, float2 b) { a.x += b.x; a.y += b.y; }
__device__ __forceinline__ void rope_add(float4& a, float4 b) { a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w; }
// x = the shares' sum in share order.  Several shares travel together: a share is an L2 access away, and a head that fetches one after
// the other waits for each.
template <typename V>
__device__ __forceinline__ void rope_sum_shares(const float* src, int n_parts, int64_t part_stride, int d, float* x, int lane) {
    constexpr int W = sizeof(V) / 4, AHEAD = W == 4 ? 4 : 8;
    for (int i = lane * W; i < d; i += 32 * W) {
        V v = *reinterpret_cast<const V*>(src + i);
        for (int sp = 1; sp < n_parts; sp += AHEAD) {
            V w[AHEAD];
#pragma unroll
            for (int j = 0; j < AHEAD; ++j)
                if (sp + j < n_parts) w[j] = *reinterpret_cast<const V*>(src + (int64_t)(sp + j) * part_stride + i);
#pragma unroll
            for (int j = 0; j < AHEAD; ++j)
                if (sp + j < n_parts) rope_add(v, w[j]);
        }
        *reinterpret_cast<V*>(x + i) = v;
    }
}

// The same for up to N heads of one warp that lie d floats each: their first loads, and those of every share, are on their way together.
template <typename V, int N>
__device__ __forceinline__ void rope_sum_heads(const float* const (&src)[N], const int (&n_parts)[N], const int64_t (&stride)[N], int n, int d, float* const (&x)[N], int lane) {
    constexpr int W = sizeof(V) / 4;
    int most = 1;
#pragma unroll
    for (int k = 0; k < N; ++k)
        if (k < n) most = max(most, n_parts[k]);
    for (int i = lane * W; i < d; i += 32 * W) {
        V v[N];
#pragma unroll
        for (int k = 0; k < N; ++k)
            if (k < n) v[k] = *reinterpret_cast<const V*>(src[k] + i);
        constexpr int AHEAD = 3;
        for (int sp = 1; sp < most; sp += AHEAD) {
            V w[AHEAD][N];
#pragma unroll
            for (int j = 0; j < AHEAD; ++j)
#pragma unroll
                for (int k = 0; k < N; ++k)
                    if (k < n && sp + j < n_parts[k]) w[j][k] = *reinterpret_cast<const V*>(src[k] + (int64_t)(sp + j) * stride[k] + i);
#pragma unroll
            for (int j = 0; j < AHEAD; ++j)
#pragma unroll
                for (int k = 0; k < N; ++k)
                    if (k < n && sp + j < n_parts[k]) rope_add(v[k], w[j][k]);
        }
#pragma unroll
        for (int k = 0; k < N; ++k)
            if (k < n) *reinterpret_cast<V*>(x[k] + i) = v[k];
    }
}

// What a lane turns its share of a head by: constant tables, so they can be fetched ahead of everything.
struct RopeAngles {
    float c[RK_MAX_D / 64], s[RK_MAX_D / 64];
};
__device__ __forceinline__ RopeAngles rope_angles(const RopeKvArgs& a, int position, int lane) {
    RopeAngles r;
    const int half = a.rotary_dim / 2;
    const float* c = a.cos_t + (int64_t)position * half;
    const float* s = a.sin_t + (int64_t)position * half;
#pragma unroll
    for (int j = 0; j < RK_MAX_D / 64; ++j) {
        const int i = lane + 32 * j;
        r.c[j] = a.cos_t != nullptr && i < half ? c[i] : 0.f;
        r.s[j] = a.cos_t != nullptr && i < half ? s[i] : 0.f;
    }
    return r;
}

// Where a head's f32 vector begins.  kind: 0 = q, 1 = k, 2 = v; hh = head index within its kind; t = packed token row.
__device__ __forceinline__ int rope_head_width(const RopeKvArgs& a, int kind) { return kind == 2 && a.dv > 0 ? a.dv : a.d; }
__device__ __forceinline__ const float* rope_head_source(const RopeKvArgs& a, int kind, int hh, int t) {
    const int d = rope_head_width(a, kind);
    return kind == 0 ? a.q + (int64_t)t * a.ldq + hh * d : (kind == 1 ? a.k + (int64_t)t * a.ldk + hh * d : a.v + (int64_t)t * a.ldv + hh * d);
}

// One warp: bias, norm and rotation of the sums in x (the warp's row of shared memory), zeros up to the row width; a __syncwarp at the end.
__device__ __forceinline__ void rope_head_finish(const RopeKvArgs& a, int kind, int hh, const RopeAngles& angles, float* x, int lane) {
    const int d = rope_head_width(a, kind), half = a.rotary_dim / 2;
    const float* bias = kind == 0 ? a.q_bias : (kind == 1 ? a.k_bias : a.v_bias);
    if (bias != nullptr) {
        __syncwarp();
        for (int i = lane; i < d; i += 32) x[i] += bias[hh * d + i];
    }
    for (int i = d + lane; i < rope_row_width(a); i += 32) x[i] = 0.f;
    __syncwarp();

    const float* nw = kind == 0 ? a.q_norm_w : (kind == 1 ? a.k_norm_w : nullptr);
    if (nw != nullptr) {
        float ss = 0.f;
        for (int i = lane; i < d; i += 32) ss += x[i] * x[i];
        ss = warp_sum(ss);
        float m = sqrtf(ss / (float)d + a.norm_eps);
        for (int i = lane; i < d; i += 32) x[i] = x[i] / m * nw[i];
        __syncwarp();
    }
    if (kind != 2 && a.cos_t != nullptr) {
        float r1[RK_MAX_D / 64], r2[RK_MAX_D / 64];
        const int step = a.interleaved ? 2 : 1, off = a.interleaved ? 1 : half;
#pragma unroll
        for (int j = 0; j < RK_MAX_D / 64; ++j) {
            const int i = lane + 32 * j;
            if (i >= half) break;
            const float x1 = x[i * step], x2 = x[i * step + off];
            r1[j] = __fsub_rn(__fmul_rn(x1, angles.c[j]), __fmul_rn(x2, angles.s[j]));
            r2[j] = __fadd_rn(__fmul_rn(x1, angles.s[j]), __fmul_rn(x2, angles.c[j]));
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < RK_MAX_D / 64; ++j) {
            const int i = lane + 32 * j;
            if (i >= half) break;
            x[i * step] = r1[j];
            x[i * step + off] = r2[j];
        }
        __syncwarp();
    }
}

// One warp, one head: x holds the finished head (zero-filled to the row width) on return.
__device__ __forceinline__ void rope_head_prepare(const RopeKvArgs& a, int kind, int hh, int t, int position, float* x, int lane) {
    const int d = rope_head_width(a, kind);
    const float* src = rope_head_source(a, kind, hh, t);
    const int n_parts = kind == 2 ? a.v_splits : a.qk_splits;
    const int64_t part_stride = kind == 2 ? a.v_split_stride : a.qk_split_stride;
    RopeAngles angles = {};
    if (kind != 2) angles = rope_angles(a, position, lane);   // the rotation's angles do not wait for the shares
    const uintptr_t place = reinterpret_cast<uintptr_t>(src) | (uintptr_t)(part_stride * 4);
    if ((d & 127) == 0 && (place & 15) == 0) rope_sum_shares<float4>(src, n_parts, part_stride, d, x, lane);
    else if ((d & 63) == 0 && (place & 7) == 0) rope_sum_shares<float2>(src, n_parts, part_stride, d, x, lane);
    else rope_sum_shares<float>(src, n_parts, part_stride, d, x, lane);
    rope_head_finish(a, kind, hh, angles, x, lane);
}

}  // namespace mk
