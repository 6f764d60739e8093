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

// One warp.  kind: 0 = q, 1 = k, 2 = v; hh = head index within its kind; t = packed token row; x = the warp's row
// of shared memory, holding the finished head (zero-filled to the row width) on return (after a __syncwarp).
__device__ __forceinline__ void rope_head_prepare(const RopeKvArgs& a, int kind, int hh, int t, int position, float* x, int lane) {
    const int d = kind == 2 && a.dv > 0 ? a.dv : a.d;
    const float* src = kind == 0 ? a.q + (int64_t)t * a.ldq + hh * d : (kind == 1 ? a.k + (int64_t)t * a.ldk + hh * d : a.v + (int64_t)t * a.ldv + hh * d);
    const int n_parts = kind == 2 ? a.v_splits : a.qk_splits;
    const int64_t part_stride = kind == 2 ? a.v_split_stride : a.qk_split_stride;
    // the rotation's angles do not wait for the shares
    const bool turns = kind != 2 && a.cos_t != nullptr;
    const int half = a.rotary_dim / 2;
    float rc[RK_MAX_D / 64], rs[RK_MAX_D / 64];
    if (turns) {
        const float* c = a.cos_t + (int64_t)position * half;
        const float* s = a.sin_t + (int64_t)position * half;
#pragma unroll
        for (int j = 0; j < RK_MAX_D / 64; ++j) {
            const int i = lane + 32 * j;
            rc[j] = i < half ? c[i] : 0.f;
            rs[j] = i < half ? s[i] : 0.f;
        }
    }
    const uintptr_t place = reinterpret_cast<uintptr_t>(src) | (uintptr_t)(part_stride * 4);
    if ((d & 127) == 0 && (place & 15) == 0) rope_sum_shares<float4>(src, n_parts, part_stride, d, x, lane);
    else if ((d & 63) == 0 && (place & 7) == 0) rope_sum_shares<float2>(src, n_parts, part_stride, d, x, lane);
    else rope_sum_shares<float>(src, n_parts, part_stride, d, x, lane);
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
    if (turns) {
        float r1[RK_MAX_D / 64], r2[RK_MAX_D / 64];
        const int step = a.interleaved ? 2 : 1, off = a.interleaved ? 1 : half;
#pragma unroll
        for (int j = 0; j < RK_MAX_D / 64; ++j) {
            const int i = lane + 32 * j;
            if (i >= half) break;
            const float x1 = x[i * step], x2 = x[i * step + off];
            r1[j] = __fsub_rn(__fmul_rn(x1, rc[j]), __fmul_rn(x2, rs[j]));
            r2[j] = __fadd_rn(__fmul_rn(x1, rs[j]), __fmul_rn(x2, rc[j]));
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

}  // namespace mk
