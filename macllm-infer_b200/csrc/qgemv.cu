// Quantised matrix-vector kernels for decode rows: y[t][n] = sum_k x[t][k] * W[n][k].
//
// Replaces, on this path, the reference's LinearOp::Quantized forward
// (src/model_weights.rs:346-377 -> candle QMatMul): weights stay in their GGUF block format in
// HBM (block sizes src/gguf.rs:386-408), activations arrive as 8-bit blocks, and every block dot
// product is an exact integer sum (dp4a) scaled in f32 - the arithmetic of the reference's CPU path.
//
// Only the weights are promised to the compiler as constant (const __restrict__): a load of such memory may move in front of pdl_wait(), and
// what a predecessor produces must not.
//
// Memory plan: a warp streams the blocks of its output rows with 128-bit (Q4_K,
// Q8_0) or 64-bit (Q6_K planes) loads, eight lanes per 256-weight block, so a warp consumes whole
// 128-byte lines; activations (T*K bytes) are re-read from L1/L2.  Each weight byte leaves HBM once
// per call when T <= NT; larger T re-walks the row from cache in passes.  Where there are warps for every
// scheduler all the same, a warp takes R output rows that follow one another: their weights travel together, and an activation that was
// fetched meets all of them (with one row per warp and eight sums whatever T, 32000 x 2048 in Q6_K took 26 us at one activation row, this 15).
// Two to eight activation rows of a tall Q6_K matrix go to tensor cores instead (q6k_rows.cu).
#include "kernels.h"
#include "mma_bf16.cuh"
#include <algorithm>

namespace mk {

namespace {

constexpr int GEMV_WARPS = 4;
constexpr int NT_MAX = 8;  // most activation rows of a pass

// Optional expert grouping: blockIdx.y selects the expert, whose output rows are [offsets[e], offsets[e+1]).
struct Group {
    const int32_t* offsets = nullptr;
    const int32_t* src_row = nullptr;
};
__device__ __forceinline__ void group_range(const Group& g, int T, int& t_begin, int& t_end) {
    if (g.offsets != nullptr) { t_begin = g.offsets[blockIdx.y]; t_end = g.offsets[blockIdx.y + 1]; }
    else { t_begin = 0; t_end = T; }
}
__device__ __forceinline__ int src_of(const Group& g, int t) { return g.src_row != nullptr ? g.src_row[t] : t; }

__device__ __forceinline__ void q4k_scale_min(const uint8_t* s, int j, int& sc, int& mn) {
    if (j < 4) {
        sc = s[j] & 63;
        mn = s[j + 4] & 63;
    } else {
        sc = (s[j + 4] & 0xF) | ((s[j - 4] >> 6) << 4);
        mn = (s[j + 4] >> 4) | ((s[j] >> 6) << 4);
    }
}

template <int NT>
__device__ __forceinline__ void finish_rows(float (&acc)[NT], int n, int out, int t0, int T, float* y, int ldy, float out_scale,
                                            float softcap) {
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        float v = warp_sum(acc[t]);
        if ((threadIdx.x & 31) == 0 && t0 + t < T && n < out) {
            v *= out_scale;
            if (softcap != 0.f) v = tanhf(v * (1.0f / softcap)) * softcap;
            y[(int64_t)(t0 + t) * ldy + n] = v;
        }
    }
}

// ---------------------------------------------------------------- Q4_K
template <int NT, int R>
__global__ void __launch_bounds__(GEMV_WARPS * 32) qgemv_q4k_kernel(const uint8_t* __restrict__ W, int nb, int out,
                                                                    const int8_t* xq,
                                                                    const float* xd,
                                                                    const int16_t* xbs, int T,
                                                                    float* __restrict__ y, int ldy, float out_scale,
                                                                    float softcap, Group grp) {
    pdl_trigger();
    bool waited = grp.offsets != nullptr;  // the weights do not wait for the predecessor, row ranges and activations do
    if (waited) pdl_wait();
    const int n0 = (blockIdx.x * GEMV_WARPS + (threadIdx.x >> 5)) * R;
    if (n0 >= out) {
        if (!waited) pdl_wait();
        return;
    }
    int lane = threadIdx.x & 31;
    int part = lane & 7;       // 16-byte slice of the 128 nibble bytes
    int j = part >> 1;         // 64-weight chunk
    int h = part & 1;          // half of the chunk's 32 bytes
    const int K = nb * 256;
    const uint8_t* w_row[R];  // a row behind the last one reads the last one and is not stored
#pragma unroll
    for (int r = 0; r < R; ++r) w_row[r] = W + ((int64_t)blockIdx.y * out + min(n0 + r, out - 1)) * nb * 144;
    int t_first;
    group_range(grp, T, t_first, T);

    for (int t0 = t_first; t0 < T; t0 += NT) {
        float acc[R][NT] = {};
        int rows = min(NT, T - t0);
        for (int ib = lane >> 3; ib < nb; ib += 4) {
            uint32_t ql[R][4], qh[R][4];
            float d[R], dmin[R];
            int sc_lo[R], m_lo[R], sc_hi[R], m_hi[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const uint8_t* blk = w_row[r] + (int64_t)ib * 144;
                uint4 q = *reinterpret_cast<const uint4*>(blk + 16 + 16 * part);
                uint32_t dm = *reinterpret_cast<const uint32_t*>(blk);
                d[r] = __half2float(__ushort_as_half((unsigned short)(dm & 0xFFFF)));
                dmin[r] = __half2float(__ushort_as_half((unsigned short)(dm >> 16)));
                q4k_scale_min(blk + 4, 2 * j, sc_lo[r], m_lo[r]);
                q4k_scale_min(blk + 4, 2 * j + 1, sc_hi[r], m_hi[r]);
                const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    ql[r][i] = w[i] & 0x0F0F0F0Fu;
                    qh[r][i] = (w[i] >> 4) & 0x0F0F0F0Fu;
                }
            }
            if (!waited) {
                pdl_wait();
                waited = true;
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                if (t < rows) {
                    const int64_t xrow = src_of(grp, t0 + t);
                    const int8_t* xr = xq + xrow * K + ib * 256 + 64 * j + 16 * h;
                    const int4 xl = *reinterpret_cast<const int4*>(xr), xh = *reinterpret_cast<const int4*>(xr + 32);
                    const int16_t* bs = xbs + xrow * (K / 16) + ib * 16 + 4 * j + h;
                    const int b0 = (int)bs[0], b2 = (int)bs[2];
                    const float dx = xd[xrow * nb + ib];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        int s_lo = __dp4a((int)ql[r][0], xl.x, 0);
                        s_lo = __dp4a((int)ql[r][1], xl.y, s_lo);
                        s_lo = __dp4a((int)ql[r][2], xl.z, s_lo);
                        s_lo = __dp4a((int)ql[r][3], xl.w, s_lo);
                        int s_hi = __dp4a((int)qh[r][0], xh.x, 0);
                        s_hi = __dp4a((int)qh[r][1], xh.y, s_hi);
                        s_hi = __dp4a((int)qh[r][2], xh.z, s_hi);
                        s_hi = __dp4a((int)qh[r][3], xh.w, s_hi);
                        int isum = sc_lo[r] * s_lo + sc_hi[r] * s_hi;
                        int msum = m_lo[r] * b0 + m_hi[r] * b2;
                        acc[r][t] += dx * (d[r] * (float)isum - dmin[r] * (float)msum);
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) finish_rows<NT>(acc[r], n0 + r, out, t0, T, y, ldy, out_scale, softcap);
    }
    if (!waited) pdl_wait();  // a lane without blocks
}

// ---------------------------------------------------------------- Q6_K (planar layout)
template <int NT, int R>
__global__ void __launch_bounds__(GEMV_WARPS * 32) qgemv_q6k_kernel(const uint8_t* __restrict__ ql_p,
                                                                    const uint8_t* __restrict__ qh_p,
                                                                    const int8_t* __restrict__ sc_p,
                                                                    const __half* __restrict__ d_p, int nb, int out,
                                                                    const int8_t* xq,
                                                                    const float* xd, int T,
                                                                    float* __restrict__ y, int ldy, float out_scale,
                                                                    float softcap, Group grp) {
    pdl_trigger();
    bool waited = grp.offsets != nullptr;  // the weights do not wait for the predecessor, row ranges and activations do
    if (waited) pdl_wait();
    const int n0 = (blockIdx.x * GEMV_WARPS + (threadIdx.x >> 5)) * R;
    if (n0 >= out) {
        if (!waited) pdl_wait();
        return;
    }
    int lane = threadIdx.x & 31;
    int part = lane & 7;
    int half = part >> 2;          // 128-weight half of the block
    int l0 = (part & 3) * 8;       // eight consecutive positions inside the half
    const int K = nb * 256;
    int64_t row_blk[R];  // a row behind the last one reads the last one and is not stored
#pragma unroll
    for (int r = 0; r < R; ++r) row_blk[r] = ((int64_t)blockIdx.y * out + min(n0 + r, out - 1)) * nb;
    int t_first;
    group_range(grp, T, t_first, T);

    for (int t0 = t_first; t0 < T; t0 += NT) {
        float acc[R][NT] = {};
        int rows = min(NT, T - t0);
        for (int ib = lane >> 3; ib < nb; ib += 4) {
            uint32_t g[R][4][2];  // four groups of eight 6-bit values, re-centred to [-32, 31]
            int sc[R][4];
            float d[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int64_t b = row_blk[r] + ib;
                const uint2 qa = *reinterpret_cast<const uint2*>(ql_p + b * 128 + half * 64 + l0);
                const uint2 qb = *reinterpret_cast<const uint2*>(ql_p + b * 128 + half * 64 + 32 + l0);
                const uint2 qhh = *reinterpret_cast<const uint2*>(qh_p + b * 64 + half * 32 + l0);
                const int8_t* scale = sc_p + b * 16 + half * 8 + (l0 >> 4);
#pragma unroll
                for (int i = 0; i < 4; ++i) sc[r][i] = scale[2 * i];
                d[r] = __half2float(d_p[b]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint2 lo = (i & 1) ? qb : qa;
                    const int sh = (i >> 1) * 4;
                    g[r][i][0] = __vsub4(((lo.x >> sh) & 0x0F0F0F0Fu) | (((qhh.x >> (2 * i)) & 0x03030303u) << 4), 0x20202020u);
                    g[r][i][1] = __vsub4(((lo.y >> sh) & 0x0F0F0F0Fu) | (((qhh.y >> (2 * i)) & 0x03030303u) << 4), 0x20202020u);
                }
            }
            if (!waited) {
                pdl_wait();
                waited = true;
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                if (t < rows) {
                    const int64_t xrow = src_of(grp, t0 + t);
                    const int8_t* xr = xq + xrow * K + ib * 256 + half * 128 + l0;
                    int2 x[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const int2*>(xr + 32 * i);
                    const float dx = xd[xrow * nb + ib];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        int isum = 0;
#pragma unroll
                        for (int i = 0; i < 4; ++i) isum += sc[r][i] * __dp4a((int)g[r][i][1], x[i].y, __dp4a((int)g[r][i][0], x[i].x, 0));
                        acc[r][t] += dx * (d[r] * (float)isum);
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) finish_rows<NT>(acc[r], n0 + r, out, t0, T, y, ldy, out_scale, softcap);
    }
    if (!waited) pdl_wait();  // a lane without blocks
}

// ---------------------------------------------------------------- Q8_0 (planar layout)
template <int NT, int R>
__global__ void __launch_bounds__(GEMV_WARPS * 32) qgemv_q80_kernel(const int8_t* __restrict__ qs_p,
                                                                    const __half* __restrict__ d_p, int K, int out,
                                                                    const int8_t* xq,
                                                                    const float* xd, int T,
                                                                    float* __restrict__ y, int ldy, float out_scale,
                                                                    float softcap, Group grp) {
    pdl_trigger();
    bool waited = grp.offsets != nullptr;  // the weights do not wait for the predecessor, row ranges and activations do
    if (waited) pdl_wait();
    const int n0 = (blockIdx.x * GEMV_WARPS + (threadIdx.x >> 5)) * R;
    if (n0 >= out) {
        if (!waited) pdl_wait();
        return;
    }
    int lane = threadIdx.x & 31;
    int nb = K / 32;
    int64_t w_row[R];  // a row behind the last one reads the last one and is not stored
#pragma unroll
    for (int r = 0; r < R; ++r) w_row[r] = (int64_t)blockIdx.y * out + min(n0 + r, out - 1);
    int t_first;
    group_range(grp, T, t_first, T);
    for (int t0 = t_first; t0 < T; t0 += NT) {
        float acc[R][NT] = {};
        int rows = min(NT, T - t0);
        for (int b = lane; b < nb; b += 32) {
            int4 w0[R], w1[R];
            float d[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                w0[r] = *reinterpret_cast<const int4*>(qs_p + w_row[r] * K + b * 32);
                w1[r] = *reinterpret_cast<const int4*>(qs_p + w_row[r] * K + b * 32 + 16);
                d[r] = __half2float(d_p[w_row[r] * nb + b]);
            }
            if (!waited) {
                pdl_wait();
                waited = true;
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                if (t < rows) {
                    const int64_t xrow = src_of(grp, t0 + t);
                    const int8_t* xr = xq + xrow * K + b * 32;
                    const int4 x0 = *reinterpret_cast<const int4*>(xr), x1 = *reinterpret_cast<const int4*>(xr + 16);
                    const float dx = xd[xrow * nb + b];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        int s = __dp4a(w0[r].x, x0.x, 0);
                        s = __dp4a(w0[r].y, x0.y, s);
                        s = __dp4a(w0[r].z, x0.z, s);
                        s = __dp4a(w0[r].w, x0.w, s);
                        s = __dp4a(w1[r].x, x1.x, s);
                        s = __dp4a(w1[r].y, x1.y, s);
                        s = __dp4a(w1[r].z, x1.z, s);
                        s = __dp4a(w1[r].w, x1.w, s);
                        acc[r][t] += (float)s * (d[r] * dx);
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) finish_rows<NT>(acc[r], n0 + r, out, t0, T, y, ldy, out_scale, softcap);
    }
    if (!waited) pdl_wait();  // a lane without blocks
}

// ---------------------------------------------------------------- one row per warp, Q6_K and Q8_0
// The sums of the two kernels above, row by row and with the wait ahead of everything: written without arrays over the rows, the compiler makes
// 40 and 58 us of 2048 x 11008 in Q6_K at 5 and 8 activation rows, where the kernel above takes 55 and 77.
__global__ void __launch_bounds__(GEMV_WARPS * 32) qgemv_q6k_row_kernel(const uint8_t* __restrict__ ql_p,
                                                                    const uint8_t* __restrict__ qh_p,
                                                                    const int8_t* __restrict__ sc_p,
                                                                    const __half* __restrict__ d_p, int nb, int out,
                                                                    const int8_t* xq,
                                                                    const float* xd, int T,
                                                                    float* __restrict__ y, int ldy, float out_scale,
                                                                    float softcap, Group grp) {
    pdl_trigger();
    pdl_wait();
    int n = blockIdx.x * GEMV_WARPS + (threadIdx.x >> 5);
    if (n >= out) return;
    int lane = threadIdx.x & 31;
    int part = lane & 7;
    int half = part >> 2;          // 128-weight half of the block
    int l0 = (part & 3) * 8;       // eight consecutive positions inside the half
    const int K = nb * 256;
    int64_t row_blk = ((int64_t)blockIdx.y * out + n) * nb;
    int t_first;
    group_range(grp, T, t_first, T);

    for (int t0 = t_first; t0 < T; t0 += NT_MAX) {
        float acc[NT_MAX];
#pragma unroll
        for (int t = 0; t < NT_MAX; ++t) acc[t] = 0.f;
        int rows = min(NT_MAX, T - t0);
        for (int ib = lane >> 3; ib < nb; ib += 4) {
            int64_t b = row_blk + ib;
            uint2 qa = *reinterpret_cast<const uint2*>(ql_p + b * 128 + half * 64 + l0);
            uint2 qb = *reinterpret_cast<const uint2*>(ql_p + b * 128 + half * 64 + 32 + l0);
            uint2 qhh = *reinterpret_cast<const uint2*>(qh_p + b * 64 + half * 32 + l0);
            const int8_t* sc = sc_p + b * 16 + half * 8 + (l0 >> 4);
            int s0 = sc[0], s1 = sc[2], s2 = sc[4], s3 = sc[6];
            float d = __half2float(d_p[b]);
            // four groups of eight 6-bit values, re-centred to [-32, 31]
            uint32_t g[4][2];
            g[0][0] = __vsub4((qa.x & 0x0F0F0F0Fu) | (((qhh.x >> 0) & 0x03030303u) << 4), 0x20202020u);
            g[0][1] = __vsub4((qa.y & 0x0F0F0F0Fu) | (((qhh.y >> 0) & 0x03030303u) << 4), 0x20202020u);
            g[1][0] = __vsub4((qb.x & 0x0F0F0F0Fu) | (((qhh.x >> 2) & 0x03030303u) << 4), 0x20202020u);
            g[1][1] = __vsub4((qb.y & 0x0F0F0F0Fu) | (((qhh.y >> 2) & 0x03030303u) << 4), 0x20202020u);
            g[2][0] = __vsub4(((qa.x >> 4) & 0x0F0F0F0Fu) | (((qhh.x >> 4) & 0x03030303u) << 4), 0x20202020u);
            g[2][1] = __vsub4(((qa.y >> 4) & 0x0F0F0F0Fu) | (((qhh.y >> 4) & 0x03030303u) << 4), 0x20202020u);
            g[3][0] = __vsub4(((qb.x >> 4) & 0x0F0F0F0Fu) | (((qhh.x >> 6) & 0x03030303u) << 4), 0x20202020u);
            g[3][1] = __vsub4(((qb.y >> 4) & 0x0F0F0F0Fu) | (((qhh.y >> 6) & 0x03030303u) << 4), 0x20202020u);
#pragma unroll
            for (int t = 0; t < NT_MAX; ++t) {
                if (t < rows) {
                    const int64_t xrow = src_of(grp, t0 + t);
                    const int8_t* xr = xq + xrow * K + ib * 256 + half * 128 + l0;
                    int2 x0 = *reinterpret_cast<const int2*>(xr);
                    int2 x1 = *reinterpret_cast<const int2*>(xr + 32);
                    int2 x2 = *reinterpret_cast<const int2*>(xr + 64);
                    int2 x3 = *reinterpret_cast<const int2*>(xr + 96);
                    int i0 = __dp4a((int)g[0][1], x0.y, __dp4a((int)g[0][0], x0.x, 0));
                    int i1 = __dp4a((int)g[1][1], x1.y, __dp4a((int)g[1][0], x1.x, 0));
                    int i2 = __dp4a((int)g[2][1], x2.y, __dp4a((int)g[2][0], x2.x, 0));
                    int i3 = __dp4a((int)g[3][1], x3.y, __dp4a((int)g[3][0], x3.x, 0));
                    int isum = s0 * i0 + s1 * i1 + s2 * i2 + s3 * i3;
                    acc[t] += xd[xrow * nb + ib] * (d * (float)isum);
                }
            }
        }
        finish_rows<NT_MAX>(acc, n, out, t0, T, y, ldy, out_scale, softcap);
    }
}

__global__ void __launch_bounds__(GEMV_WARPS * 32) qgemv_q80_row_kernel(const int8_t* __restrict__ qs_p,
                                                                    const __half* __restrict__ d_p, int K, int out,
                                                                    const int8_t* xq,
                                                                    const float* xd, int T,
                                                                    float* __restrict__ y, int ldy, float out_scale,
                                                                    float softcap, Group grp) {
    pdl_trigger();
    pdl_wait();
    int n = blockIdx.x * GEMV_WARPS + (threadIdx.x >> 5);
    if (n >= out) return;
    int lane = threadIdx.x & 31;
    int nb = K / 32;
    const int8_t* wq = qs_p + ((int64_t)blockIdx.y * out + n) * K;
    const __half* wd = d_p + ((int64_t)blockIdx.y * out + n) * nb;
    int t_first;
    group_range(grp, T, t_first, T);
    for (int t0 = t_first; t0 < T; t0 += NT_MAX) {
        float acc[NT_MAX];
#pragma unroll
        for (int t = 0; t < NT_MAX; ++t) acc[t] = 0.f;
        int rows = min(NT_MAX, T - t0);
        for (int b = lane; b < nb; b += 32) {
            int4 w0 = *reinterpret_cast<const int4*>(wq + b * 32);
            int4 w1 = *reinterpret_cast<const int4*>(wq + b * 32 + 16);
            float d = __half2float(wd[b]);
#pragma unroll
            for (int t = 0; t < NT_MAX; ++t) {
                if (t < rows) {
                    const int64_t xrow = src_of(grp, t0 + t);
                    const int8_t* xr = xq + xrow * K + b * 32;
                    int4 x0 = *reinterpret_cast<const int4*>(xr);
                    int4 x1 = *reinterpret_cast<const int4*>(xr + 16);
                    int s = __dp4a(w0.x, x0.x, 0);
                    s = __dp4a(w0.y, x0.y, s);
                    s = __dp4a(w0.z, x0.z, s);
                    s = __dp4a(w0.w, x0.w, s);
                    s = __dp4a(w1.x, x1.x, s);
                    s = __dp4a(w1.y, x1.y, s);
                    s = __dp4a(w1.z, x1.z, s);
                    s = __dp4a(w1.w, x1.w, s);
                    acc[t] += (float)s * (d * xd[xrow * nb + b]);
                }
            }
        }
        finish_rows<NT_MAX>(acc, n, out, t0, T, y, ldy, out_scale, softcap);
    }
}

// ---------------------------------------------------------------- F32 (router)
constexpr int F32_GEMV_ROWS = 8;
// y[t][n] = sum_k x[t][k] * W[n][k] for a small f32 matrix (the MoE router).  One warp per output n and run of
// F32_GEMV_ROWS rows of x (blockIdx.y): the rows' sums advance side by side, so a warp has a row's worth of independent
// loads in flight per step instead of one chain.  The sum of one (row, output) pair is always formed the same way -
// lane-strided partial sums in ascending k, then the warp tree - whatever the grid or the number of rows.
__global__ void __launch_bounds__(GEMV_WARPS * 32) f32_gemv_kernel(const float* __restrict__ W, int out, int in,
                                                                   const float* x, int T,
                                                                   float* __restrict__ y) {
    pdl_trigger();
    pdl_wait();
    int n = blockIdx.x * GEMV_WARPS + (threadIdx.x >> 5);
    if (n >= out) return;
    int lane = threadIdx.x & 31;
    const float* w = W + (int64_t)n * in;
    const int t0 = (int)blockIdx.y * F32_GEMV_ROWS;
    const int rows = min(F32_GEMV_ROWS, T - t0);
    const float* xr = x + (int64_t)t0 * in;
    float acc[F32_GEMV_ROWS];
#pragma unroll
    for (int r = 0; r < F32_GEMV_ROWS; ++r) acc[r] = 0.f;
    if (rows == F32_GEMV_ROWS) {
#pragma unroll 4
        for (int k = lane; k < in; k += 32) {
            const float wv = w[k];
#pragma unroll
            for (int r = 0; r < F32_GEMV_ROWS; ++r) acc[r] += xr[(int64_t)r * in + k] * wv;
        }
    } else {
        for (int k = lane; k < in; k += 32) {
            const float wv = w[k];
#pragma unroll
            for (int r = 0; r < F32_GEMV_ROWS; ++r)
                if (r < rows) acc[r] += xr[(int64_t)r * in + k] * wv;
        }
    }
#pragma unroll
    for (int r = 0; r < F32_GEMV_ROWS; ++r) {
        const float v = warp_sum(acc[r]);
        if (lane == 0 && r < rows) y[(int64_t)(t0 + r) * out + n] = v;
    }
}

// The same sums for many rows.  A CTA of 4 x 4 warps takes F32_TILE_OUT outputs and 4 R rows, a warp eight of the outputs with R of the rows: a
// value of x meets eight others and one of W meets R.  Both pass through shared memory, F32_TILE_K columns at a time and F32_TILE_STAGES - 1
// of these on their way, because what bounds the plain loads is that a warp can't have enough of them under way beside 64 sums; the tile
// is nearly square because the L2 then bounds the copies (1420 rows x 128 outputs x 2048: 64 us with eight rows and outputs per warp
// straight from the L1, 34 with tiles of 128 x 10, this 28; the multiply-adds take 11).
// A lane's columns and their order are those of the kernel above, columns behind the end are zeros: the same bits.
constexpr int F32_TILE_OUT = 32, F32_TILE_K = 64, F32_TILE_STAGES = 4, F32_TILE_WARPS = 16, F32_WARP_OUT = 8;
template <int R>
__global__ void __launch_bounds__(F32_TILE_WARPS * 32) f32_gemv_tile_kernel(const float* __restrict__ W, int out, int in, const float* x, int T,
                                                                            float* __restrict__ y) {
    extern __shared__ __align__(16) float f32_tile[];
    constexpr int ROWS = 4 * R, STAGE = (F32_TILE_OUT + ROWS) * F32_TILE_K, VECS = F32_TILE_K / 4;
    pdl_trigger();
    const int n0 = (int)blockIdx.x * F32_TILE_OUT, t0 = (int)blockIdx.y * ROWS, lane = threadIdx.x & 31, warp = (int)(threadIdx.x >> 5);
    const int wn = (warp & 3) * F32_WARP_OUT, wt = (warp >> 2) * R;   // this warp's first output and row of the tile
    const int chunks = (in + F32_TILE_K - 1) / F32_TILE_K;
    // rows and outputs behind the end repeat the last one and are not stored
    auto fetch = [&](int c, bool weights) {
        float* to = f32_tile + (c % F32_TILE_STAGES) * STAGE + (weights ? 0 : F32_TILE_OUT * F32_TILE_K);
        for (int i = threadIdx.x; i < (weights ? F32_TILE_OUT : ROWS) * VECS; i += F32_TILE_WARPS * 32) {
            const int row = i / VECS, k = c * F32_TILE_K + (i % VECS) * 4;
            const float* from = weights ? W + (int64_t)min(n0 + row, out - 1) * in : x + (int64_t)min(t0 + row, T - 1) * in;
            mc_cp_async16(to + i * 4, from + (k < in ? k : 0), k < in);
        }
    };
    for (int c = 0; c < F32_TILE_STAGES - 1 && c < chunks; ++c) fetch(c, true);   // the weights don't depend on the predecessor
    pdl_wait();
    for (int c = 0; c < F32_TILE_STAGES - 1; ++c) {
        if (c < chunks) fetch(c, false);
        mc_cp_commit();
    }
    float acc[R][F32_WARP_OUT] = {};
    for (int c = 0; c < chunks; ++c) {
        mc_cp_wait<F32_TILE_STAGES - 2>();
        __syncthreads();   // chunk c is here for everyone, and everyone is done with the one whose place the next takes
        if (c + F32_TILE_STAGES - 1 < chunks) { fetch(c + F32_TILE_STAGES - 1, true); fetch(c + F32_TILE_STAGES - 1, false); }
        mc_cp_commit();
        const float* ws = f32_tile + (c % F32_TILE_STAGES) * STAGE + wn * F32_TILE_K + lane;
        const float* xs = f32_tile + (c % F32_TILE_STAGES) * STAGE + (F32_TILE_OUT + wt) * F32_TILE_K + lane;
#pragma unroll
        for (int k = 0; k < F32_TILE_K; k += 32) {
            float wv[F32_WARP_OUT];
#pragma unroll
            for (int j = 0; j < F32_WARP_OUT; ++j) wv[j] = ws[j * F32_TILE_K + k];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float xv = xs[r * F32_TILE_K + k];
#pragma unroll
                for (int j = 0; j < F32_WARP_OUT; ++j) acc[r][j] += xv * wv[j];
            }
        }
    }
    mc_cp_wait<0>();
    // The warp's tree for eight outputs at once: each of its first three steps hands half of the sums to the other lane of the pair, the pairs
    // and with them the bits are those of eight trees.
    const int hi = lane >> 4, mid = (lane >> 3) & 1, lo = (lane >> 2) & 1;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        float a4[4], a2[2];
#pragma unroll
        for (int j = 0; j < 4; ++j) a4[j] = (hi ? acc[r][j + 4] : acc[r][j]) + __shfl_xor_sync(0xffffffffu, hi ? acc[r][j] : acc[r][j + 4], 16);
#pragma unroll
        for (int j = 0; j < 2; ++j) a2[j] = (mid ? a4[j + 2] : a4[j]) + __shfl_xor_sync(0xffffffffu, mid ? a4[j] : a4[j + 2], 8);
        float v = (lo ? a2[1] : a2[0]) + __shfl_xor_sync(0xffffffffu, lo ? a2[0] : a2[1], 4);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        v += __shfl_xor_sync(0xffffffffu, v, 1);
        const int n = n0 + wn + 4 * hi + 2 * mid + lo, t = t0 + wt + r;
        if ((lane & 3) == 0 && n < out && t < T) y[(int64_t)t * out + n] = v;
    }
}

template <int R>
void launch_f32_tile(const float* W, int out, int in, const float* x, int T, float* y, cudaStream_t s) {
    const size_t smem = (size_t)F32_TILE_STAGES * (F32_TILE_OUT + 4 * R) * F32_TILE_K * sizeof(float);
    ensure_dynamic_smem(reinterpret_cast<const void*>(&f32_gemv_tile_kernel<R>), smem);
    launch_pdl(f32_gemv_tile_kernel<R>, dim3((unsigned)((out + F32_TILE_OUT - 1) / F32_TILE_OUT), (unsigned)((T + 4 * R - 1) / (4 * R))), dim3(F32_TILE_WARPS * 32),
               smem, s, W, out, in, x, T, y);
}

}  // namespace

template <int NT, int R>
static void launch_qgemv_rows(const QWeight& W, const ActQ& x, int T, float* y, int ldy, float out_scale, float softcap, int experts, Group grp, cudaStream_t s) {
    dim3 grid((unsigned)((W.rows + GEMV_WARPS * R - 1) / (GEMV_WARPS * R)), (unsigned)experts);
    switch (W.type) {
        case QT_Q4_K:
            launch_pdl(qgemv_q4k_kernel<NT, R>, grid, dim3(GEMV_WARPS * 32), 0, s, (const uint8_t*)W.p0, (int)(W.cols / 256), (int)W.rows, x.qs, x.d, x.bsums, T, y, ldy, out_scale, softcap, grp);
            break;
        case QT_Q6_K:
            if constexpr (R == 1)
                launch_pdl(qgemv_q6k_row_kernel, grid, dim3(GEMV_WARPS * 32), 0, s, (const uint8_t*)W.p0, (const uint8_t*)W.p1, (const int8_t*)W.p2, (const __half*)W.p3, (int)(W.cols / 256), (int)W.rows,
                           x.qs, x.d, T, y, ldy, out_scale, softcap, grp);
            else
                launch_pdl(qgemv_q6k_kernel<NT, R>, grid, dim3(GEMV_WARPS * 32), 0, s, (const uint8_t*)W.p0, (const uint8_t*)W.p1, (const int8_t*)W.p2, (const __half*)W.p3,
                                                                      (int)(W.cols / 256), (int)W.rows, x.qs, x.d, T, y, ldy, out_scale, softcap, grp);
            break;
        case QT_Q8_0:
            if constexpr (R == 1 && NT > 1)
                launch_pdl(qgemv_q80_row_kernel, grid, dim3(GEMV_WARPS * 32), 0, s, (const int8_t*)W.p0, (const __half*)W.p1, (int)W.cols, (int)W.rows, x.qs, x.d, T, y, ldy, out_scale, softcap, grp);
            else
                launch_pdl(qgemv_q80_kernel<NT, R>, grid, dim3(GEMV_WARPS * 32), 0, s, (const int8_t*)W.p0, (const __half*)W.p1, (int)W.cols, (int)W.rows, x.qs, x.d, T, y, ldy, out_scale, softcap,
                                                                      grp);
            break;
        default:
            throw std::runtime_error("launch_qgemv: unsupported weight type");
    }
}

static void launch_qgemv_impl(const QWeight& W, const ActQ& x, int T, float* y, int ldy, float out_scale, float softcap,
                              int experts, Group grp, cudaStream_t s) {
    // several output rows per warp only while there are warps for every scheduler all the same
    const bool many = W.rows * experts >= 148 * 4 * 8 * 4;
    if (grp.offsets != nullptr || (!many && T > 4)) launch_qgemv_rows<NT_MAX, 1>(W, x, T, y, ldy, out_scale, softcap, experts, grp, s);
    else if (!many && T == 1) launch_qgemv_rows<1, 1>(W, x, T, y, ldy, out_scale, softcap, experts, grp, s);
    else if (!many) launch_qgemv_rows<4, 1>(W, x, T, y, ldy, out_scale, softcap, experts, grp, s);
    else if (T == 1) launch_qgemv_rows<1, 4>(W, x, T, y, ldy, out_scale, softcap, experts, grp, s);
    else if (T <= 4) launch_qgemv_rows<4, 2>(W, x, T, y, ldy, out_scale, softcap, experts, grp, s);
    else launch_qgemv_rows<NT_MAX, 2>(W, x, T, y, ldy, out_scale, softcap, experts, grp, s);
    MK_LAUNCH_CHECK();
}

void launch_qgemv(const QWeight& W, const ActQ& x, int T, float* y, int ldy, float out_scale, float softcap,
                  cudaStream_t s) {
    if (T <= 0 || W.rows <= 0) return;
    // a tile of sixteen rows for every SM: 2368 x 2048 10.2 us against 10.2 at two activation rows, 10.1 / 12.3 at four, 10.2 / 16.4 at
    // eight; 8192 x 2048 12.6 / 16.4, 12.5 / 20.7, 14.2 / 30.7; 32000 x 2048 21.4 / 30.7, 21.1 / 38.7, 22.5 / 69.7 (caches flushed)
    if (W.rows >= (int64_t)16 * device_sm_count() && q6k_rows_cover(W, x, T)) return launch_q6k_rows(W, x, T, y, ldy, out_scale, softcap, s);
    launch_qgemv_impl(W, x, T, y, ldy, out_scale, softcap, 1, Group{}, s);
}

void launch_qgemv_grouped(const QWeight& W, int experts, const int32_t* offsets, const int32_t* src_row, const ActQ& x,
                          float* y, int ldy, cudaStream_t s) {
    if (experts <= 0 || W.rows <= 0) return;
    Group g;
    g.offsets = offsets;
    g.src_row = src_row;
    launch_qgemv_impl(W, x, 0, y, ldy, 1.0f, 0.f, experts, g, s);
}

void launch_f32_gemv(const float* W, int out, int in, const float* x, int T, float* y, cudaStream_t s) {
    if (T <= 0) return;
    const unsigned runs = (unsigned)((T + F32_GEMV_ROWS - 1) / F32_GEMV_ROWS);
    // Tiles once an eighth of this kernel's warps would still give every SM's schedulers one; they take as few rows as keep the CTAs to one per SM,
    // 48 at most (the sums' registers).  A tile computes 32 outputs whatever there are: with 17 or more it is the faster one (24 us against 36 at
    // 4096 rows x 2048 columns), in its first round from 12 on (25 against 33); with 8 it takes 30 us instead of 19 (4800 rows), and behind
    // the first round 16 take 63 instead of 55 (8192 rows).
    const int64_t columns = (out + F32_TILE_OUT - 1) / F32_TILE_OUT, places = std::max<int64_t>(148 / columns, 1), rows = (T + places - 1) / places;
    const bool full = out > F32_TILE_OUT / 2 || (out >= 12 && rows <= 48);
    if (full && (int64_t)runs * out / 8 >= 148 * 4 && in % 4 == 0 && ((reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(x)) & 15) == 0) {
        if (rows <= 16) launch_f32_tile<4>(W, out, in, x, T, y, s);
        else if (rows <= 24) launch_f32_tile<6>(W, out, in, x, T, y, s);
        else if (rows <= 32) launch_f32_tile<8>(W, out, in, x, T, y, s);
        else if (rows <= 40) launch_f32_tile<10>(W, out, in, x, T, y, s);
        else launch_f32_tile<12>(W, out, in, x, T, y, s);
        MK_LAUNCH_CHECK();
        return;
    }
    dim3 grid((unsigned)((out + GEMV_WARPS - 1) / GEMV_WARPS), runs);
    launch_pdl(f32_gemv_kernel, grid, dim3(GEMV_WARPS * 32), 0, s, W, out, in, x, T, y);
    MK_LAUNCH_CHECK();
}

}  // namespace mk
