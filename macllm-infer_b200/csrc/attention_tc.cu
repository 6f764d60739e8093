// Tensor-core varlen paged GQA attention for f16 KV pools: the work lists of a tick and its one-token lanes (prefill chunks:
// attention_umma.cu).
//
// Same operator as attention.cu (the replacement of macllm_kernels::paged_attention_batch,
// crates/macllm-kernels/src/paged_attention.rs:614-709, and of dense_causal_attention,
// src/decoder.rs:4580-4670; visibility rule src/decoder.rs:4515-4532), restructured for bandwidth:
// one CTA reads the pages of one KV head for the whole query group, global -> shared with 16-byte cp.async; Q.K^T and P.V run
// on the tensor cores (mma.sync m16n8k16, f16 operands, f32 accumulators) and the online softmax stays in f32 registers.  The
// keys of a lane are shared out over the four warps of a CTA (warp-private cp.async rings, merge in shared memory) and,
// when few lanes have long histories, over several CTAs as well (scratch: unnormalised partial outputs +
// running max / sum per head, merged by the CTA that arrives last).  Queries are rounded to f16 once; K/V are read
// as stored.
#include "kernels.h"
#include "attention_tc.h"
#include "rope_head.cuh"
#include "quant_blocks.cuh"
#include <algorithm>

namespace mk {

namespace {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
    int bytes = valid ? 16 : 0;  // src-size 0 zero-fills the 16 destination bytes
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_half2(float x, float y) {
    __half2 h = __floats2half2_rn(x, y);
    return *reinterpret_cast<uint32_t*>(&h);
}

// The 8 x 8 tile of f16 numbers that a warp holds as (row lane / 4, columns 2 (lane % 4), + 1), transposed.
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t v) {
    uint32_t r;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}

// What f16 rounding left of two attention weights, as f16 numbers themselves.
__device__ __forceinline__ uint32_t pack_half2_rest(float x, float y, uint32_t rounded) {
    const float2 r = __half22float2(*reinterpret_cast<const __half2*>(&rounded));
    return pack_half2(x - r.x, y - r.y);
}

// cap * tanh(v / cap) as cap - 2 cap / (1 + exp(2 v / cap)): off by a few 1e-7 of the cap, which is what a score's own rounding costs.
__device__ __forceinline__ float capped(float v, float cap, float two_over_cap) {
    return cap - __fdividef(2.0f * cap, 1.0f + __expf(fminf(v * two_over_cap, 80.0f)));
}

// 1 / denominator of a row with running maximum m and sum l of exp(score - m), when the softmax also counts exp(sink).
__device__ __forceinline__ float sink_scale(float m, float l, float sink) {
    const float top = fmaxf(m, sink), f = __expf(m - top);
    return f / (l * f + __expf(sink - top));
}

// One-token lanes.  Work item = entries[blockIdx.x] = (lane, share, n_shares) x KV head.  The four warps of the
// CTA take the 16-key tiles of the share round-robin, each through its own ring of cp.async stages (no
// block-wide barrier inside the loop), keep their own running max / sum / output, and merge through shared
// memory at the end.  n_shares == 1: the CTA writes the normalised output.  Otherwise it writes its unnormalised
// partial, and the CTA that arrives last at the lane's counter merges the shares.
// A KV head has at most eight query heads, so the heads are the N of the products and keys (scores) or dimensions (outputs) the M: S^T = K Q^T, O^T = V^T P^T.
// With the heads as M half of every product and accumulator was zeros.  A lane then holds two heads of its tile's keys g and g + 8; the weights turn
// into the operand of the second product by two 8 x 8 transposes.
// History does not wait for the predecessor: every key but the newest was written before this tick's first kernel, so the first tiles are
// requested ahead of pdl_wait.  THREADS: while the CTAs have an SM each, four more warps help with what is not a walk - a CTA has up to ten
// head vectors to prepare, whose shares come from the L2 one after the other (4 lanes of 300 keys, 32 heads of 64 over 4: 17 -> 11 us a launch, one
// lane of 200, 16 heads of 128 over 4: 13 -> 9); with two CTAs on an SM the registers are worth more (64 lanes: 27 us, 37 with the help).
template <int D, int STAGES, bool EXACT, int THREADS, int WALKERS>
__global__ void __launch_bounds__(THREADS) attn_decode_kernel(AttnTcArgs a) {
    constexpr int DP = D + 8;
    constexpr int KT = 16;
    constexpr int NT_O = D / 16;      // tiles of 16 dimensions
    constexpr int OP = D + 4;         // floats between heads of a warp's partial result: a fragment's lanes hit all banks
    constexpr int CHUNKS = D / 8;
    constexpr int RING_HALVES = STAGES * 2 * KT * DP;  // per warp: STAGES x (K tile + V tile)
    static_assert(RING_HALVES * 2 >= 8 * OP * 4 + 8 * 2 * 4, "a warp's ring must hold its partial result");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __half* Qs = reinterpret_cast<__half*>(smem_raw);  // [16][DP]
    __half* rings = Qs + 16 * DP;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int gid = lane >> 2, tq = lane & 3;
    const int kvh = blockIdx.y;
    const int g = a.q_heads / a.kv_heads;
    const float two_over_cap = a.softcap != 0.f ? 2.0f / a.softcap : 0.f;
    // one 32-byte record per work item, so that nothing but the block table and the queries is a dependent load
    const int4 e0 = reinterpret_cast<const int4*>(a.entries)[2 * blockIdx.x];
    const int4 e1 = reinterpret_cast<const int4*>(a.entries)[2 * blockIdx.x + 1];
    const int lane_id = e0.x, split = e0.y, n_splits = e0.z, start_pos = e0.w, table_off = e1.x, q_off = e1.y, first_entry = e1.z;
    const int ldq = a.ldq > 0 ? a.ldq : a.q_heads * D;

    // Rows straight from the projection's output (see AttnTcArgs::fused_rope): whole heads per warp, the head vectors staged
    // in f32; the group's query heads, and in the CTA that walks the lane's newest keys also the new K and V rows, which
    // reach the pool before any tile is requested (block-wide barrier below).
    constexpr int WARPS = THREADS / 32, MAX_HEADS = (10 + WARPS - 1) / WARPS;   // of a warp
    __shared__ __align__(16) float head_stage[WARPS * MAX_HEADS][D];
    RopeAngles angles = {};
    if (a.fused_rope) angles = rope_angles(a.rk, start_pos, lane);
    auto put_head = [&](int h, const float* xs) {  // head h of the group's query heads, then the new K and V row
        if (h < g) {
            for (int i = lane; i < D; i += 32) Qs[h * DP + i] = __float2half_rn(xs[i]);
        } else {
            const int64_t blk = a.tables[table_off + (start_pos >> a.bt_shift)];
            const int64_t base = ((kv_page_index(blk, a.layer, a.layers, a.pool_blocks) * a.kv_heads + kvh) * a.block_tokens +
                                  (start_pos & (a.block_tokens - 1))) * (int64_t)D;
            __half* pool = reinterpret_cast<__half*>(h == g ? a.rk.k_pool : a.rk.v_pool);
            for (int i = lane; i < D; i += 32) pool[base + i] = __float2half_rn(xs[i]);
        }
    };
    auto prepare_heads = [&](int n_heads) {
        const float* src[MAX_HEADS];
        float* xs[MAX_HEADS];
        int parts[MAX_HEADS];
        int64_t stride[MAX_HEADS];
        uintptr_t place = 0;
        int n = 0;
#pragma unroll
        for (int k = 0; k < MAX_HEADS; ++k) {
            const int h = warp + k * WARPS, kind = h < g ? 0 : (h == g ? 1 : 2);
            xs[k] = head_stage[warp + k * WARPS];
            src[k] = nullptr;
            parts[k] = kind == 2 ? a.rk.v_splits : a.rk.qk_splits;
            stride[k] = kind == 2 ? a.rk.v_split_stride : a.rk.qk_split_stride;
            if (h < n_heads) {
                src[k] = rope_head_source(a.rk, kind, kind == 0 ? kvh * g + h : kvh, q_off);
                place |= reinterpret_cast<uintptr_t>(src[k]) | (uintptr_t)(stride[k] * 4);
                n = k + 1;
            }
        }
        const bool whole = a.rk.d == D && rope_head_width(a.rk, 2) == D;
        if (whole && D % 128 == 0 && (place & 15) == 0) rope_sum_heads<float4>(src, parts, stride, n, D, xs, lane);
        else if (whole && (place & 7) == 0) rope_sum_heads<float2>(src, parts, stride, n, D, xs, lane);
        else
            for (int k = 0; k < n; ++k) {
                const int kind = warp + k * WARPS < g ? 0 : (warp + k * WARPS == g ? 1 : 2);
                rope_sum_shares<float>(src[k], parts[k], stride[k], rope_head_width(a.rk, kind), xs[k], lane);
            }
#pragma unroll
        for (int k = 0; k < MAX_HEADS; ++k) {
            if (k >= n) break;
            const int h = warp + k * WARPS, kind = h < g ? 0 : (h == g ? 1 : 2);
            rope_head_finish(a.rk, kind, kind == 0 ? kvh * g + h : kvh, angles, xs[k], lane);
            put_head(h, xs[k]);
        }
    };
    const int p = start_pos;  // the query's position
    int k_lo = attention_first_key(p, a.window, a.chunk);
    int k_hi = p + 1;
    {
        int len = k_hi - k_lo;
        int chunk = ((len + n_splits - 1) / n_splits + 15) / 16 * 16;
        k_lo = k_lo + split * chunk;
        k_hi = min(k_hi, k_lo + chunk);
    }
    const int k_begin = k_lo / 16 * 16;
    const int n_tiles = k_hi > k_begin ? (k_hi - k_begin + KT - 1) / KT : 0;
    const int my_tiles = warp < WALKERS && n_tiles > warp ? (n_tiles - warp + WALKERS - 1) / WALKERS : 0;  // tiles warp, warp + WALKERS, ...

    const __half* kp = reinterpret_cast<const __half*>(a.k_pool);
    const __half* vp = reinterpret_cast<const __half*>(a.v_pool);
    __half* ring = rings + (warp % WALKERS) * RING_HALVES;
    uint32_t tile_blk = 0;
    auto load_tile = [&](int i) {  // the warp's i-th tile into stage i % STAGES (called with i = 0, 1, 2, ... in order)
        __half* kd = ring + (i % STAGES) * 2 * KT * DP;
        __half* vd = kd + KT * DP;
        // 16 keys starting at a multiple of 16 lie in one page (block_tokens is a multiple of 16): one table
        // lookup, then the tile is one contiguous run of 16 * D halves in each pool
        const int pos0 = k_begin + (warp + WALKERS * i) * KT;
        // the page ids of the warp's next 32 tiles sit in the lanes (fetched together, off the critical path)
        if ((i & 31) == 0) {
            const int t = i + lane;
            tile_blk = t < my_tiles ? a.tables[table_off + ((k_begin + (warp + WALKERS * t) * KT) >> a.bt_shift)] : 0u;
        }
        const int64_t blk = __shfl_sync(0xffffffffu, tile_blk, i & 31);
        const int64_t src0 = ((kv_page_index(blk, a.layer, a.layers, a.pool_blocks) * a.kv_heads + kvh) * a.block_tokens +
                              (pos0 & (a.block_tokens - 1))) * (int64_t)D;
        const int n_valid = k_hi - pos0;  // keys of the tile inside the share
#pragma unroll
        for (int j = lane; j < KT * CHUNKS; j += 32) {
            const int key = j / CHUNKS, c = (j % CHUNKS) * 8;
            const bool valid = key < n_valid;
            const int64_t src = valid ? src0 + (int64_t)j * 8 : 0;
            cp_async16(kd + key * DP + c, kp + src, valid);
            cp_async16(vd + key * DP + c, vp + src, valid);
        }
    };

    // tiles that may travel before the predecessor is done: all but the one with the newest key
    const int old_tiles = my_tiles - (my_tiles > 0 && k_begin + (warp + WALKERS * (my_tiles - 1)) * KT + KT > p ? 1 : 0);
    const int early = min(old_tiles, STAGES - 1);
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i)
        if (i < early) {
            load_tile(i);
            cp_async_commit();
        }
    // rows of the operand without a query head
    for (int i = tid; i < (8 - g) * CHUNKS; i += THREADS) *reinterpret_cast<uint4*>(Qs + (g + i / CHUNKS) * DP + (i % CHUNKS) * 8) = make_uint4(0u, 0u, 0u, 0u);
    pdl_wait();
    if (a.fused_rope) {
        prepare_heads(g + (split == n_splits - 1 ? 2 : 0));
    } else {
        // the group's query heads -> rows 0..g-1 of the operand
        for (int i = tid; i < g * CHUNKS; i += THREADS) {
            const int item = i / CHUNKS, c = (i - item * CHUNKS) * 8;
            const float* src = a.q + (int64_t)q_off * ldq + (kvh * g + item) * D + c;
            const float4 x0 = *reinterpret_cast<const float4*>(src), x1 = *reinterpret_cast<const float4*>(src + 4);
            const __half2 h[4] = {__floats2half2_rn(x0.x, x0.y), __floats2half2_rn(x0.z, x0.w), __floats2half2_rn(x1.x, x1.y), __floats2half2_rn(x1.z, x1.w)};
            *reinterpret_cast<uint4*>(Qs + item * DP + c) = *reinterpret_cast<const uint4*>(h);
        }
    }
    __syncthreads();  // the queries, and the new K / V rows for every tile load that follows
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i)
        if (i >= early) {
            if (i < my_tiles) load_tile(i);
            cp_async_commit();
        }
    pdl_trigger();

    float o_acc[NT_O][4];   // (dimension gid, heads 2 tq, 2 tq + 1), (dimension gid + 8, the same)
#pragma unroll
    for (int j = 0; j < NT_O; ++j) o_acc[j][0] = o_acc[j][1] = o_acc[j][2] = o_acc[j][3] = 0.f;
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};   // of the two heads; the sum counts this lane's keys only
    constexpr bool Q_IN_REGS = D <= 128;
    uint32_t qf[Q_IN_REGS ? D / 32 : 1][4];
    const __half* q_at = Qs + (lane & 7) * DP + (lane >> 3) * 8;
    if (Q_IN_REGS) {
#pragma unroll
        for (int kk = 0; kk < D / 32; ++kk) ldmatrix_x4(qf[Q_IN_REGS ? kk : 0], q_at + kk * 32);
    }

    for (int i = 0; i < my_tiles; ++i) {
        if (i + STAGES - 1 < my_tiles) load_tile(i + STAGES - 1);
        cp_async_commit();
        cp_async_wait<STAGES - 1>();
        __syncwarp();
        const __half* kt = ring + (i % STAGES) * 2 * KT * DP;
        const __half* vt = kt + KT * DP;

        float sc[4], even[4] = {0.f, 0.f, 0.f, 0.f}, odd[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int kk = 0; kk < D / 32; ++kk) {
            uint32_t a0[4], a1[4], bf[4];
            if (!Q_IN_REGS) ldmatrix_x4(bf, q_at + kk * 32);
            ldmatrix_x4(a0, kt + (lane & 15) * DP + kk * 32 + (lane >> 4) * 8);
            ldmatrix_x4(a1, kt + (lane & 15) * DP + kk * 32 + 16 + (lane >> 4) * 8);
            mma16816(even, a0, Q_IN_REGS ? qf[Q_IN_REGS ? kk : 0][0] : bf[0], Q_IN_REGS ? qf[Q_IN_REGS ? kk : 0][1] : bf[1]);
            mma16816(odd, a1, Q_IN_REGS ? qf[Q_IN_REGS ? kk : 0][2] : bf[2], Q_IN_REGS ? qf[Q_IN_REGS ? kk : 0][3] : bf[3]);
        }
        const int tile_pos = k_begin + (warp + WALKERS * i) * KT;
        // a tile that lies wholly inside the share needs no masking (heads that do not exist hold zeros and are never stored)
        const bool full_tile = tile_pos >= k_lo && tile_pos + KT <= k_hi;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int pos = tile_pos + gid + 8 * (e >> 1);
            float v = (even[e] + odd[e]) * a.scale;
            if (a.softcap != 0.f) v = capped(v, a.softcap, two_over_cap);
            sc[e] = full_tile || (pos >= k_lo && pos < k_hi) ? v : -INFINITY;  // k_lo / k_hi carry causality and the window
        }
        float alpha[2], m_use[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float top = fmaxf(sc[h], sc[2 + h]);
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 4));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 8));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 16));
            const float m_new = fmaxf(m_run[h], top);
            m_use[h] = m_new == -INFINITY ? 0.f : m_new;
            alpha[h] = m_run[h] == -INFINITY ? 0.f : __expf(m_run[h] - m_use[h]);
            m_run[h] = m_new;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[e] = sc[e] == -INFINITY ? 0.f : __expf(sc[e] - m_use[e & 1]);
        l_run[0] = l_run[0] * alpha[0] + (sc[0] + sc[2]);
        l_run[1] = l_run[1] * alpha[1] + (sc[1] + sc[3]);
#pragma unroll
        for (int j = 0; j < NT_O; ++j) {
            o_acc[j][0] *= alpha[0];
            o_acc[j][1] *= alpha[1];
            o_acc[j][2] *= alpha[0];
            o_acc[j][3] *= alpha[1];
        }
        const uint32_t p0 = pack_half2(sc[0], sc[1]), p1 = pack_half2(sc[2], sc[3]);
        const uint32_t b0 = transpose_8x8(p0), b1 = transpose_8x8(p1);
        uint32_t r0 = 0u, r1 = 0u;
        if constexpr (EXACT) {
            r0 = transpose_8x8(pack_half2_rest(sc[0], sc[1], p0));
            r1 = transpose_8x8(pack_half2_rest(sc[2], sc[3], p1));
        }
#pragma unroll
        for (int j = 0; j < NT_O; ++j) {
            uint32_t af[4];
            ldmatrix_x4_trans(af, vt + ((lane >> 4) * 8 + (lane & 7)) * DP + j * 16 + ((lane >> 3) & 1) * 8);
            mma16816(o_acc[j], af, b0, b1);
            if constexpr (EXACT) mma16816(o_acc[j], af, r0, r1);
        }
        __syncwarp();  // the stage is refilled by the next iteration's load
    }
    cp_async_wait<0>();
    __syncwarp();

    // each warp leaves (max, sum, output) of its live heads in its own ring, then everyone merges
    float* w_o = reinterpret_cast<float*>(ring);            // [8][OP]
    float* w_ml = w_o + 8 * OP;                              // [8][2]
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 4);
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 8);
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 16);
        const int item = 2 * tq + h;
        if (item >= g || warp >= WALKERS) continue;
#pragma unroll
        for (int j = 0; j < NT_O; ++j) {
            w_o[item * OP + j * 16 + gid] = o_acc[j][h];
            w_o[item * OP + j * 16 + gid + 8] = o_acc[j][2 + h];
        }
        if (gid == 0) {
            w_ml[item * 2] = m_run[h];
            w_ml[item * 2 + 1] = l_run[h];
        }
    }
    __syncthreads();
    const int64_t slot = ((int64_t)blockIdx.x * a.kv_heads + kvh) * 16;
    // merged, normalised outputs of this (lane, KV head): g * D consecutive values of the lane's output row, eight per thread (one head's)
    auto finish = [&](auto&& values_of) {
        const int64_t row = q_off;
        const int col0 = kvh * g * D;
        for (int i8 = tid; i8 < g * D / 8; i8 += THREADS) {
            float v[8];
            values_of(i8 * 8, v);
            if (a.out != nullptr) store8(a.out + row * a.q_heads * D + col0 + i8 * 8, v);
            // one warp per 256-wide group (g * D is a multiple of 256 where the rows are quantised)
            if (a.qout.qs != nullptr) quant_group(v, lane, a.qkind, a.qout, row, a.q_heads * D, col0 / 256 + (i8 >> 5));
            else if (a.out_h != nullptr) {
                __half2 h[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
                *reinterpret_cast<uint4*>(a.out_h + row * a.q_heads * D + col0 + i8 * 8) = *reinterpret_cast<const uint4*>(h);
            }
        }
    };
    // the walkers' sums of eight values of one head, as one walker's
    auto merged_local = [&](int idx, float (&o)[8], float& m_out, float& l_out) {
        const int item = idx / D, c = idx - item * D;
        const float* first = reinterpret_cast<const float*>(rings);
        constexpr int STEP = RING_HALVES / 2;   // floats between walkers
        float mw[WALKERS], m = -INFINITY, l = 0.f;
#pragma unroll
        for (int w = 0; w < WALKERS; ++w) {
            mw[w] = first[w * STEP + 8 * OP + item * 2];
            m = fmaxf(m, mw[w]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = 0.f;
#pragma unroll
        for (int w = 0; w < WALKERS; ++w) {
            const float f = mw[w] == -INFINITY ? 0.f : __expf(mw[w] - m);   // a walker without keys left zeros
            float x[8];
            load8(first + w * STEP + item * OP + c, x);
            l += first[w * STEP + 8 * OP + item * 2 + 1] * f;
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] += x[i] * f;
        }
        m_out = m;
        l_out = l;
    };
    auto normalise = [&](int idx, float (&o)[8], float m, float l) {
        if (a.sink != nullptr) {
            const float s = sink_scale(m, l, a.sink[kvh * g + idx / D]);
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] *= s;
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = o[i] / l;
        }
    };
    if (n_splits == 1) {
        finish([&](int idx, float (&o)[8]) {
            float m, l;
            merged_local(idx, o, m, l);
            normalise(idx, o, m, l);
        });
    } else {
        for (int i8 = tid; i8 < g * D / 8; i8 += THREADS) {
            const int idx = i8 * 8, item = idx / D, c = idx - item * D;
            float o[8], m, l;
            merged_local(idx, o, m, l);
            store8(a.part_o + (slot + item) * D + c, o);
            if (c == 0) {
                a.part_ml[(slot + item) * 2] = m;
                a.part_ml[(slot + item) * 2 + 1] = l;
            }
        }
        // The lane's keys were shared out over several CTAs: the CTA that arrives last at the lane's counter adds
        // the shares in share order (so the result does not depend on which one that is) and resets the counter.
        __shared__ int s_last;
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            int prev = atomicAdd(&a.counters[lane_id * a.kv_heads + kvh], 1);
            s_last = prev == n_splits - 1 ? 1 : 0;
            if (prev == n_splits - 1) a.counters[lane_id * a.kv_heads + kvh] = 0;
        }
        __syncthreads();
        if (s_last) {
            __threadfence();
            finish([&](int idx, float (&o)[8]) {
                const int item = idx / D, c = idx - item * D;
                const int64_t first = ((int64_t)first_entry * a.kv_heads + kvh) * 16 + item, step = (int64_t)a.kv_heads * 16;
                float m = -INFINITY, l = 0.f;
                for (int sp = 0; sp < n_splits; ++sp) m = fmaxf(m, __ldcg(a.part_ml + (first + sp * step) * 2));
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = 0.f;
#pragma unroll 4
                for (int sp = 0; sp < n_splits; ++sp) {
                    const int64_t ps = first + sp * step;
                    const float ms = __ldcg(a.part_ml + ps * 2), f = ms == -INFINITY ? 0.f : __expf(ms - m);
                    const float4 x = __ldcg(reinterpret_cast<const float4*>(a.part_o + ps * D + c)), y = __ldcg(reinterpret_cast<const float4*>(a.part_o + ps * D + c + 4));
                    l += __ldcg(a.part_ml + ps * 2 + 1) * f;
                    o[0] += x.x * f; o[1] += x.y * f; o[2] += x.z * f; o[3] += x.w * f;
                    o[4] += y.x * f; o[5] += y.y * f; o[6] += y.z * f; o[7] += y.w * f;
                }
                normalise(idx, o, m, l);
            });
        }
    }
}

// Merge the key shares of one-token lanes: grid (decode lane, kv head), one warp per query head of the group.
__global__ void attn_combine_kernel(AttnTcArgs a, int D) {
    pdl_trigger();
    pdl_wait();
    const int dl = blockIdx.x, kvh = blockIdx.y;
    const int lane_id = a.dec_lanes[3 * dl], first = a.dec_lanes[3 * dl + 1], n_splits = a.dec_lanes[3 * dl + 2];
    const int g = a.q_heads / a.kv_heads;
    const int hq = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (hq >= g) return;
    float m = -INFINITY;
    for (int s = 0; s < n_splits; ++s) m = fmaxf(m, a.part_ml[(((int64_t)(first + s) * a.kv_heads + kvh) * 16 + hq) * 2]);
    float l = 0.f;
    for (int s = 0; s < n_splits; ++s) {
        const float* ml = a.part_ml + (((int64_t)(first + s) * a.kv_heads + kvh) * 16 + hq) * 2;
        if (ml[0] != -INFINITY) l += ml[1] * __expf(ml[0] - m);
    }
    const int q_off = a.cu_seqlens[lane_id];
    float* o = a.out + (int64_t)q_off * a.q_heads * D + (kvh * g + hq) * D;
    for (int c = lane; c < D; c += 32) {
        float acc = 0.f;
        for (int s = 0; s < n_splits; ++s) {
            int64_t slot = ((int64_t)(first + s) * a.kv_heads + kvh) * 16 + hq;
            float ms = a.part_ml[slot * 2];
            if (ms != -INFINITY) acc += a.part_o[slot * D + c] * __expf(ms - m);
        }
        o[c] = acc / l;
    }
}

template <int D, bool EXACT>
void launch_for_dim(const AttnTcArgs& a, cudaStream_t s) {
    if (a.n_entries > 0) {
        constexpr int STAGES = D >= 256 ? 2 : 3;
        constexpr int ALONE_WALKERS = D >= 256 ? 4 : 8;
        auto smem = [](int walkers) { return (size_t)(16 + walkers * STAGES * 2 * 16) * (D + 8) * sizeof(__half); };
        dim3 grid((unsigned)a.n_entries, (unsigned)a.kv_heads);
        const bool alone = a.n_entries * a.kv_heads <= kPlanSms;
        auto* kernel = alone ? attn_decode_kernel<D, STAGES, EXACT, 256, ALONE_WALKERS> : attn_decode_kernel<D, STAGES, EXACT, 128, 4>;
        const size_t bytes = smem(alone ? ALONE_WALKERS : 4);
        ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), bytes);
        launch_pdl(kernel, grid, dim3(alone ? 256 : 128), bytes, s, a);
        MK_LAUNCH_CHECK();
    }
    if (a.n_dec_lanes > 0) {  // lanes whose keys were shared out over several CTAs
        dim3 grid((unsigned)a.n_dec_lanes, (unsigned)a.kv_heads);
        launch_pdl(attn_combine_kernel, grid, dim3(32 * (a.q_heads / a.kv_heads)), 0, s, a, (int)D);
        MK_LAUNCH_CHECK();
    }
}

}  // namespace

bool attention_tc_supported(int q_heads, int kv_heads, int head_dim, int block_tokens, bool kv_f16) {
    int g = kv_heads > 0 ? q_heads / kv_heads : 0;
    if (block_tokens < 16 || (block_tokens & (block_tokens - 1)) != 0) return false;  // pages hold whole 16-key tiles
    return kv_f16 && (head_dim == 64 || head_dim == 128 || head_dim == 256) && (g == 1 || g == 2 || g == 4 || g == 8) &&
           q_heads == g * kv_heads;
}

int attention_tc_prefill_width(int q_heads, int kv_heads, int dim, int vdim, int block_tokens) {
    if (!attention_tc_supported(q_heads, kv_heads, 64, block_tokens, true)) return 0;
    const int need = std::max(dim, vdim);
    for (int d : {64, 128, 192, 256})
        if (need <= d && (d != 192 || vdim <= 128)) return d;
    return 0;
}

int attention_tc_tile_rows(int q_heads, int kv_heads) { return kAttnItems / (q_heads / kv_heads); }

int attention_tc_max_entries(int lanes, int kv_heads) { return std::max(lanes + lanes / 2, kAttnTargetCtas / std::max(1, kv_heads)) + 1; }

void plan_attention_tc(const int32_t* start_pos, const int32_t* n_tokens, const int32_t* n_blocks, int lanes, int q_heads,
                       int kv_heads, AttnTcPlan& plan, int chunk, int window) {
    auto visible = [&](int i) { return start_pos[i] + 1 - attention_first_key(start_pos[i], window, chunk); };  // keys of a one-token lane
    plan.tiles.clear();
    plan.entries.clear();
    plan.dec_lanes.clear();
    const int tile_rows = attention_tc_tile_rows(q_heads, kv_heads);
    struct Walk { int keys, lane, row0; };
    std::vector<Walk> walks;
    // One-token lanes: every CTA should walk about the same number of keys, and all CTAs should fit on the GPU at
    // once.  Share size = total keys / CTA slots per KV head, raised until the shares of all lanes fit.
    int n_dec = 0;
    int64_t total_keys = 0;
    for (int i = 0; i < lanes; ++i)
        if (n_tokens[i] == 1) { ++n_dec; total_keys += visible(i); }
    // Once the lanes alone give every SM a CTA, sharing keys out only adds merge work and repeated query preparation
    // (measured at 64 lanes x 4 KV heads with histories within twice their mean: +1.4 % on the whole benchmark
    // without shares).  Then only a lane more than twice as long as the mean is cut, so that one long history among
    // many short ones does not set the length of the launch.
    const bool filled = n_dec * kv_heads >= kPlanSms;
    const int slots = filled ? n_dec + n_dec / 2 : std::max(n_dec, kAttnTargetCtas / std::max(1, kv_heads));
    int share = (int)std::max<int64_t>(kAttnMinSplitKeys, filled ? 2 * (total_keys / std::max(1, n_dec)) : (total_keys + slots - 1) / std::max(1, slots));
    share = (share + 63) / 64 * 64;
    auto shares_of = [&](int ctx) { return std::max(1, std::min(kAttnMaxSplits, (ctx + share - 1) / share)); };
    for (;;) {
        int64_t ctas = 0;
        for (int i = 0; i < lanes; ++i)
            if (n_tokens[i] == 1) ctas += shares_of(visible(i));
        if (ctas <= slots || share > (1 << 20)) break;
        share += 64;
    }
    int q_off = 0, table_off = 0;
    for (int i = 0; i < lanes; q_off += n_tokens[i], table_off += n_blocks[i], ++i) {
        if (n_tokens[i] == 1) {
            const int splits = shares_of(visible(i));
            const int first = plan.n_entries();
            for (int sidx = 0; sidx < splits; ++sidx) {
                const int32_t rec[8] = {i, sidx, splits, start_pos[i], table_off, q_off, first, 0};
                plan.entries.insert(plan.entries.end(), rec, rec + 8);
            }
        } else {
            for (int r0 = 0; r0 < n_tokens[i]; r0 += tile_rows) {
                const int first = start_pos[i] + r0, last = start_pos[i] + std::min(r0 + tile_rows, n_tokens[i]) - 1;
                walks.push_back({last + 1 - attention_first_key(first, window, chunk), i, r0});
            }
        }
    }
    // longest walks first: the last round of CTAs is then made of short ones
    std::stable_sort(walks.begin(), walks.end(), [](const Walk& x, const Walk& y) { return x.keys > y.keys; });
    for (const Walk& w : walks) {
        plan.tiles.push_back(w.lane);
        plan.tiles.push_back(w.row0);
    }
}

int launch_paged_attention_tc(const AttnTcArgs& a_in, cudaStream_t s) {
    AttnTcArgs a = a_in;
    const bool prefill_192 = a.d == 192 && a.n_entries == 0 && a.n_dec_lanes == 0 && a.dv > 0 && a.dv <= 128 && a.exact_weights &&
                             attention_tc_prefill_width(a.q_heads, a.kv_heads, 192, a.dv, a.block_tokens) == 192;
    if (!prefill_192 && !attention_tc_supported(a.q_heads, a.kv_heads, a.d, a.block_tokens, true))
        throw std::runtime_error("launch_paged_attention_tc: unsupported shape");
    if (a.rot_dims > 0 && (a.n_entries > 0 || a.rot_from % 8 != 0 || a.cos_t == nullptr || a.sin_t == nullptr))
        throw std::runtime_error("launch_paged_attention_tc: queries turn on their way into prefill tiles only");
    if (a.out == nullptr && a.out_h == nullptr && a.qout.qs == nullptr) throw std::runtime_error("launch_paged_attention_tc: no output");
    if (a.sink != nullptr && a.n_dec_lanes > 0) throw std::runtime_error("launch_paged_attention_tc: the separate merge pass knows no sink");
    if (a.out == nullptr && a.n_dec_lanes > 0) throw std::runtime_error("launch_paged_attention_tc: the separate merge pass writes f32 rows");
    a.bt_shift = 0;
    while ((1 << a.bt_shift) < a.block_tokens) ++a.bt_shift;
    if (a.n_tiles > 0) launch_attention_umma(a, s);
    switch (a.d) {
        case 64: a.exact_weights ? launch_for_dim<64, true>(a, s) : launch_for_dim<64, false>(a, s); break;
        case 128: a.exact_weights ? launch_for_dim<128, true>(a, s) : launch_for_dim<128, false>(a, s); break;
        case 192: break;
        case 256: a.exact_weights ? launch_for_dim<256, true>(a, s) : launch_for_dim<256, false>(a, s); break;
        default: throw std::runtime_error("launch_paged_attention_tc: unsupported head_dim");
    }
    return (a.n_tiles > 0 ? 1 : 0) + (a.n_entries > 0 ? 1 : 0) + (a.n_dec_lanes > 0 ? 1 : 0);
}

}  // namespace mk
