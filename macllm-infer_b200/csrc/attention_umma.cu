// Prefill chunks of paged GQA attention on the fifth-generation tensor cores (see attention_tc.h for the operator).
//
// A CTA owns 128 (query row, query head) items of one KV head and walks the keys they see in tiles of 64.  Warp 4 brings the
// pages of a tile into shared memory with TMA (one box of 16 keys x 64 columns per page and panel, 128-byte swizzle).  Warp 5
// issues the products: scores Q K^T (128 x 64, f32) into one of two areas of tensor memory, and O += P V with P as the A operand
// in tensor memory, over the scores it was made from, and V read with the keys as the reduction.  Warps 0 - 3 hold one item per
// thread: a row of scores comes in one piece, so maximum and sum need no exchange; P goes back as f16 (EXACT: as the f16 number
// and the f16 rounding of what it left, two products).  The scores of the next tile are made while this tile's softmax runs.
// The running maximum follows only when a tile exceeds it by more than kSlack (weights stay below 2^kSlack, well inside f16), so
// the accumulators in tensor memory are hardly ever rescaled (conditional rescaling, as the authors of FlashAttention-4 describe it).  Every wait
// is bounded.
//
// What bounds it: exponentials (16 per clock and SM; a soft cap takes two more per score) and the tensor pipe are about level at head size
// 128.  Heads of up to 128 run two CTAs per SM (96 KB of shared memory, 256 columns of tensor memory each), so that one's softmax runs under
// the other's products; wider ones take the SM to themselves.
// Measured on a B200 beside the kernel before it (mma.sync, 64 items per CTA): 16 heads of 256 over 8 KV heads, ticks of 2048 tokens of
// prompts of up to 8192, capped scores: 545 -> 144 us per launch; 32 heads of 128 over 8, 512-token chunks behind a prefix of 2048:
// 236 -> 53 us; 16 heads of 128 over 4, prompts of 32 - 1024 tokens: 70 -> 27 us.
#include "attention_tc.h"
#include "hgemm_tc.h"
#include "tile_phases.h"
#include "umma.cuh"
#include <cuda.h>

namespace mk {

namespace {

using namespace umma;

constexpr int AU_ITEMS = kAttnItems;
constexpr int AU_KEYS = 64;
constexpr int AU_PAGE = 16;                       // keys of a box: pages hold a multiple of them
constexpr int AU_PANEL = AU_KEYS * 128;           // bytes of 64 columns of a tile
constexpr int AU_QPANEL = AU_ITEMS * 128;
constexpr int AU_THREADS = 192;
constexpr float kSlack = 8.f;                     // base-2 logarithm
constexpr float kLog2e = 1.4426950408889634f;

template <int D, int DV>
struct Au {
    static constexpr int PANELS = D / 64, VPANELS = DV / 64;
    static constexpr int STAGES = D == 64 ? 4 : 2;
    static constexpr int K_BYTES = PANELS * AU_PANEL, V_BYTES = VPANELS * AU_PANEL, Q_BYTES = PANELS * AU_QPANEL;
    static constexpr size_t SMEM = 1024 + (size_t)Q_BYTES + (size_t)STAGES * (K_BYTES + V_BYTES);
    static constexpr int TMEM = DV + 2 * AU_KEYS <= 256 ? 256 : 512;
    static constexpr int CTAS = D <= 128 ? 2 : 1;
};

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t half2_bits(float x, float y) {
    const __half2 h = __floats2half2_rn(x, y);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t half2_rest(float x, float y, uint32_t rounded) {
    const float2 r = __half22float2(*reinterpret_cast<const __half2*>(&rounded));
    return half2_bits(x - r.x, y - r.y);
}
// cap * tanh(v / cap) as cap - 2 cap / (1 + exp(2 v / cap)): off by a few 1e-7 of the cap, which is what a score's own rounding costs.
__device__ __forceinline__ float capped_score(float v, float cap, float two_over_cap) {
    return cap - __fdividef(2.0f * cap, 1.0f + __expf(fminf(v * two_over_cap, 80.0f)));
}

template <int D, int DV, bool EXACT>
__global__ void __launch_bounds__(AU_THREADS, Au<D, DV>::CTAS)
attn_umma_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ AttnTcArgs a) {
    using L = Au<D, DV>;
    constexpr int ST = L::STAGES;
    extern __shared__ uint8_t au_smem[];
    __shared__ uint64_t bars[4 * ST + 7];
    __shared__ uint32_t tmem_slot;
    uint64_t *k_full = bars, *k_empty = bars + ST, *v_full = bars + 2 * ST, *v_empty = bars + 3 * ST, *s_full = bars + 4 * ST, *p_full = s_full + 2, *q_full = s_full + 4,
             *o_done = s_full + 5;
    uint8_t* qs = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(au_smem) + 1023) & ~(uintptr_t)1023);
    uint8_t* ks = qs + L::Q_BYTES;
    uint8_t* vs = ks + ST * L::K_BYTES;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        for (int i = 0; i < ST; ++i) {
            bar_init(&k_full[i], 1);
            bar_init(&k_empty[i], 1);
            bar_init(&v_full[i], 1);
            bar_init(&v_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            bar_init(&s_full[i], 1);
            bar_init(&p_full[i], AU_ITEMS);
            bar_init(&o_done[i], 1);
        }
        bar_init(q_full, AU_ITEMS);
        bar_init_fence();
    }
    if (warp == 5) tmem_alloc(&tmem_slot, L::TMEM);
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_trigger();
    // the work list, the lanes' headers and their block tables were staged ahead of the tick's first launch; everything else waits
    const int g = a.q_heads / a.kv_heads;
    const int work = blockIdx.x / a.kv_heads, kvh = blockIdx.x - work * a.kv_heads;
    const int lane_id = a.tiles[2 * work], row0 = a.tiles[2 * work + 1];
    const int rows_shift = __ffs(AU_ITEMS / g) - 1, rows_per_head = 1 << rows_shift;  // groups are powers of two
    const LaneHeader hdr = a.hdr[lane_id];
    const int n_rows = min(rows_per_head, hdr.n_tokens - row0);
    const int p_first = hdr.start_pos + row0, p_last = p_first + n_rows - 1;
    const int k_hi = p_last + 1;
    const int k_begin = attention_first_key(p_first, a.window, a.chunk) / AU_PAGE * AU_PAGE;
    const int n_tiles = (k_hi - k_begin + AU_KEYS - 1) / AU_KEYS;

    if (warp == 4) {
        // ---- loader
        bool ok = true;
        uint32_t page = 0;
        int t = 0;
        if (lane == 0) {
            prefetch_tensormap(&tm_k);
            prefetch_tensormap(&tm_v);
        }
        if (k_begin + lane * AU_PAGE < k_hi) page = a.tables[hdr.table_off + ((k_begin + lane * AU_PAGE) >> a.bt_shift)];
        pdl_wait();
        for (; t < n_tiles && ok; ++t) {
            const int pos0 = k_begin + t * AU_KEYS, pages = min(AU_KEYS / AU_PAGE, (k_hi - pos0 + AU_PAGE - 1) / AU_PAGE);
            if ((t & 7) == 0 && t > 0) {  // the page ids of the next eight tiles sit in the lanes
                const int pos = pos0 + lane * AU_PAGE;
                page = pos < k_hi ? a.tables[hdr.table_off + (pos >> a.bt_shift)] : 0u;
            }
            const int st = t % ST;
            const uint32_t ph = (uint32_t)(t / ST & 1) ^ 1;
            const int of = lane / L::PANELS, panel = lane % L::PANELS, vof = lane / L::VPANELS, vpanel = lane % L::VPANELS;
            const uint32_t blk = __shfl_sync(0xffffffffu, page, (t & 7) * 4 + (of & 3)), vblk = __shfl_sync(0xffffffffu, page, (t & 7) * 4 + (vof & 3));
            auto row_of = [&](uint32_t b, int i) {
                return (int)((kv_page_index(b, a.layer, a.layers, a.pool_blocks) * a.kv_heads + kvh) * a.block_tokens + ((pos0 + i * AU_PAGE) & (a.block_tokens - 1)));
            };
            ok = bar_wait(&k_empty[st], ph);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            if (lane == 0) bar_expect_tx(&k_full[st], (uint32_t)(pages * AU_PAGE * D * 2));
            __syncwarp();
            if (of < pages) tma_load_2d(smem_u32(ks) + st * L::K_BYTES + panel * AU_PANEL + of * (AU_PAGE * 128), &tm_k, panel * 64, row_of(blk, of), &k_full[st]);
            ok = bar_wait(&v_empty[st], ph);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            if (lane == 0) bar_expect_tx(&v_full[st], (uint32_t)(pages * AU_PAGE * DV * 2));
            __syncwarp();
            if (vof < pages) tma_load_2d(smem_u32(vs) + st * L::V_BYTES + vpanel * AU_PANEL + vof * (AU_PAGE * 128), &tm_v, vpanel * 64, row_of(vblk, vof), &v_full[st]);
        }
        if (!ok) {
            if (lane == 0) atomicExch(a.status, 31);
            for (int u = max(0, t - ST); u <= t && u < n_tiles; ++u) {  // copies in flight land before the CTA ends
                bar_wait(&k_full[u % ST], u / ST & 1);
                if (u < t) bar_wait(&v_full[u % ST], u / ST & 1);
            }
        }
    } else if (warp == 5) {
        // ---- MMA issuer
        pdl_wait();
        if (lane == 0) {
            constexpr uint32_t i_scores = f16_idesc(AU_ITEMS, AU_KEYS, false), i_out = f16_idesc(AU_ITEMS, DV, true);
            const uint32_t q_addr = smem_u32(qs), k_addr = smem_u32(ks), v_addr = smem_u32(vs);
            auto scores = [&](int t) {
                const int st = t % ST, area = tile_phase(t).at;
                if (!bar_wait(&k_full[st], t / ST & 1)) return false;
                fence_after();
                const uint64_t q = sw128_desc(q_addr), k = sw128_desc(k_addr + st * L::K_BYTES);
#pragma unroll
                for (int i = 0; i < D / 16; ++i)
                    mma(tmem + DV + area * AU_KEYS, q + (i >> 2) * (AU_QPANEL / 16) + (i & 3) * 2, k + (i >> 2) * (AU_PANEL / 16) + (i & 3) * 2, i_scores, i > 0);
                commit(&k_empty[st]);
                commit(&s_full[area]);
                return true;
            };
            bool ok = bar_wait(q_full, 0);
            fence_after();
            ok = ok && scores(0);
            for (int t = 0; t < n_tiles && ok; ++t) {
                // scores of tile t + 1 go to the area that P of tile t - 1 occupied: its product was issued before, and products of one
                // thread run in the order of their issue
                if (t + 1 < n_tiles) ok = scores(t + 1);
                const int st = t % ST;
                const TilePhase ph = tile_phase(t);
                ok = ok && bar_wait(&v_full[st], t / ST & 1) && bar_wait(&p_full[ph.at], ph.parity);
                if (!ok) break;
                fence_after();
                const uint32_t p = tmem + DV + ph.at * AU_KEYS;
                const uint64_t v = sw128_desc(v_addr + st * L::V_BYTES, AU_PANEL);
#pragma unroll
                for (int i = 0; i < AU_KEYS / 16; ++i) {
                    mma_tmem_a(tmem, p + i * 8, v + i * 128, i_out, t > 0 || i > 0);
                    if constexpr (EXACT) mma_tmem_a(tmem, p + AU_KEYS / 2 + i * 8, v + i * 128, i_out, true);
                }
                commit(&v_empty[st]);
                commit(&o_done[ph.at]);
            }
            if (!ok) atomicExch(a.status, 32);
        }
    } else {
        // ---- one item per thread
        const int ldq = a.ldq > 0 ? a.ldq : a.q_heads * D, ldo = a.q_heads * D;
        constexpr int CHUNKS = D / 8, BATCH = 8;
        pdl_wait();
        const int64_t first_row = a.cu_seqlens[lane_id] + row0;
        // the queries, eight pieces of a thread on their way together: a short prompt's CTA waits for little else (a launch of 64 rows, 16 heads of 128
        // over 4, took 14.5 us with four at a time and the work list read behind the wait, this 10.0; 16 heads of 256 over 8: 21.3 and 14.4; 64 lanes
        // of 32 rows, 32 heads of 128 over 8: 36.4 and 27.1)
#pragma unroll 1
        for (int i0 = tid; i0 < AU_ITEMS * CHUNKS; i0 += BATCH * AU_ITEMS) {
            float4 x[BATCH][2];
#pragma unroll
            for (int k = 0; k < BATCH; ++k) {
                const int i = i0 + k * AU_ITEMS, item = i / CHUNKS, c = (i - item * CHUNKS) * 8, hq = item >> rows_shift, r = item & (rows_per_head - 1);
                x[k][0] = x[k][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r < n_rows) {
                    const float* src = a.q + (first_row + r) * ldq + (kvh * g + hq) * D + c;
                    x[k][0] = *reinterpret_cast<const float4*>(src);
                    x[k][1] = *reinterpret_cast<const float4*>(src + 4);
                }
            }
#pragma unroll
            for (int k = 0; k < BATCH; ++k) {
                const int i = i0 + k * AU_ITEMS, item = i / CHUNKS, c = (i - item * CHUNKS) * 8, r = item & (rows_per_head - 1);
                float4 &x0 = x[k][0], &x1 = x[k][1];
                if (r < n_rows && c >= a.rot_from && c < a.rot_from + a.rot_dims) {
                    const int64_t pair0 = (int64_t)(p_first + r) * (a.rot_dims / 2) + (c - a.rot_from) / 2;
                    float* p[4][2] = {{&x0.x, &x0.y}, {&x0.z, &x0.w}, {&x1.x, &x1.y}, {&x1.z, &x1.w}};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (c - a.rot_from + 2 * j >= a.rot_dims) break;
                        const float cs = a.cos_t[pair0 + j], sn = a.sin_t[pair0 + j], u = *p[j][0], v = *p[j][1];
                        *p[j][0] = u * cs - v * sn;
                        *p[j][1] = v * cs + u * sn;
                    }
                }
                *reinterpret_cast<uint4*>(qs + (c >> 6) * AU_QPANEL + item * 128 + (((c & 63) * 2) ^ ((item & 7) << 4))) =
                    make_uint4(half2_bits(x0.x, x0.y), half2_bits(x0.z, x0.w), half2_bits(x1.x, x1.y), half2_bits(x1.z, x1.w));
            }
        }
        fence_async_smem();
        bar_arrive(q_full);

        const int hq = tid >> rows_shift, r = tid & (rows_per_head - 1);
        const int pos = p_first + r, lo = attention_first_key(pos, a.window, a.chunk), lo_last = attention_first_key(p_last, a.window, a.chunk);
        const uint32_t my = tmem + ((uint32_t)(warp * 32) << 16);
        const float two_over_cap = a.softcap != 0.f ? 2.0f / a.softcap : 0.f;
        const float unit = a.softcap != 0.f ? a.scale : a.scale * kLog2e;  // scores are base-2 logarithms
        float m_run = -INFINITY, sum = 0.f;
        bool ok = true;
        for (int t = 0; t < n_tiles; ++t) {
            const TilePhase ph = tile_phase(t);
            ok = __all_sync(0xffffffffu, bar_wait(&s_full[ph.at], ph.parity));
            if (!ok) break;
            fence_after();
            const uint32_t s_at = my + DV + ph.at * AU_KEYS;
            float s[AU_KEYS];
            tmem_ld32(s_at, reinterpret_cast<uint32_t*>(s));
            tmem_ld32(s_at + 32, reinterpret_cast<uint32_t*>(s) + 32);
            tmem_wait_ld();
            const int pos0 = k_begin + t * AU_KEYS;
            if (a.softcap != 0.f) {
#pragma unroll
                for (int j = 0; j < AU_KEYS; ++j) s[j] = capped_score(s[j] * unit, a.softcap, two_over_cap) * kLog2e;
            } else {
#pragma unroll
                for (int j = 0; j < AU_KEYS; ++j) s[j] *= unit;
            }
            if (pos0 + AU_KEYS - 1 > p_first || pos0 < lo_last) {  // uniform: some row does not see the whole tile
#pragma unroll
                for (int j = 0; j < AU_KEYS; ++j) s[j] = pos0 + j <= pos && pos0 + j >= lo && pos0 + j < k_hi ? s[j] : -INFINITY;
            }
            float top[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
            for (int j = 4; j < AU_KEYS; ++j) top[j & 3] = fmaxf(top[j & 3], s[j]);
            const float m_tile = fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3]));
            const bool grow = m_tile > m_run + kSlack;  // also when there was none yet
            if (__any_sync(0xffffffffu, grow)) {
                const float m_new = grow ? m_tile : m_run;
                const float alpha = m_run == -INFINITY ? 1.0f : ex2(m_run - m_new);
                if (t > 0) {
                    const TilePhase before = tile_phase(t - 1);
                    ok = __all_sync(0xffffffffu, bar_wait(&o_done[before.at], before.parity));
                    if (!ok) break;
                    fence_after();
#pragma unroll 1
                    for (int c = 0; c < DV; c += 32) {
                        uint32_t o[32];
                        tmem_ld32(my + c, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
                        tmem_st32(my + c, o);
                    }
                }
                sum *= alpha;
                m_run = m_new;
            }
            const float m_use = m_run == -INFINITY ? 0.f : m_run;
            float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < AU_KEYS; ++j) {
                s[j] = ex2(s[j] - m_use);
                part[j & 3] += s[j];
            }
            sum += (part[0] + part[1]) + (part[2] + part[3]);
            uint32_t w[AU_KEYS / 2];
#pragma unroll
            for (int j = 0; j < AU_KEYS / 2; ++j) w[j] = half2_bits(s[2 * j], s[2 * j + 1]);
            tmem_st32(s_at, w);
            if constexpr (EXACT) {
#pragma unroll
                for (int j = 0; j < AU_KEYS / 2; ++j) w[j] = half2_rest(s[2 * j], s[2 * j + 1], w[j]);
                tmem_st32(s_at + AU_KEYS / 2, w);
            }
            if (t == n_tiles - 1 && k_hi - pos0 < AU_KEYS) {
                // behind the last key the tile holds what its pages, or the ring, held before: weights of 0 need finite values there
                ok = __all_sync(0xffffffffu, bar_wait(&v_full[t % ST], t / ST & 1));
                if (!ok) break;
                const int first = k_hi - pos0, pieces = (AU_KEYS - first) * 8;
                for (int i = tid; i < pieces * L::VPANELS; i += AU_ITEMS)
                    *reinterpret_cast<uint4*>(vs + (t % ST) * L::V_BYTES + (i / pieces) * AU_PANEL + first * 128 + (i % pieces) * 16) = make_uint4(0u, 0u, 0u, 0u);
                fence_async_smem();
            }
            tmem_wait_st();
            fence_before();
            bar_arrive(&p_full[ph.at]);
        }
        if (ok) {
            const TilePhase last = tile_phase(n_tiles - 1);
            ok = __all_sync(0xffffffffu, bar_wait(&o_done[last.at], last.parity));
        }
        if (ok) {
            fence_after();
            float inv = 1.0f / sum;
            if (a.sink != nullptr) {
                const float m = m_run * 0.6931471805599453f, sink = a.sink[kvh * g + hq], top = fmaxf(m, sink), f = __expf(m - top);
                inv = f / (sum * f + __expf(sink - top));
            }
            const int64_t at = (first_row + r) * ldo + (kvh * g + hq) * D;
#pragma unroll 1
            for (int c = 0; c < DV; c += 32) {
                uint32_t o[32];
                tmem_ld32(my + c, o);
                tmem_wait_ld();
                if (r >= n_rows) continue;
                if (a.out != nullptr) {
#pragma unroll
                    for (int j = 0; j < 32; j += 4)
                        *reinterpret_cast<float4*>(a.out + at + c + j) = make_float4(__uint_as_float(o[j]) * inv, __uint_as_float(o[j + 1]) * inv, __uint_as_float(o[j + 2]) * inv,
                                                                                   __uint_as_float(o[j + 3]) * inv);
                }
                if (a.out_h != nullptr) {
#pragma unroll
                    for (int j = 0; j < 32; j += 8) {
                        uint32_t h[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) h[i] = half2_bits(__uint_as_float(o[j + 2 * i]) * inv, __uint_as_float(o[j + 2 * i + 1]) * inv);
                        *reinterpret_cast<uint4*>(a.out_h + at + c + j) = make_uint4(h[0], h[1], h[2], h[3]);
                    }
                }
            }
        } else if (lane == 0) {
            atomicExch(a.status, 33);
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 5) {
        fence_after();
        tmem_dealloc(tmem, L::TMEM);
    }
}

template <int D, int DV, bool EXACT>
void launch_variant(const AttnTcArgs& a, cudaStream_t s) {
    using L = Au<D, DV>;
    const uint64_t rows = (uint64_t)a.pool_pages * (uint64_t)a.kv_heads * (uint64_t)a.block_tokens;
    alignas(64) CUtensorMap tk, tv;
    encode_tma_2d(&tk, false, a.k_pool, D, rows, D * 2, 64, AU_PAGE, true);
    encode_tma_2d(&tv, false, a.v_pool, D, rows, D * 2, 64, AU_PAGE, true);
    auto* kernel = attn_umma_kernel<D, DV, EXACT>;
    ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), L::SMEM);
    launch_pdl(kernel, dim3((unsigned)(a.n_tiles * a.kv_heads)), dim3(AU_THREADS), L::SMEM, s, tk, tv, a);
    MK_LAUNCH_CHECK();
}

}  // namespace

void launch_attention_umma(const AttnTcArgs& a, cudaStream_t s) {
    if (a.status == nullptr) throw std::runtime_error("launch_attention_umma: a wait that gives up has nowhere to say so");
    if (a.pool_pages <= 0) throw std::runtime_error("launch_attention_umma: the pools' size is missing");
    switch (a.d) {
        case 64: a.exact_weights ? launch_variant<64, 64, true>(a, s) : launch_variant<64, 64, false>(a, s); break;
        case 128: a.exact_weights ? launch_variant<128, 128, true>(a, s) : launch_variant<128, 128, false>(a, s); break;
        case 192: launch_variant<192, 128, true>(a, s); break;
        case 256: a.exact_weights ? launch_variant<256, 256, true>(a, s) : launch_variant<256, 256, false>(a, s); break;
        default: throw std::runtime_error("launch_attention_umma: unsupported head_dim");
    }
}

}  // namespace mk
