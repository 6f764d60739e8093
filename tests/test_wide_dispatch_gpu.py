"""Dispatch edges of the kernels that take several rows, outputs or experts at a time: matrix-vector products of large matrices
(up to four output rows per warp), the router's product and choices at every register size, expert chunks above 64 rows."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(mk):
    return importlib.import_module("macllm_infer_b200.ops"), importlib.import_module("macllm_infer_b200._capi")


@pytest.mark.parametrize("name", ["TYPE_Q4_K", "TYPE_Q6_K", "TYPE_Q8_0"])
@pytest.mark.parametrize("T", [1, 2, 4, 5, 8, 9])
def test_matrix_vector_products_of_large_matrices(env, orc, name, T):
    ops, capi = env
    kind, rows, cols = getattr(capi, name), 18951, 512   # odd: the last warp's rows end behind the matrix
    w = ops.seed_tensor(0, 3, 0.02, kind, rows, cols)
    x = np.random.default_rng(T).standard_normal((T, cols)).astype(np.float32)
    got, want = ops.qmatmul(kind, w, rows, cols, x, capi.PATH_GEMV), orc.qmatmul(kind, w, rows, cols, x, 1)
    # the block sums are whole numbers; 16 blocks of at most a few units are added in another order: 2^-24 of the sum of magnitudes each
    assert np.abs(got - want).max() < 1e-5


@pytest.mark.parametrize("experts,k", [(8, 8), (40, 3), (64, 8), (65, 8), (128, 8), (129, 32), (256, 2), (257, 9), (1000, 33), (1024, 1)])
def test_router_choices_at_every_register_size(env, orc, experts, k):
    ops, _ = env
    logits = np.random.default_rng(experts + k).standard_normal((37, experts)).astype(np.float32)
    logits[1] = logits[1].round()                        # ties
    logits[2] = 0.0
    sel, w = ops.moe_route(logits, k)
    want_sel, want_w = orc.moe_route(logits, k)
    assert np.array_equal(sel, want_sel) and np.abs(w - want_w).max() < 1e-6


@pytest.mark.parametrize("T,experts,cols", [(297, 128, 2048), (600, 128, 2052), (1010, 130, 100), (1184, 128, 64), (1420, 128, 2048), (2001, 129, 516),
                                            (300, 128, 2050), (1, 4096, 64), (4800, 8, 64), (4736, 12, 64), (7105, 16, 64), (7104, 16, 64), (2700, 17, 64)])
def test_router_product_of_many_rows(env, T, experts, cols):
    ops, _ = env
    rng = np.random.default_rng(T)
    w, x = rng.standard_normal((experts, cols)).astype(np.float32), rng.standard_normal((T, cols)).astype(np.float32)
    got = ops.router_logits(w, x)
    # a lane's share of the columns in f32, then a tree of five: 2^-24 of the sum of magnitudes for each addition
    off_by = (cols / 32 + 6) * 2.0 ** -24 * (np.abs(x.astype(np.float64)) @ np.abs(w.T.astype(np.float64)))
    assert (np.abs(got - x.astype(np.float64) @ w.T.astype(np.float64)) <= off_by).all()
    for t in {0, T // 2, T - 1}:                          # the same bits as for the row by itself
        assert np.array_equal(ops.router_logits(w, x[t:t + 1])[0], got[t])


@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("counts", [[129, 0, 1, 128, 65, 300], [127, 128, 129, 64]])
def test_expert_chunks_above_64_rows(env, orc, counts, gated):
    ops, capi = env
    experts, rows, cols = len(counts), 256, 512
    off = np.concatenate([[0], np.cumsum(counts)])
    x = np.random.default_rng(1).standard_normal((off[-1], cols)).astype(np.float32)
    bank = [ops.seed_tensor(0, 10 + e, 0.02, capi.TYPE_Q4_K, rows, cols) for e in range(experts)]
    up = [ops.seed_tensor(0, 50 + e, 0.02, capi.TYPE_Q4_K, rows, cols) for e in range(experts)]
    got = ops.grouped_qmatmul(capi.TYPE_Q4_K, np.concatenate(bank), experts, rows, cols, x, off, capi.PATH_STREAM, np.concatenate(up) if gated else None)
    for e in range(experts):
        r = slice(off[e], off[e + 1])
        if off[e] == off[e + 1]:
            continue
        want = orc.qmatmul(orc.Q4_K, bank[e], rows, cols, x[r], 1)
        # The f16 images against the exact blocks.  A weight is scale * q - minimum; at a deviation of 0.02 the product is about 0.04
        # and the minimum 0.035 in size, and each of these, the difference and the activation is rounded once: at most 2^-11 of
        # itself, evenly spread (1 / sqrt 3 of that as a deviation).  In units of 0.02: sqrt(2^2 + 1.75^2 + 1 + 1) / sqrt 3 = 1.74
        # per term, the terms' signs at random; six deviations of the sum.
        off_by = 6 * 1.74 * 2.0 ** -11 * 0.02 * cols ** 0.5
        if gated:
            u = orc.qmatmul(orc.Q4_K, up[e], rows, cols, x[r], 1)
            off_by *= 2 * np.abs(want).max() + np.abs(u).max() + 1   # both factors' errors, and the f16 result's
            want = orc.act_mul(want, u, 0)
        assert np.abs(got[r] - want).max() < off_by


@pytest.mark.parametrize("kv_dtype", [np.float32, np.float16])
@pytest.mark.parametrize("q_heads,kv_heads,d,rotary", [(1, 1, 64, 64), (8, 1, 64, 64), (4, 1, 128, 128), (1, 1, 256, 256), (2, 2, 256, 0), (4, 1, 128, 64), (2, 2, 96, 96)])
def test_rotation_of_whole_heads(env, orc, kv_dtype, q_heads, kv_heads, d, rotary):
    """Head counts that leave a warp's last run of heads short; part-turned and odd-sized heads take the other kernel."""
    ops, _ = env
    bt, layers, layer, lens, starts = 16, 2, 1, [19, 5], [0, 40]
    rng = np.random.default_rng(d + q_heads)
    tables, T = [[4, 0], [2, 5, 1]], sum(lens)
    pools = [rng.standard_normal((6, layers, kv_heads, bt, d)).astype(np.float32).astype(kv_dtype) for _ in range(2)]
    q, k, v = (rng.standard_normal((T, n * d)).astype(np.float32) for n in (q_heads, kv_heads, kv_heads))
    cos, sin = orc.rope_tables(10000.0, rotary, 64) if rotary else (None, None)
    qn, kn = ((1 + 0.1 * rng.standard_normal(d)).astype(np.float32) for _ in range(2)) if q_heads != 2 else (None, None)
    kp, vp = (p.copy() for p in pools)
    res = ops.attention_step(q, k, v, kp, vp, tables, starts, lens, q_heads=q_heads, kv_heads=kv_heads, head_dim=d, block_tokens=bt, layers=layers, layer=layer,
                             scale=d ** -0.5, cos_table=cos, sin_table=sin, rotary_dim=rotary, q_norm_w=qn, k_norm_w=kn, norm_eps=1e-6)
    want_q, want_k = (x if w is None else orc.rmsnorm(x.reshape(-1, d), w, 1e-6).reshape(x.shape) for x, w in ((q, qn), (k, kn)))
    if rotary:
        want_q = orc.rope_apply(want_q, q_heads, d, rotary, res["positions"], cos, sin)
        want_k = orc.rope_apply(want_k, kv_heads, d, rotary, res["positions"], cos, sin)
    okp, ovp = (p.copy() for p in pools)
    orc.kv_scatter(want_k, v, okp, ovp, res["slots"], kv_heads, d, bt, layers, layer)
    # values below 8: a sum of squares in another order, a division and two products: a few 2^-24 of them (in f16 one rounding more)
    assert np.abs(res["q_rot"] - want_q).max() < 4e-6
    assert np.abs(kp.astype(np.float32) - okp.astype(np.float32)).max() < (4e-6 if kv_dtype == np.float32 else 2.0 ** -8) and np.array_equal(vp, ovp)
