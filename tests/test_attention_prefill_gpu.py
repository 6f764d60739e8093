"""The prefill kernel of paged attention (tcgen05) against the scalar kernel on the same pools, at the edges of its tiles of 64 keys
and 128 (row, head) items, with histories that begin inside a page, scores whose maximum keeps moving, and pools that hold NaN
wherever no key was written (ragged tile ends must not let them through)."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops(mk):
    return importlib.import_module("macllm_infer_b200.ops")


@pytest.mark.parametrize("geom", [(8, 8, 64), (32, 4, 64), (4, 4, 128), (16, 4, 128), (16, 8, 256), (16, 2, 256)])
@pytest.mark.parametrize("window,softcap,bt", [(0, 0.0, 16), (70, 0.0, 16), (0, 30.0, 32)])
def test_prefill_tiles_match_the_scalar_kernel(ops, geom, window, softcap, bt):
    q_heads, kv_heads, d = geom
    layers, layer = 2, 1
    lanes = [(0, 2), (0, 63), (0, 64), (1, 64), (15, 3), (47, 17), (48, 16), (63, 2), (200, 129), (130, 65), (0, 257), (77, 1)]
    rng = np.random.default_rng(d + q_heads + window)
    blocks = sum((s + n + bt - 1) // bt for s, n in lanes) + 3
    order = rng.permutation(blocks)
    tables, k_pool, v_pool, at = [], *(np.full((blocks, layers, kv_heads, bt, d), np.nan, np.float16) for _ in range(2)), 0
    for s, n in lanes:
        used = (s + n + bt - 1) // bt
        tables.append([int(b) for b in order[at:at + used]])
        at += used
        for p in range(s):  # the history; later keys are larger, so that the running maximum moves by more than the kernel's slack
            k_pool[tables[-1][p // bt], layer, :, p % bt] = rng.standard_normal((kv_heads, d)) * (1 + p / 64)
            v_pool[tables[-1][p // bt], layer, :, p % bt] = rng.standard_normal((kv_heads, d))
    T = sum(n for _, n in lanes)
    pos = np.concatenate([np.arange(s, s + n) for s, n in lanes])
    q = rng.standard_normal((T, q_heads * d)).astype(np.float16).astype(np.float32)  # exact as the kernel's operand
    k = (rng.standard_normal((T, kv_heads * d)) * (1 + pos[:, None] / 64)).astype(np.float32)
    v = rng.standard_normal((T, kv_heads * d)).astype(np.float32)
    out = [ops.attention_step(q, k, v, k_pool.copy(), v_pool.copy(), tables, [s for s, _ in lanes], [n for _, n in lanes], q_heads=q_heads, kv_heads=kv_heads,
                              head_dim=d, block_tokens=bt, layers=layers, layer=layer, scale=d ** -0.5, softcap=softcap, window=window, kernel=kernel)["out"]
           for kernel in (1, 2)]
    assert np.isfinite(out[0]).all() and np.isfinite(out[1]).all()
    # f16 weights: each is off by at most 2^-11 of itself, so their mean of values by 2^-11 of the largest value; the sums are f32
    assert np.abs(out[0] - out[1]).max() <= 1.2 * 2.0 ** -11 * np.abs(v_pool[np.isfinite(v_pool)].astype(np.float32)).max(initial=np.abs(v).max())


@pytest.mark.parametrize("q_heads,kv_heads,d,dv", [(8, 8, 64, 64), (16, 2, 64, 40), (8, 2, 128, 128), (8, 1, 128, 96), (4, 2, 192, 128), (8, 1, 192, 128), (8, 2, 256, 256), (4, 4, 256, 200)])
@pytest.mark.parametrize("exact,rule,sink,turned", [(True, "all", False, False), (True, "window", True, True), (True, "chunk", False, True), (False, "chunk", True, False),
                                                    (False, "all", True, True), (True, "cap", True, False)])
def test_forms_of_mixer_built_decoders(ops, q_heads, kv_heads, d, dv, exact, rule, sink, turned):
    """Two f16 weights, heads of 192 x 128, sinks, chunks and windows, and queries that turn on their way in, against the sums in 64 bits."""
    exact = exact or d == 192   # which has no other form
    bt, layers, layer, g = 16, 2, 1, q_heads // kv_heads
    window, chunk, cap = 70 if rule == "window" else 0, 128 if rule == "chunk" else 0, 30.0 if rule == "cap" else 0.0
    lanes = [(0, 2), (0, 64), (1, 64), (47, 17), (48, 16), (126, 5), (200, 129), (0, 257)]
    rng = np.random.default_rng(d + q_heads + dv)
    blocks = sum(-(-(s + n) // bt) for s, n in lanes) + 2
    order = rng.permutation(blocks)
    k_pool, v_pool = (np.full((blocks, layers, kv_heads, bt, d), np.nan, np.float16) for _ in range(2))
    tables, at, keys, values = [], 0, [], []
    for s, n in lanes:
        used = -(-(s + n) // bt)
        tables.append([int(b) for b in order[at:at + used]])
        at += used
        p = np.arange(s + n)
        k = (rng.standard_normal((s + n, kv_heads, d)) * (1 + p[:, None, None] / 64)).astype(np.float16)
        v = rng.standard_normal((s + n, kv_heads, d)).astype(np.float16)
        for pool, x in ((k_pool, k), (v_pool, v)):
            for i in p:
                pool[tables[-1][i // bt], layer, :, i % bt] = x[i]
        keys.append(k.astype(np.float64))
        values.append(v.astype(np.float64))
    T, most = sum(n for _, n in lanes), max(s + n for s, n in lanes)
    # queries of few bits, and "angles" whose products with them are exact: what enters the product is then the same on both sides
    q = (rng.integers(-32, 33, (T, q_heads, d)) / 16).astype(np.float32)
    rot_from, dims = (8, 24) if turned else (0, 0)
    cos, sin = (rng.choice([-1.0, -0.5, 0.0, 0.25, 0.5, 1.0], (most, dims // 2)).astype(np.float32) for _ in range(2)) if turned else (None, None)
    sinks = rng.standard_normal(q_heads).astype(np.float32) * 3 if sink else None
    out, half = ops.attention_prefill(q.reshape(T, -1), k_pool, v_pool, tables, [s for s, _ in lanes], [n for _, n in lanes], q_heads=q_heads, kv_heads=kv_heads, head_dim=d,
                                      block_tokens=bt, layers=layers, layer=layer, scale=d ** -0.5, softcap=cap, window=window, chunk=chunk, value_dim=dv,
                                      exact_weights=exact, sink=sinks, cos_table=cos, sin_table=sin, rot_from=rot_from)
    out, half, row = out.reshape(T, q_heads, d), half.reshape(T, q_heads, d), 0
    for (s, n), k, v in zip(lanes, keys, values):
        x = q[row:row + n].astype(np.float64)
        pos = np.arange(s, s + n)
        if turned:
            c, w = cos[pos][:, None].astype(np.float64), sin[pos][:, None].astype(np.float64)
            a, b = x[..., rot_from:rot_from + dims:2].copy(), x[..., rot_from + 1:rot_from + dims:2].copy()
            x[..., rot_from:rot_from + dims:2], x[..., rot_from + 1:rot_from + dims:2] = a * c - b * w, b * c + a * w
        for h in range(q_heads):
            score = x[:, h] @ k[:, h // g].T * d ** -0.5
            size = np.sqrt((x[:, h] ** 2 @ k[:, h // g].T ** 2).max()) * d ** -0.5   # of a score's partial sums, whose terms' signs are at random
            if cap:
                score = cap * np.tanh(score / cap)
            seen = np.arange(s + n)[None] <= pos[:, None]
            if window:
                seen &= np.arange(s + n)[None] > pos[:, None] - window
            if chunk:
                seen &= np.arange(s + n)[None] >= (pos // chunk * chunk)[:, None]
            score = np.where(seen, score, -np.inf)
            top = score.max(1, keepdims=True) if sinks is None else np.maximum(score.max(1, keepdims=True), sinks[h])
            e = np.exp(score - top)
            want = e @ v[:, h // g, :dv] / (e.sum(1, keepdims=True) + (0 if sinks is None else np.exp(sinks[h] - top)))
            got = out[row:row + n, h, :dv]
            # A weight is off by its score's absolute error: d products summed in steps of 16 and some roundings besides, 2^-23 of a partial sum
            # each, at random, six deviations; a soft cap takes the score through two more exponentials, a few 2^-22 of the cap.  Then the
            # weight itself: one f16 number is off by 2^-11 of it, two by 2^-22, and what lies below f16's least step by 2^-25 of a weight of
            # 1 for each key.  All of it times the largest value, and as much again for the denominator.  With two f16 numbers that is
            # below what one was seen to be off by (1.2e-3).
            off_by = 6 * size * (d / 16 + 8) ** 0.5 * 2.0 ** -23 + 8 * cap * 2.0 ** -22 + (s + n) * 2.0 ** -25 + (2.0 ** -22 if exact else 2.0 ** -11)
            assert np.abs(got - want).max() <= 2 * off_by * np.abs(v).max()
            assert np.array_equal(half[row:row + n, h, :dv], got.astype(np.float16))
        row += n
    assert d != 192 or np.isnan(out[..., 128:]).all()
