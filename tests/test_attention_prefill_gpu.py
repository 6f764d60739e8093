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
