"""The batch descriptor of a tick (cu_seqlens, positions, slots, last rows) with more lanes than a warp and more than a block of
threads."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [31, 33, 1024, 1100])
def test_descriptor_of_many_lanes(mk, lanes):
    ops = importlib.import_module("macllm_infer_b200.ops")
    rng = np.random.default_rng(lanes)
    bt, start, n = 16, rng.integers(0, 40, lanes), rng.integers(1, 4, lanes)
    used = -(-(start + n) // bt)
    ends = np.cumsum(used)
    order = rng.permutation(int(ends[-1]) + 2)
    tables = [[int(b) for b in order[e - u:e]] for e, u in zip(ends, used)]
    pool = [np.zeros((len(order), 1, 1, bt, 4), np.float32) for _ in range(2)]
    x = rng.standard_normal((int(n.sum()), 4)).astype(np.float32)
    got = ops.attention_step(x, x, x, *pool, tables, start, n, q_heads=1, kv_heads=1, head_dim=4, block_tokens=bt, layers=1, layer=0, scale=0.5)
    pos = np.concatenate([np.arange(s, s + k) for s, k in zip(start, n)])
    lane = np.repeat(np.arange(lanes), n)
    assert np.array_equal(got["cu_seqlens"], np.concatenate([[0], np.cumsum(n)]))
    assert np.array_equal(got["last_index"], np.cumsum(n) - 1) and np.array_equal(got["positions"], pos)
    assert np.array_equal(got["slots"], [tables[l][p // bt] * bt + p % bt for l, p in zip(lane, pos)])
