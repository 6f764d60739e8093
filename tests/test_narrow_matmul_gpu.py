"""Matmuls of a few rows by warps that stream their own weights: row counts around the token tiles of 8 and 16, matrices that end inside a 16-row tile and
inside a 128-row unit, one block of K, K that does not share out evenly over warps, more row groups than CTAs; against the CPU oracle."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["Q4_K", "Q6_K"])
@pytest.mark.parametrize("T,rows,cols", [(1, 16, 256), (1, 130, 256), (3, 300, 1024), (7, 1000, 2816), (8, 2048, 11008), (8, 3072, 2048), (5, 8200, 512), (1, 2049, 4096)])
def test_blocks(mk, orc, name, T, rows, cols):
    ops, capi = (importlib.import_module("macllm_infer_b200." + n) for n in ("ops", "_capi"))
    kind = getattr(capi, "TYPE_" + name)
    w = ops.seed_tensor(0, 11, 0.02, kind, rows, cols)
    x = np.random.default_rng(T + rows).standard_normal((T, cols)).astype(np.float32)
    got = ops.qmatmul(kind, w, rows, cols, x, capi.PATH_STREAM)
    want = orc.qmatmul(getattr(orc, name), w, rows, cols, x, 1)
    # a weight carries two f16 roundings, an activation one (2^-11 of each at most, a third of that in the mean square): a result of size
    # 0.02 sqrt(cols) is off by 2^-11 * sqrt(3 / 3) of that in the mean square at most; 6 deviations cover every value here
    assert np.isfinite(got).all() and np.abs(got - want).max() <= 6 * 2.0 ** -11 * 0.02 * cols ** 0.5


@pytest.mark.parametrize("T,rows,cols", [(1, 16, 256), (9, 130, 256), (16, 300, 1280), (7, 1000, 2816), (16, 2048, 11008), (8, 3072, 2048), (15, 8200, 512)])
def test_images(mk, orc, T, rows, cols):
    ops, capi = (importlib.import_module("macllm_infer_b200." + n) for n in ("ops", "_capi"))
    w = ops.seed_tensor(0, 12, 0.02, capi.TYPE_Q8_0, rows, cols)
    x = np.random.default_rng(T + rows).standard_normal((T, cols)).astype(np.float32)
    got = ops.qmatmul(capi.TYPE_Q8_0, w, rows, cols, x, capi.PATH_HALF)
    want = orc.qmatmul(orc.Q8_0, w, rows, cols, x, 1)
    # both operands are rounded to f16 once
    assert np.isfinite(got).all() and np.abs(got - want).max() <= 6 * 2.0 ** -11 * (2 / 3) ** 0.5 * 0.02 * cols ** 0.5


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("T,F,cols", [(1, 8, 256), (3, 520, 1024), (16, 1500, 2048), (9, 5632, 512)])
def test_gated_images(mk, orc, act, T, F, cols):
    ops, capi = (importlib.import_module("macllm_infer_b200." + n) for n in ("ops", "_capi"))
    gate, up = (ops.seed_tensor(0, s, 0.02, capi.TYPE_Q8_0, F, cols) for s in (13, 14))
    x = np.random.default_rng(T + F).standard_normal((T, cols)).astype(np.float32)
    got = ops.gated_ffn(capi.TYPE_Q8_0, gate, up, F, cols, x, act)
    g, u = (orc.qmatmul(orc.Q8_0, w, F, cols, x, 1) for w in (gate, up))
    want = orc.act_mul(g, u, act)
    # each sum is off as above; the product adds them (the activations' slopes stay below 1.13), then one f16 rounding of the result
    err = 6 * 2.0 ** -11 * (2 / 3) ** 0.5 * 0.02 * cols ** 0.5
    assert (np.abs(got - want) <= err * (1.13 * np.abs(u) + np.abs(g) + err) + 2.0 ** -11 * np.abs(want) + 1e-6).all()
