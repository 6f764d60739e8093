"""The forms of the matmuls of a few rows that whole models put together: two matrices in one launch (of one block format or of two, in either order), gate and up
in one, bf16 images with several inputs, and scattered results; at the row counts around their token tiles and one behind what they take."""
import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STD = 0.02


@pytest.fixture(scope="module")
def env(mk):
    return importlib.import_module("macllm_infer_b200.ops"), importlib.import_module("macllm_infer_b200._capi")


@pytest.mark.parametrize("first", ["Q4_K", "Q6_K"])
@pytest.mark.parametrize("second", ["Q4_K", "Q6_K"])
@pytest.mark.parametrize("T,rows,rows2,cols", [(1, 128, 16, 256), (3, 384, 130, 1280), (8, 2560, 512, 2048), (7, 4224, 1000, 512), (9, 384, 130, 1280)])
def test_two_block_matrices(env, orc, first, second, T, rows, rows2, cols):
    ops, capi = env
    k1, k2 = (getattr(capi, "TYPE_" + n) for n in (first, second))
    w1, w2 = ops.seed_tensor(0, 21, STD, k1, rows, cols), ops.seed_tensor(0, 22, STD, k2, rows2, cols)
    x = np.random.default_rng(T + rows).standard_normal((T, cols)).astype(np.float32)
    any_q6 = capi.TYPE_Q6_K if "Q6_K" in (first, second) else capi.TYPE_Q4_K
    assert (ops.narrow_matmul_plan(capi.PATH_STREAM, any_q6, rows + rows2, cols, T) is not None) == (T <= 8)
    got = ops.stacked_qmatmul(k1, w1, rows, k2, w2, rows2, cols, x)
    want = np.concatenate([orc.qmatmul(getattr(orc, first), w1, rows, cols, x, 1), orc.qmatmul(getattr(orc, second), w2, rows2, cols, x, 1)], axis=1)
    # two f16 roundings of a weight, one of an activation, 2^-11 each at most and a third of that in the mean square; 6 deviations
    assert np.isfinite(got).all() and np.abs(got - want).max() <= 6 * 2.0 ** -11 * STD * cols ** 0.5


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("T,F,cols,narrow", [(1, 8, 256, True), (2, 520, 1024, True), (8, 1500, 2048, True), (5, 5632, 512, True), (1, 9472, 256, False), (8, 9472, 256, False),
                                             (9, 520, 1024, False)])
def test_gate_and_up_in_blocks(env, orc, act, T, F, cols, narrow):
    ops, capi = env
    assert (ops.narrow_matmul_plan(capi.PATH_STREAM, capi.TYPE_Q4_K, 2 * F, cols, T, gated=True) is not None) == narrow
    gate, up = (ops.seed_tensor(0, s, STD, capi.TYPE_Q4_K, F, cols) for s in (23, 24))
    x = np.random.default_rng(T + F).standard_normal((T, cols)).astype(np.float32)
    got = ops.stacked_qmatmul(capi.TYPE_Q4_K, gate, F, capi.TYPE_Q4_K, up, F, cols, x, act)
    g, u = (orc.qmatmul(orc.Q4_K, w, F, cols, x, 1) for w in (gate, up))
    want = orc.act_mul(g, u, act)
    # each sum is off as above; the product adds them (the activations' slopes stay below 1.13), then one f16 rounding of the result
    err = 6 * 2.0 ** -11 * STD * cols ** 0.5
    assert np.isfinite(got).all() and (np.abs(got - want) <= err * (1.13 * np.abs(u) + np.abs(g) + err) + 2.0 ** -11 * np.abs(want) + 1e-6).all()


def bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a)).bfloat16().double().numpy()


def sums(w, x):
    """The products in 64 bits, and what 32-bit sums of them may be off by: up to four roundings at every step of 16 columns and 32 more where slices and shares
    meet, each at most 2^-23 of the largest partial sum."""
    w, x = bf16(w), bf16(x)
    return x @ w.T, (x.shape[1] / 4 + 32) * 2.0 ** -23 * (np.abs(x) @ np.abs(w).T)


@pytest.mark.parametrize("T", [1, 8, 9, 16, 17])
@pytest.mark.parametrize("rows,cols", [(16, 64), (300, 1088), (2049, 2048)])
def test_bf16_images(env, T, rows, cols):
    ops, _ = env
    r = np.random.default_rng(rows + T)
    w, x = STD * r.standard_normal((rows, cols)), r.standard_normal((T, cols))
    want, err = sums(w.astype(np.float32), x.astype(np.float32))
    assert (np.abs(ops.bf16_matmul(w, x) - want) <= err).all()


@pytest.mark.parametrize("T", [1, 8, 9, 16, 17])
@pytest.mark.parametrize("groups,cols", [((128, 384), 1088), ((256, 128, 640, 128), 192), ((128,) * 8, 2048), ((8192, 128, 1024), 64)])
def test_inputs_of_their_own(env, T, groups, cols):
    ops, _ = env
    r = np.random.default_rng(cols + T)
    w, x = (STD * r.standard_normal((sum(groups), cols))).astype(np.float32), r.standard_normal((len(groups), T, cols)).astype(np.float32)
    got, at = ops.bf16_matmul(w, x, groups), 0
    for g, n in enumerate(groups):
        want, err = sums(w[at:at + n], x[g])
        assert (np.abs(got[:, at:at + n] - want) <= err).all(), g
        at += n


@pytest.mark.parametrize("T", [1, 7, 16, 17])
@pytest.mark.parametrize("part_rows,part_valid,parts,rest,gates,turned", [(96, 80, 3, 0, 0, False), (128, 128, 2, 72, 0, True), (64, 50, 5, 33, 1, False), (128, 96, 4, 0, 3, True)])
def test_scattered_results(env, T, part_rows, part_valid, parts, rest, gates, turned):
    ops, _ = env
    cols, kept = 704, part_rows * parts
    r = np.random.default_rng(kept + T)
    w, x = (STD * r.standard_normal((kept + rest, cols))).astype(np.float32), r.standard_normal((T, cols)).astype(np.float32)
    row_map = r.permutation(T) if turned else None
    gate = r.standard_normal((gates, T, parts * part_valid)).astype(np.float32) if gates else None
    got, got_rest = ops.bf16_matmul_scattered(w, x, part_rows, part_valid, row_map, kept if rest else None, gate)
    want, err = sums(w, x)
    columns = (np.arange(parts)[:, None] * part_rows + np.arange(part_valid)).ravel()
    to = np.arange(T) if row_map is None else row_map
    scale = 1.0 if gate is None else 1 / (1 + np.exp(-gate.astype(np.float64).sum(0)))[to]   # rows of the gate go by destination
    # a gate of three f32 terms and its sigmoid: a few roundings of 2^-24 each
    assert (np.abs(got[to] - want[:, columns] * scale) <= err[:, columns] + 2e-6 * np.abs(want[:, columns])).all()
    if rest:
        assert (np.abs(got_rest - want[:, kept:]) <= err[:, kept:]).all()
