"""The host-side plans of the two TMA matmuls (no GPU): how a launch is cut into tiles, K shares and partial-sum slots.
Invariants the consumer kernels rely on, and the plans of the benchmark's shapes (SmolLM3-3B: hidden 2048, q|k|v 3072,
gate|up 22016, FFN 11008)."""
import importlib

import numpy as np
import pytest

SMS = 148


@pytest.fixture(scope="module")
def env(mk):
    return importlib.import_module("macllm_infer_b200.ops"), importlib.import_module("macllm_infer_b200._capi")


def test_f16_gemm_plans_of_the_benchmark_shapes(env):
    ops, capi = env
    qkv = ops.matmul_plan(capi.PATH_HALF, 3072, 2048, 64)
    assert (qkv["bn"], qkv["row_tiles"], qkv["splits"]) == (64, 24, 6)           # 144 CTAs of one 64-lane decode tick
    down = ops.matmul_plan(capi.PATH_HALF, 2048, 11008, 64)
    assert (down["row_tiles"], down["splits"], down["kb_per_split"]) == (16, 9, 20)
    gate_up = ops.matmul_plan(capi.PATH_HALF, 22016, 2048, 2048)
    assert (gate_up["bn"], gate_up["n_tiles"], gate_up["splits"]) == (256, 8, 1)  # wide ticks never share K
    qkv = ops.matmul_plan(capi.PATH_HALF, 3072, 2048, 2048)
    assert (qkv["bn"], qkv["pairs"], qkv["splits"]) == (256, 1, 1)               # 96 tiles of two CTAs on 74 places beat three rounds of 128 x 128
    assert ops.half_matmul_plan(3072, 2048, 2048, may_pair=False)["bn"] == 128    # 2.6 rounds of 128 beat 1.3 rounds of 256
    head = ops.matmul_plan(capi.PATH_HALF, 128256, 2048, 64)
    assert head["splits"] == 1                                                    # enough row tiles already


@pytest.mark.parametrize("rows,cols", [(256, 2048), (2048, 2048), (3072, 2048), (2048, 11008), (22016, 2048), (12288, 4096), (1152, 768)])
@pytest.mark.parametrize("T", [2, 9, 33, 64, 65, 128, 512, 2048])
def test_f16_gemm_plan_invariants(env, rows, cols, T):
    ops, capi = env
    p = ops.matmul_plan(capi.PATH_HALF, rows, cols, T)
    assert p["bn"] in (64, 128, 256) and p["bn"] * p["n_tiles"] >= T > p["bn"] * (p["n_tiles"] - 1)
    assert p["row_tiles"] == -(-rows // 128)
    kb = cols // 64
    assert 1 <= p["splits"] <= 16 and p["kb_per_split"] * p["splits"] >= kb > p["kb_per_split"] * (p["splits"] - 1)
    if p["splits"] > 1:
        assert p["kb_per_split"] >= 4 and p["partial_floats"] == p["splits"] * T * rows <= (16 << 20) // 4
    else:
        assert p["partial_floats"] == 0
    assert ops.matmul_plan(capi.PATH_HALF, rows, cols, T, max_splits=1)["splits"] == 1
    assert p["pairs"] in (0, 1) and (p["pairs"] == 0 or (T > 128 and p["bn"] == 256))
    assert ops.half_matmul_plan(rows, cols, T) == p and ops.half_matmul_plan(rows, cols, T, may_pair=False)["pairs"] == 0
    # shares never take more than the scratch there is; with room for one less, a plan of fewer shares
    for floats in (0, p["partial_floats"] - 1, p["partial_floats"]):
        less = ops.half_matmul_plan(rows, cols, T, scratch_floats=max(floats, 0))
        assert less["partial_floats"] <= max(floats, 0) and less["kb_per_split"] * less["splits"] >= kb
        assert less == p if floats == p["partial_floats"] else floats < 0 or less["splits"] < p["splits"] or p["splits"] == 1


@pytest.mark.parametrize("rows,cols,T", [(22016, 2048, 2048), (2048, 11008, 2048), (8192, 2048, 2048), (9812, 1280, 129), (9812, 512, 2049), (1100, 11008, 700)])
def test_wide_calls_run_in_pairs_and_say_so(env, rows, cols, T):
    """The shapes of the pair kernel's own tests, an odd number of row tiles among them, and those the rule was measured at."""
    ops, capi = env
    p = ops.matmul_plan(capi.PATH_HALF, rows, cols, T)
    assert p["pairs"] == 1 and p["bn"] == 256 and p["n_tiles"] == -(-T // 256) and p["row_tiles"] == -(-rows // 128)


@pytest.mark.parametrize("rows,cols,T", [(2048, 2048, 1420), (2048, 2048, 2048), (3072, 2048, 1024), (8192, 256, 4096), (4096, 1024, 1800), (5120, 512, 1024), (8192, 768, 300)])
def test_short_k_and_single_rounds_stay_on_one_cta(env, rows, cols, T):
    """Where pairs measured slower, by up to 17 %: their launch and their stores weigh more than what they save on loads."""
    ops, capi = env
    assert ops.matmul_plan(capi.PATH_HALF, rows, cols, T)["pairs"] == 0


@pytest.mark.parametrize("rows,cols", [(2560, 2048), (2048, 2048), (22016, 2048), (2048, 11008), (1000, 11008), (128, 256), (128256, 2048)])
@pytest.mark.parametrize("T", [2, 17, 33, 64])
def test_streamed_matmul_plan_invariants(env, rows, cols, T):
    ops, capi = env
    p = ops.matmul_plan(capi.PATH_STREAM, rows, cols, T)
    nb = cols // 256
    assert p["row_tiles"] == -(-rows // 128) and p["tiles_per_group"] in (1, 2, 4)
    assert p["groups"] == -(-p["row_tiles"] // p["tiles_per_group"]) and p["items"] == p["groups"] * nb
    assert 1 <= p["ctas"] <= min(SMS, p["items"])   # at most one persistent CTA per SM
    assert 1 <= p["slots"] <= 16 and p["bn"] >= T and p["bn"] in (16, 32, 64)
    assert p["partial_floats"] == (p["slots"] * T * rows if p["slots"] > 1 else 0)
    assert p["partial_floats"] * 4 <= 24 << 20
    if p["slots"] == 1:
        assert p["ctas"] <= p["groups"]             # whole groups: every result is complete in one CTA
    whole = ops.matmul_plan(capi.PATH_STREAM, rows, cols, T, max_splits=1)
    assert whole["slots"] == 1 and whole["ctas"] == min(SMS, whole["groups"])


def test_streamed_matmul_plans_of_the_benchmark_shapes(env):
    ops, capi = env
    gate_up = ops.matmul_plan(capi.PATH_STREAM, 22016, 2048, 64)
    assert (gate_up["ctas"], gate_up["tiles_per_group"], gate_up["slots"]) == (148, 2, 3)   # 4.6 items of two units per CTA
    down = ops.matmul_plan(capi.PATH_STREAM, 2048, 11008, 64)
    assert (down["ctas"], down["tiles_per_group"]) == (148, 1) and down["slots"] <= 11
    head = ops.matmul_plan(capi.PATH_STREAM, 128256, 2048, 64)
    assert head["slots"] == 1 and head["ctas"] == 148                                          # 32 MB per slot: never cut


@pytest.mark.parametrize("experts,rows,total,most", [(256, 18432, 16384, 65), (512, 9216, 8192, 4000), (128, 36864, 8192, 65), (128, 6144, 11360, 89),
                                                     (8, 28672, 4096, 2000), (1024, 128, 65536, 65), (16, 128, 40, 17), (3, 384, 64, 64), (5, 256, 16, 9)])
def test_grouped_plans_take_what_64_row_chunks_take(env, experts, rows, total, most):
    """Chunks of 128 rows halve the chunks of full experts but not the one that every expert adds, and a job has half the row tiles: where that
    would not fit the table of a CTA's jobs, chunks are 64 rows."""
    ops, _ = env
    p, tiles = ops.grouped_matmul_plan(experts, rows, total, most), rows // 128

    def jobs(width, r):
        return -(-((total // width + experts) * (tiles // r)) // SMS) + 1

    assert p["jobs"] == jobs(p["rows"], p["tiles"]) <= p["table"] == 320
    if most > 64:
        assert p["rows"] == (128 if jobs(128, 1) <= p["table"] else 64)
    else:
        assert p["rows"] // 2 < max(most, 9) <= p["rows"]
    assert p["tiles"] == (2 if tiles % 2 == 0 and p["rows"] <= 64 else 1)


def test_plans_refuse_what_the_kernels_do_not_cover(env):
    ops, capi = env
    with pytest.raises(capi.MkError):
        ops.matmul_plan(capi.PATH_STREAM, 2048, 2048, 65)
    with pytest.raises(capi.MkError):
        ops.matmul_plan(capi.PATH_HALF, 2048, 100, 64)
    with pytest.raises(capi.MkError):
        ops.matmul_plan(capi.PATH_GEMV, 2048, 2048, 4)
