"""Wide calls of the f16-image GEMM run in 256 x 256 tiles of two CTAs: an odd last row tile, ragged rows and tokens, one and
several rounds of CTAs, short and long K, K shares; against the CPU oracle."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,rows,cols", [(129, 9812, 1280), (2049, 9812, 512), (1030, 9600, 1280), (513, 2048, 4096), (700, 1100, 11008), (600, 2176, 11008)])
def test_pairs_of_ctas_match_the_oracle(mk, orc, T, rows, cols):
    ops, capi = (importlib.import_module("macllm_infer_b200." + n) for n in ("ops", "_capi"))
    assert ops.matmul_plan(capi.PATH_HALF, rows, cols, T)["pairs"] == 1
    w = ops.seed_tensor(0, 7, 0.02, capi.TYPE_Q4_K, rows, cols)
    x = np.random.default_rng(T).standard_normal((T, cols)).astype(np.float32)
    got = ops.qmatmul(capi.TYPE_Q4_K, w, rows, cols, x, capi.PATH_HALF)
    want = orc.qmatmul(capi.TYPE_Q4_K, w, rows, cols, x, 1)
    # both operands are rounded to f16 once (2^-11 of each, independent): sqrt(cols) * 0.02 is the size of a result, its error's
    # deviation 2^-11 * sqrt(2 / 3) of that, and 5 deviations cover 2e7 results
    assert np.isfinite(got).all() and np.abs(got - want).max() <= 5 * 2.0 ** -11 * (2 / 3) ** 0.5 * 0.02 * cols ** 0.5


@pytest.mark.parametrize("T,rows,cols", [(2049, 9812, 512), (129, 9812, 1280), (513, 2048, 4096)])
def test_launches_that_follow_one_another_leave_nothing_behind(mk, T, rows, cols):
    """Short K: most of a CTA's stages are still to be handed back when its last load is out, and the next launch's CTAs take the place of
    those that end; the bits after 200 launches in a row are those of the first."""
    ops, capi = (importlib.import_module("macllm_infer_b200." + n) for n in ("ops", "_capi"))
    assert ops.matmul_plan(capi.PATH_HALF, rows, cols, T)["pairs"] == 1
    w = ops.seed_tensor(0, 7, 0.02, capi.TYPE_Q4_K, rows, cols)
    x = np.random.default_rng(T).standard_normal((T, cols)).astype(np.float32)
    first = ops.qmatmul(capi.TYPE_Q4_K, w, rows, cols, x, capi.PATH_HALF)
    ops.qmatmul_time(capi.TYPE_Q4_K, w, rows, cols, x, capi.PATH_HALF, 200)
    assert np.array_equal(first, ops.qmatmul(capi.TYPE_Q4_K, w, rows, cols, x, capi.PATH_HALF))
