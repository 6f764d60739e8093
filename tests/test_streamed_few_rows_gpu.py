"""The streamed matmul through tensor memory at up to eight rows: the matrices above the line where warps that stream their own weights leave off, in both block
formats, with partial sums and with whole groups of row tiles per CTA; against the CPU oracle."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [16, 1])
@pytest.mark.parametrize("name,T,rows,cols", [("Q4_K", 2, 16512, 2048), ("Q4_K", 8, 3100, 11008), ("Q6_K", 1, 16500, 2048), ("Q6_K", 5, 131201, 256), ("Q6_K", 8, 3100, 11008)])
def test_large_matrices(mk, orc, monkeypatch, name, T, rows, cols, splits):
    ops, capi = (importlib.import_module("macllm_infer_b200." + n) for n in ("ops", "_capi"))
    kind = getattr(capi, "TYPE_" + name)
    assert ops.narrow_matmul_plan(capi.PATH_STREAM, kind, rows, cols, T) is None
    monkeypatch.setenv("MACLLM_B200_QS_SPLITS", str(splits))
    w = ops.seed_tensor(0, 31, 0.02, kind, rows, cols)
    x = np.random.default_rng(T + rows).standard_normal((T, cols)).astype(np.float32)
    got = ops.qmatmul(kind, w, rows, cols, x, capi.PATH_STREAM)
    want = orc.qmatmul(getattr(orc, name), w, rows, cols, x, 1)
    # two f16 roundings of a weight, one of an activation, 2^-11 each at most and a third of that in the mean square; 6 deviations
    assert np.isfinite(got).all() and np.abs(got - want).max() <= 6 * 2.0 ** -11 * 0.02 * cols ** 0.5
