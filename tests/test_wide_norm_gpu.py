"""Residual add and norm of wide ticks: the bits of narrow calls, for rows that do not share out evenly over the SMs and widths that leave some
warps without a group."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sandwich", [False, True])
@pytest.mark.parametrize("rows,dim", [(1184, 2048), (1300, 256), (2049, 2048), (600, 3584), (1777, 2304), (593, 4096)])
def test_rows_equal_those_of_narrow_calls(mk, rows, dim, sandwich):
    ops = importlib.import_module("macllm_infer_b200.ops")
    r = np.random.default_rng(rows)
    h, a = (r.standard_normal((rows, dim)).astype(np.float32) for _ in range(2))
    w, pw = ((1 + 0.1 * r.standard_normal(dim)).astype(np.float32) for _ in range(2))
    pw = pw if sandwich else None
    h1, n1 = ops.add_norm(h, a, 0.5, pw, w, 1e-6)
    parts = [ops.add_norm(h[i:i + 500], a[i:i + 500], 0.5, pw, w, 1e-6) for i in range(0, rows, 500)]
    assert np.array_equal(h1, np.concatenate([p[0] for p in parts])) and np.array_equal(n1, np.concatenate([p[1] for p in parts]))


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("rows,dim", [(1184, 2048), (1300, 256), (2049, 2048), (600, 3584), (593, 4096)])
def test_quantised_rows_equal_those_of_narrow_calls(mk, rows, dim, kind):
    """The blocks, their factors and sums and the f16 image, and the image alone, whose blocks stay as they were."""
    ops = importlib.import_module("macllm_infer_b200.ops")
    r = np.random.default_rng(rows + kind)
    h, a = (r.standard_normal((rows, dim)).astype(np.float32) for _ in range(2))
    h[5, :256] = -a[5, :256]           # a block of zeros
    h[rows - 1, 7] = 300.0
    w = (1 + 0.1 * r.standard_normal(dim)).astype(np.float32)
    whole = ops.add_norm_quant(h, a, 1.0, None, w, 1e-6, kind, fill=77)
    parts = [ops.add_norm_quant(h[i:i + 500], a[i:i + 500], 1.0, None, w, 1e-6, kind, fill=77) for i in range(0, rows, 500)]
    for got, want in zip(whole, zip(*parts)):
        assert np.array_equal(got, np.concatenate(want))
    # a plain quantisation of the normed rows makes the same blocks
    qs, d, bs = ops.quantize(ops.add_norm(h, a, 1.0, None, w, 1e-6)[1], kind)
    assert np.array_equal(whole[1], qs) and np.array_equal(whole[2], d) and (kind == 1 or np.array_equal(whole[3], bs))
    f16 = (d.repeat(256 if kind == 0 else 32, axis=1) * qs).astype(np.float16)
    assert np.array_equal(whole[4], f16)
    for lo, hi in ((0, rows), (0, 500)):
        h1, qs, d, bs, xh = ops.add_norm_quant(h[lo:hi], a[lo:hi], 1.0, None, w, 1e-6, kind, half_only=True, fill=77)
        assert np.array_equal(xh, whole[4][lo:hi]) and np.array_equal(h1, whole[0][lo:hi])
        assert (qs == 77).all() and (d == 77).all() and (bs == 77).all()
