"""Residual add and norm of wide ticks, several rows per CTA: the bits of the kernel that gives every row a CTA, for rows that do not share out evenly over the
CTAs and widths that leave some warps without a group."""
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
