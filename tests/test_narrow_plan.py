"""The host-side plan of matmuls of a few rows (no GPU): which calls it takes, and cuts that fit the scratch, the shared memory and the matrix."""
import importlib

import pytest

SMS = 148


@pytest.fixture(scope="module")
def env(mk):
    return importlib.import_module("macllm_infer_b200.ops"), importlib.import_module("macllm_infer_b200._capi")


def test_calls_that_are_taken(env):
    ops, capi = env
    image = lambda *a, **k: ops.narrow_matmul_plan(capi.PATH_HALF, capi.TYPE_Q8_0, *a, **k)
    blocks = lambda *a, **k: ops.narrow_matmul_plan(capi.PATH_STREAM, capi.TYPE_Q4_K, *a, **k)
    for rows in (16, 2048, 22016, 131072):
        assert image(rows, 2048, 1) and image(rows, 2048, 16) and image(rows, 2048, 17) is None
    assert image(2048, 2080, 4) is None and blocks(2048, 2112, 4) is None        # no whole steps of K
    assert blocks(2048, 11008, 8) and blocks(2048, 11008, 9) is None
    assert blocks(16384, 2048, 1) and blocks(16512, 2048, 1) is None             # 32 M weights
    # gated: by how many SMs the other kernel's whole row tiles keep busy, as measured: 59, 58, 65, 76 and 100 %
    shapes = ((11264, 2048), (22016, 2048), (24576, 4096), (28672, 3584), (75776, 2048))
    for T, taken in ((1, 3), (2, 3), (3, 2), (8, 2), (9, 0)):
        assert [blocks(*s, T, gated=True) is not None for s in shapes] == [i < taken for i in range(5)], T
    with pytest.raises(capi.MkError, match="interleaved"):
        ops.narrow_matmul_plan(capi.PATH_STREAM, capi.TYPE_Q6_K, 2048, 2048, 1, gated=True)
    with pytest.raises(capi.MkError, match="Q4_K and Q6_K"):
        ops.narrow_matmul_plan(capi.PATH_STREAM, capi.TYPE_Q8_0, 2048, 2048, 1)
    with pytest.raises(capi.MkError, match="planned on the host"):
        ops.narrow_matmul_plan(capi.PATH_GEMV, capi.TYPE_Q4_K, 2048, 2048, 1)


@pytest.mark.parametrize("rows,cols", [(16, 256), (130, 512), (2048, 2048), (3072, 2048), (2048, 11008), (8200, 1024), (3584, 7168)])
@pytest.mark.parametrize("T", [1, 3, 8, 16])
def test_cuts_fit(env, rows, cols, T):
    ops, capi = env
    for path, kind, step in ((capi.PATH_HALF, capi.TYPE_Q8_0, 64), (capi.PATH_STREAM, capi.TYPE_Q4_K, 256), (capi.PATH_STREAM, capi.TYPE_Q6_K, 256)):
        if path == capi.PATH_STREAM and T > 8:
            continue
        for gated, splits, scratch in ((False, 16, -1), (False, 16, 2 * T * rows), (False, 16, 2 * T * rows - 1), (False, 16, 0), (False, 1, -1), (True, 16, -1)):
            if gated and kind == capi.TYPE_Q6_K:
                continue
            p = ops.narrow_matmul_plan(path, kind, rows, cols, T, gated, splits, scratch)
            if p is None:   # a CTA without shares holds all of the activations: beside some 100 KB of ring and sums, T rows of cols 16-bit values
                assert (gated or splits == 1 or scratch >= 0) and 2 * T * cols > 90 * 1024
                continue
            assert p["tiles"] in (1, 2, 4, 8) and p["smem"] <= 200 * 1024
            assert 1 <= p["shares"] <= min(8, splits, cols // step) and p["ctas"] % p["shares"] == 0
            assert p["ctas"] // p["shares"] <= -(-(-(-rows // 16)) // p["tiles"])           # no CTA without a group of tiles
            assert p["ctas"] <= 2 * SMS
            assert p["partial_floats"] == (p["shares"] * T * rows if p["shares"] > 1 else 0)
            if gated or splits == 1 or scratch in (0, 2 * T * rows - 1):
                assert p["shares"] == 1
            if scratch == 2 * T * rows:
                assert p["shares"] <= 2


@pytest.mark.gpu
def test_profile_of_roles_says_when_there_are_none(env, capfd, monkeypatch):
    import numpy as np
    ops, capi = env
    monkeypatch.setenv("MACLLM_B200_QS_PROF", "1")
    w = ops.seed_tensor(0, 1, 0.02, capi.TYPE_Q4_K, 2048, 512)
    for T in (8, 9):
        ops.qmatmul(capi.TYPE_Q4_K, w, 2048, 512, np.ones((T, 512), np.float32), capi.PATH_STREAM)
        err = capfd.readouterr().err
        assert ("weight loader" in err) == (T == 9) and ("stream their own weights" in err) == (T == 8)
