"""A forward that failed on the device leaves the caller's buffers as they are, whether its logits travel in one copy (under 2 MB) or in parts."""
import ctypes as C
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [2, 15, 16, 40])
def test_a_failed_forward_leaves_the_buffers_alone(mk, tmp_path, lanes):
    eng, seed, capi = (importlib.import_module("macllm_infer_b200." + n) for n in ("engine", "seed_gguf", "_capi"))
    spec = seed.scaled("qwen3-30b-a3b", layers=1, vocab=32768, hidden=1024, experts=16)   # 16 rows are 2 MB
    # router weights that are no numbers: the choices stay in range, the forward fails when it is read
    plan = [(name, dims, kind, float("nan") if "ffn_gate_inp" in name else std) for name, dims, kind, std in seed.tensor_plan(spec)]
    path = seed._write_file(tmp_path / "m.gguf", seed._meta(spec), plan, spec, 0)
    lib = capi.lib()
    model = eng.Model.load_gguf(path, max_batch_tokens=64, max_batch_lanes=40)
    sessions = [model.new_session() for _ in range(lanes)]
    arr, keep = model._lanes([(s, np.array([5 + i], np.uint32), 0) for i, s in enumerate(sessions)])
    r = C.c_void_p()
    capi.check(lib.mk_reserve_batch(model._h, arr, lanes, C.byref(r)))
    capi.check(lib.mk_forward_batch_reserved(model._h, arr, lanes, r, capi.FWD_WANT_LOGITS | capi.FWD_WANT_TOKENS))
    logits, tokens = np.full((lanes, spec.vocab), 7.0, np.float32), np.full(lanes, 7, np.uint32)
    with pytest.raises(capi.MkError, match="non-finite logits for token row"):
        capi.check(lib.mk_read_output(model._h, logits.ctypes.data, tokens.ctypes.data))
    assert (logits == 7.0).all() and (tokens == 7).all()
    del keep
    for s in sessions:
        s.close()
    model.close()
