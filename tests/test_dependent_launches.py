"""Kernels that start under their predecessor: what the predecessor produces must not be declared constant, and the results must be those
of ordinary launches, bit for bit."""
import os
import re
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "macllm-infer_b200" / "csrc"

# The parameters that are weights, written once when a model is loaded: only these may be `const T* __restrict__` in a kernel that waits for
# its predecessor, because the compiler may move a load of such memory in front of the wait.
WEIGHTS = {
    "qgemv_q4k_kernel": {"W"},
    "qgemv_q6k_kernel": {"ql_p", "qh_p", "sc_p", "d_p"},
    "qgemv_q80_kernel": {"qs_p", "d_p"},
    "qgemv_q6k_row_kernel": {"ql_p", "qh_p", "sc_p", "d_p"},
    "qgemv_q80_row_kernel": {"qs_p", "d_p"},
    "f32_gemv_kernel": {"W"},
    "f32_gemv_tile_kernel": {"W"},
    "f32_matmul_kernel": {"w"},
    "moe_router_kernel": {"w"},
    "wkv_decay_kernel": {"w2t", "w0"},
}


def kernels():
    """(file, name, parameters, body) of every kernel."""
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
            depth, at = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(text[at], 0)
                at += 1
            params = text[m.end():at - 1]
            if text[at:].lstrip()[:1] != "{":
                continue   # a declaration
            body_from = text.index("{", at)
            depth, end = 1, body_from + 1
            while depth:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
            yield path.name, m.group(1), params, text[body_from:end]


def test_only_weights_are_declared_constant_in_kernels_that_wait():
    seen = 0
    for file, name, params, body in kernels():
        if "pdl_wait()" not in body:
            continue
        seen += 1
        constant = set(re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)", params))
        assert constant <= WEIGHTS.get(name, set()), (file, name, constant)
    assert seen > 30


def test_the_batch_descriptor_is_an_ordinary_launch_behind_the_page_copies():
    """Kernels that touch memory ahead of their wait rely on a launch that begins when everything before the tick, and the page copies, are done."""
    assert "build_batch_kernel<<<" in (CSRC / "batch.cu").read_text()
    rope = (CSRC / "rope_kv.cu").read_text()
    assert "cow_copy_kernel<uint4><<<" in rope and "cow_copy_kernel<uint16_t><<<" in rope
    assert not any(re.search(r"launch_pdl\w*\(\s*(build_batch|cow_copy)_kernel", p.read_text()) for p in CSRC.glob("*.cu"))
    upload = (CSRC / "device_lm.cpp").read_text()
    upload = upload[upload.index("void DeviceLm::upload_tick"):]
    assert 0 < upload.index("cudaMemcpyAsync(stage_dev_") < upload.index("copy_shared_pages(t)") < upload.index("launch_build_batch(")


TICKS = """
import hashlib, importlib, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import __graft_entry__ as entry
entry.load_package()
eng, seed = (importlib.import_module("macllm_infer_b200." + n) for n in ("engine", "seed_gguf"))
spec = seed.scaled("qwen3-30b-a3b", layers=2, vocab=2048, hidden=1024, experts=16)
seed.write_seed_gguf(sys.argv[2], spec, seed=0)
for path in (1, 0):   # integer matrix-vector products throughout; what the model picks
    model = eng.Model.load_gguf(sys.argv[2], kv_dtype="f16", matmul_path=path, max_batch_tokens=256, max_batch_lanes=8, kv_capacity_tokens=4096)
    rng = np.random.default_rng(0)
    sessions = [model.new_session() for _ in range(4)]
    total = hashlib.sha256()
    at = 0
    for n in [40] + [1] * 60:
        ids = [rng.integers(0, 2048, n) for _ in sessions]
        logits, tokens = model.forward_batch([(s, t, at) for s, t in zip(sessions, ids)])
        total.update(np.ascontiguousarray(logits).tobytes())
        at += n
    print(path, total.hexdigest())
"""


@pytest.mark.gpu
def test_ticks_with_and_without_early_launches_have_the_same_bits(mk, tmp_path):
    got = []
    for early in ("1", "0"):
        r = subprocess.run([sys.executable, "-c", TICKS, str(ROOT), str(tmp_path / "seed.gguf")], env={**os.environ, "MACLLM_B200_PDL": early}, capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        got.append(r.stdout.split())
    assert len(got[0]) == 4 and got[0] == got[1]
