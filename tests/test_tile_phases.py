"""The barriers of the prefill attention (macllm-infer_b200/csrc/tile_phases.h), compiled for the host: in every order of events, scores, weights and outputs are
only touched once they are complete.  No GPU."""
import ctypes as C
import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    so = tmp_path_factory.mktemp("emu") / "libtile_phases.so"
    cxx = "/usr/bin/g++" if os.access("/usr/bin/g++", os.X_OK) else "g++"
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(ROOT / "macllm-infer_b200" / "csrc"), "-o", str(so),
                    str(ROOT / "tests" / "tile_phases_emulation.cpp")], check=True)
    return C.CDLL(str(so))


@pytest.mark.parametrize("stages", [2, 4])   # of heads of 128 and more, of 64
@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 5, 6])
def test_nothing_is_touched_before_it_is_complete(emu, tiles, stages):
    assert emu.emu_tile_phases(tiles, stages) == 0


def test_one_barrier_for_all_outputs_would_not_do(emu):
    assert emu.emu_one_output_barrier(1, 2) == 0
    assert all(emu.emu_one_output_barrier(tiles, 2) > 0 for tiles in (2, 3, 4, 5))
