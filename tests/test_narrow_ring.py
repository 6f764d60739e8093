"""The ring of copies of the narrow matmul's warps (macllm-infer_b200/csrc/narrow_ring.h), compiled for the host: every copy is waited for once, in the phase it
was asked for in; a warp whose wait gave up asks for no more and leaves none under way.  No GPU: the kernel's own wait never runs out there."""
import ctypes as C
import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    so = tmp_path_factory.mktemp("emu") / "libnarrow_ring.so"
    cxx = "/usr/bin/g++" if os.access("/usr/bin/g++", os.X_OK) else "g++"
    subprocess.run([cxx, "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(ROOT / "macllm-infer_b200" / "csrc"), "-o", str(so),
                    str(ROOT / "tests" / "narrow_ring_emulation.cpp")], check=True)
    return C.CDLL(str(so))


# stages of Q6_K and Q4_K; one step to more steps than stages; groups that end at the matrix's last tile, inside a group and behind it
@pytest.mark.parametrize("stages", [3, 4])
@pytest.mark.parametrize("groups,rg_shift,sub_tile,tiles", [((0, 1), 0, 0, 1), ((0, 3), 0, 0, 3), ((2, 5), 1, 1, 9), ((0, 4), 3, 7, 25), ((3, 4), 3, 5, 26), ((0, 2), 2, 3, 3)])
@pytest.mark.parametrize("steps", [(0, 1), (1, 3), (0, 4), (2, 9)])
def test_no_copy_is_lost_and_no_barrier_is_armed_twice(emu, stages, groups, rg_shift, sub_tile, tiles, steps):
    n = (groups[1] - groups[0]) * (steps[1] - steps[0])
    for fails in range(-1, n):
        assert emu.emu_narrow_ring(stages, *groups, rg_shift, sub_tile, tiles, *steps, fails) == 0, fails
