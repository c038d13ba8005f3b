"""The scheduling order of a batch's rays (csrc/ray_plan.cuh), compiled for the CPU:
every slot exactly once, whatever part of the detector the pixels are."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "nect_b200" / "csrc"
SOURCE = """
#include "ray_plan.cuh"
extern "C" int slot(int i, int P, int cols, int sub) { return nectb::strip_slot(i, P, cols, sub); }
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(SOURCE)
    subprocess.run([cxx, "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(d / "plan.cpp"), "-o",
                    str(d / "plan.so")], check=True)
    return ctypes.CDLL(str(d / "plan.so"))


@pytest.mark.parametrize("P,cols,sub", [
    (33 * 5, 5, 1), (64 * 7, 7, 1), (31 * 9 * 3, 9, 3), (1, 1, 1), (512, 512, 1),   # whole rows
    (1, 40, 1), (17, 40, 1), (100, 512, 1), (1500, 512, 1), (40 * 33 + 39, 40, 1),   # parts of rows
])
def test_strip_order_is_a_permutation(plan, P, cols, sub):
    slots = [plan.slot(i, P, cols, sub) for i in range(P)]
    assert sorted(slots) == list(range(P))
    if P % (cols * sub) == 0:   # 32 consecutive rays of a full strip are vertical neighbours
        if P >= 32 * cols * sub:
            assert slots[:32] == [r * cols * sub for r in range(32)]
    else:
        assert slots == list(range(P))
