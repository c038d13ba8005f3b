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


@pytest.mark.parametrize("rows,cols,sub", [(1, (1 << 27) + 1, 1), (3, 300_000_001, 1), (1, 1 << 26, 4),
                                           (40, (1 << 21) + 3, 25)])
def test_strip_order_of_wide_detectors(plan, rows, cols, sub):
    """Detectors whose strip of 32 rows has more than 2^31 - 1 slots."""
    line = cols * sub
    for i in [0, 1, 31, 32, line - 1, line // 3, rows * line // 2, rows * line - 32, rows * line - 1]:
        strip = i // (32 * line)
        h, rem = min(32, rows - 32 * strip), i - strip * 32 * line
        assert plan.slot(i, rows * line, cols, sub) == (32 * strip + rem % h) * line + rem // h
