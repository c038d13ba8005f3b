"""The scheduling order of a batch's rays and the split of its workspace
(csrc/ray_plan.cuh), compiled for the CPU: every slot exactly once, whatever part of the
detector the pixels are; the stored rows a workspace of a given size keeps; how long the
weight gradients stay in the tensor cores' accumulators."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "nect_b200" / "csrc"
SOURCE = """
#include "ray_plan.cuh"
using namespace nectb;
extern "C" int slot(int i, int P, int cols, int sub) { return strip_slot(i, P, cols, sub); }
extern "C" int64_t order(int R, int P) { return (int64_t)order_bytes(R, P); }
extern "C" int64_t recommended(int R, int rounds, int64_t per_ray) {
  return (int64_t)staged_round_bytes(R, rounds, (size_t)per_ray);
}
extern "C" int claim(int R, int P) { return slots_per_claim(R, P); }
extern "C" int stretches(int64_t R, int64_t per_round, int rounds) { return accumulator_stretches(R, per_round, rounds); }
extern "C" int tiles(unsigned int chunks, int n, int blocks) { return stretch_tiles(chunks, n, blocks); }
// rows of the store, rays of a round; every part of the region inside it, in order
extern "C" int layout(int64_t at, int64_t bytes, int R, int P, int S, int64_t row, int64_t per_ray, int rounds,
                      int64_t* rows, int64_t* per_round) {
  Workspace ws;
  ws.stage = (float*)at;
  ws.stage_bytes = (size_t)bytes;
  const StageLayout L = stage_layout(ws, R, P, S, (size_t)row, (size_t)per_ray, rounds);
  *rows = L.xcap;
  *per_round = L.per_round;
  if (!L.per_round) return 1;
  const int64_t o = (int64_t)L.order, f = (int64_t)L.offs, s = (int64_t)L.block_samples, g = (int64_t)L.stage;
  const int64_t x = L.xstore ? (int64_t)L.xstore : g;
  return o >= at && (int64_t)L.block_sums >= o + 4 * (int64_t)R && f > (int64_t)L.block_sums && s >= f + 8 * (int64_t)R &&
         x > s && x % 16 == 0 && g % 16 == 0 && x + L.xcap * row <= g && g + L.per_round * per_ray <= at + bytes;
}
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
    lib = ctypes.CDLL(str(d / "plan.so"))
    i64, i32 = ctypes.c_int64, ctypes.c_int
    lib.order.restype = lib.recommended.restype = i64
    lib.recommended.argtypes = [i32, i32, i64]
    lib.stretches.argtypes = [i64, i64, i32]
    lib.layout.argtypes = [i64, i64, i32, i32, i32, i64, i64, i32, ctypes.POINTER(i64), ctypes.POINTER(i64)]
    return lib


def layout(plan, bytes_, R, P, S, row, per_ray, rounds, at=1 << 40):
    rows, per_round = ctypes.c_int64(), ctypes.c_int64()
    assert plan.layout(at, bytes_, R, P, S, row, per_ray, rounds, ctypes.byref(rows), ctypes.byref(per_round))
    return rows.value, per_round.value


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


@pytest.mark.parametrize("R,S,features", [(700, 64, 32), (24999, 100, 32), (16000, 64, 64), (4882, 512, 76),
                                          (65536, 512, 32), (262144, 512, 32), (1, 1, 32)])
@pytest.mark.parametrize("rounds", [1, 4, 16])
def test_rows_come_before_large_rounds(plan, R, S, features, rounds):
    """The recommended size keeps every row and its rounds; below it the store keeps the rows
    that rounds of R / `rounds` rays leave it, and rounds grow only into what is left."""
    row, per_ray, P = (features + 15) // 16 * 32, (S + 3) // 4 * 4 * features * 4, 512 * 512
    ob, best = plan.order(R, P), plan.recommended(R, rounds, per_ray)
    least = -(-R // rounds) * per_ray
    full = ob + best + 256 + (R * S * row + 255) // 256 * 256
    assert layout(plan, full, R, P, S, row, per_ray, rounds) == (R * S, min(R, (best + 256) // per_ray))
    for k in range(1, 200):
        size = ob + (full - ob) * k // 200
        rows, per_round = layout(plan, size, R, P, S, row, per_ray, rounds)
        if size - ob >= best + R * S * row + 256:
            want = R * S
        else:
            want = max(0, min(R * S, (size - ob - least - 256) // row))
            want = want if want >= S else 0
        if per_round:   # (the fused single pass below 64 rounds)
            assert rows == want
            assert per_round >= (least // per_ray if rows else 1)


@pytest.mark.parametrize("R", [1, 5, 16, 4882, 50000, 262144])
@pytest.mark.parametrize("rounds", [1, 3, 4, 16, 64])
@pytest.mark.parametrize("launches", range(1, 17))
def test_accumulators_hold_no_more_than_a_round(plan, R, rounds, launches):
    """However many launches a batch takes, the accumulators hold at most R / `rounds` rays."""
    per_round = -(-R // launches)
    n = plan.stretches(R, per_round, rounds)
    longest = per_round if n == 1 else min(per_round, -(-R // n))
    assert longest <= -(-R // rounds)


@pytest.mark.parametrize("chunks,stretches,blocks", [(0, 4, 444), (7, 4, 444), (525_000, 4, 444), (2**32 - 1, 2, 1),
                                                     (525_000, 64, 148), (525_000, 1, 148)])
def test_tiles_of_a_stretch(plan, chunks, stretches, blocks):
    """The blocks' stretches add up to a share of the batch's tiles, rounded up to a whole tile a block."""
    tiles = plan.tiles(chunks, stretches, blocks)
    if stretches == 1:
        assert tiles == 2**31 - 1
    else:
        assert tiles == max(1, -(-chunks // (4 * stretches * blocks)))


@pytest.mark.parametrize("R,P,want", [(1, 1, 1), (1, 64, 1), (1, 128, 2), (1, 65536, 32), (256, 65536, 4),
                                      (2000, 65536, 1), (65536, 65536, 1), (1, 2**31 - 1, 32), (0, 65536, 32)])
def test_claims(plan, R, P, want):
    assert plan.claim(R, P) == want


@pytest.mark.parametrize("shift", [0, 4, 8, 12, 20, 248])
def test_rows_are_aligned_in_any_workspace(plan, shift):
    """Stored rows (rows * 16 bytes) and staged ones start on 16-byte boundaries (checked in
    layout()) and stay inside the region, whatever the workspace's address."""
    R, S, row, per_ray, P = 700, 64, 64, 64 * 128, 4096
    full = plan.order(R, P) + plan.recommended(R, 4, per_ray) + 256 + R * S * row
    for size in (full, full + 16, full - 8, full // 2, full // 5):
        layout(plan, size, R, P, S, row, per_ray, 4, at=(1 << 40) + shift)
    assert layout(plan, full, R, P, S, row, per_ray, 4, at=(1 << 40) + shift) == (R * S, R)
