"""The points a lane counts (lane_layout.h), compiled for the host.

The reverse sweep adds a lane's counted points to a parameter's sum behind a
branch for cut-off tiles, and goes on to tensor-memory instructions that a
whole warp has to issue together: the branch may not part a warp's lanes."""
import re
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parents[1] / "rsr_b200" / "csrc"

PROGRAM = r"""
#include <stdio.h>
#include "lane_layout.h"
template <int P> static void all() {
    const uint64_t sizes[] = {8, 16, 24, 32u * P - 8, 32u * P, 32u * P + 8, 64u * P - 16, 64u * P, 10008};
    for (uint64_t n : sizes)
        for (uint64_t tile = 0; tile < n; tile += 32u * P)
            for (int lane = 0; lane < 32; ++lane) {
                printf("%d %llu %llu %d %u", P, (unsigned long long)n, (unsigned long long)tile, lane,
                       rsr::counted_points<P>(lane, tile, n));
                for (int q = 0; q < P; ++q) printf(" %u", rsr::lane_point<P>(lane, q));
                printf("\n");
            }
}
int main() { all<2>(); all<4>(); all<8>(); }
"""


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("lanes")
    (d / "lanes.cpp").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", f"-I{CSRC}", "-o", str(d / "lanes"), str(d / "lanes.cpp")], check=True)
    out = subprocess.run([str(d / "lanes")], check=True, capture_output=True, text=True).stdout
    return [[int(v) for v in line.split()] for line in out.splitlines()]


def test_mask_holds_the_points_below_the_end(rows):
    for p, n, tile, lane, mask, *points in rows:
        want = [tile + o < n for o in points]
        assert [(mask >> q) & 1 for q in range(p)] == want


def test_lanes_of_a_tile_hold_each_point_once(rows):
    tiles = {}
    for p, n, tile, lane, mask, *points in rows:
        tiles.setdefault((p, n, tile), []).extend(points)
    assert all(sorted(v) == list(range(32 * k[0])) for k, v in tiles.items())


def test_cut_off_tiles_look_the_same_to_every_lane(rows):
    tiles = {}
    for p, n, tile, lane, mask, *points in rows:
        tiles.setdefault((p, n, tile), []).append((mask > (1 << p) - 1, mask & ((1 << p) - 1)))
    mixed = 0
    for (p, n, tile), lanes in tiles.items():
        assert {cut for cut, _ in lanes} == {tile + 32 * p > n}
        mixed += len({m for _, m in lanes}) > 1
    assert mixed >= 10   # tiles whose lanes differ were among them


def test_parameter_sums_branch_for_whole_warps_only():
    """Every branch in the adjoint kernel's inline assembly is on that comparison, and declared uniform."""
    src = (CSRC / "kernels_adj.cu").read_text()
    asm = "".join(re.findall(r'"((?:[^"\\]|\\.)*)"', src[src.index("void grad_add"):src.index("// kStackWidth")]))
    branches = re.findall(r"(?:@!?\w+ )?bra(?:\.\w+)* \w+", asm)
    assert branches and all("bra.uni " in b for b in branches), branches
    for guard in re.findall(r"setp\.(\w+)\.u32 p, %(\d+), (\d+);\\n@p bra", asm):
        assert guard[0] == "gt" and int(guard[2]) + 1 in (1 << 4, 1 << 8)
    # the sums themselves: bit by bit in a cut-off tile, all P values otherwise
    assert np.array_equal(sorted({int(b) for b in re.findall(r"and\.b32 b, %\d+, (\d+);", asm)}), 2 ** np.arange(8))
