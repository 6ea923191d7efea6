"""Where cg_dia.cu parks the warp sums of a thread's rows (park_rows.cuh),
compiled for the host: every row of every group once, and nothing else."""
import shutil
import subprocess

import pytest

from conftest import ROOT

_MAIN = r"""
#include <cstdio>
#include "park_rows.cuh"
int main() {
    std::printf("%d %d %d\n", nm::kDiaCgMaxQ, nm::kDiaCgMaxOwnTiles, nm::kDiaCgTilesPerRow);
    for (int Q = 1; Q <= nm::kDiaCgMaxQ; ++Q)
        for (int q0 = 0; q0 < Q; q0 += nm::kDiaCgGroup)
            for (int lane = 0; lane < 32; ++lane)
                if (const int r = nm::park_row(lane, q0, Q); r >= 0)
                    std::printf("%d %d %d %d\n", Q, q0, lane, r);
}
"""


def _lane_of(q, count):
    """The lane that holds value q of `count` summed together: multi_warp_sum
    halves the values at the shuffles of distance 16, 8, ..., so value q ends
    where the lane's top bits are q's."""
    return q * (32 // count)


@pytest.fixture(scope="module")
def parked(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    assert cxx, "no host compiler"
    d = tmp_path_factory.mktemp("park_rows")
    (d / "main.cpp").write_text(_MAIN)
    subprocess.run([cxx, "-std=c++17", "-x", "c++", f"-I{ROOT / 'num_b200' / 'csrc'}",
                    str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    out = subprocess.run([str(d / "main")], check=True, capture_output=True, text=True).stdout
    first, *rest = ([int(c) for c in line.split()] for line in out.splitlines())
    return first, rest


def test_rows_are_parked_once_and_inside_their_room(parked):
    (most, room, per_row), rows = parked
    for Q in range(1, most + 1):
        mine = [(q0, lane, r) for q, q0, lane, r in rows if q == Q]
        assert sorted(r for _, _, r in mine) == list(range(Q))
        assert all((r + 1) * per_row <= room for _, _, r in mine)
        width = 1 << max(0, (min(Q, 8) - 1).bit_length())
        assert all(lane == _lane_of(r - q0, width) for q0, lane, r in mine)
