"""The grids of the engine's step over its tile lists (step_lists.cuh), compiled
for the host: a list has room for every entry that a grid reaches, and the key
of a kept step graph settles the launch of the kernel of the diagonal form."""
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

_MAIN = r"""
#include <cstdio>
#include "step_lists.cuh"
int main() {
    for (int64_t t = 0; t <= 3000; ++t)
        std::printf("%d %d %d %d %lld\n", nm::tile_bucket(t), nm::dia_bucket(t), nm::dia_split(t),
                    nm::dia_grid(t), (long long)nm::tile_list_room(t));
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    assert cxx, "no host compiler"
    d = tmp_path_factory.mktemp("step_lists")
    (d / "main.cpp").write_text(_MAIN)
    subprocess.run([cxx, "-std=c++17", "-x", "c++", f"-I{ROOT / 'num_b200' / 'csrc'}",
                    str(d / "main.cpp"), "-o", str(d / "main")], check=True)
    out = subprocess.run([str(d / "main")], check=True, capture_output=True, text=True).stdout
    v = np.array([[int(c) for c in line.split()] for line in out.splitlines()])
    return dict(zip(["bucket", "dia", "split", "grid", "room"], v.T))


def test_every_entry_a_grid_reaches_is_in_the_list(rules):
    tiles = np.arange(rules["grid"].size)
    on = tiles > 0
    # bs_spmv_dia's last CTA, and the one-CTA-per-tile kernels'
    last = (rules["grid"][on] - 1) >> rules["split"][on]
    assert np.all(last < rules["room"][on])
    assert np.all(rules["bucket"] <= rules["room"])
    # whole tiles are covered: every tile by each of its CTAs
    assert np.all(rules["grid"][on] >= tiles[on] << rules["split"][on])
    assert rules["grid"][0] == 0
    # at least two CTAs to a tile, at most one to a row block (4,096 / 256)
    assert set(rules["split"]) == {1, 2, 3, 4}


def test_the_graph_key_settles_the_launch(rules):
    launch = {}
    for key, split, grid in zip(rules["dia"], rules["split"], rules["grid"]):
        launch.setdefault(int(key), set()).add((int(split), int(grid)))
    launch.pop(0)  # no such kernel in the graph
    assert all(len(v) == 1 for v in launch.values())
    # the grid alone does not: one of 512 CTAs stands for several splits
    assert len({s for s, g in set().union(*launch.values()) if g == 512}) > 1
