"""How the multi-RHS kernels of the diagonal form cut their work
(batch_shape.cuh), compiled for the host: every (row, column) belongs to one
lane of one CTA, and the grid is counted without overflow, so that the launch
can refuse one that does not fit."""
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

_MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "batch_shape.cuh"
int main() {
    long long n, k;
    int vec, sms;
    while (std::scanf("%lld %lld %d %d", &n, &k, &vec, &sms) == 4) {
        const nm::DiaBatchShape b = nm::dia_batch_shape(n, k, vec, sms);
        std::printf("%d %d %d %d %lld\n", b.lg, b.nchunk, b.chunk_cols, b.run, (long long)b.grid);
    }
}
"""


@pytest.fixture(scope="module")
def shapes(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    assert cxx, "no host compiler"
    d = tmp_path_factory.mktemp("batch_shape")
    (d / "main.cpp").write_text(_MAIN)
    subprocess.run([cxx, "-std=c++17", "-x", "c++", f"-I{ROOT / 'num_b200' / 'csrc'}",
                    str(d / "main.cpp"), "-o", str(d / "main")], check=True)

    def run(cases):
        text = "\n".join(" ".join(map(str, c)) for c in cases)
        out = subprocess.run([str(d / "main")], input=text, check=True, capture_output=True,
                             text=True).stdout
        return [[int(v) for v in line.split()] for line in out.splitlines()]
    return run


def test_every_row_and_column_once(shapes):
    cases = [(n, k, vec, 148) for n in (1, 7, 128, 191, 193, 5000)
             for k in list(range(1, 70)) + [127, 128, 129, 1000] for vec in (1, 2)
             if k % vec == 0]
    for (n, k, vec, _), (lg, nchunk, cols, run, grid) in zip(cases, shapes(cases)):
        step = 128 >> lg
        assert run % step == 0 and 0 < run <= 192
        assert grid == -(-n // run) * nchunk
        seen = np.zeros(k, int)
        for chunk in range(nchunk):
            for lane in range(1 << lg):
                c = chunk * cols + lane * vec
                if c < min(k, (chunk + 1) * cols):
                    seen[c:c + vec] += 1
        assert np.all(seen == 1)


def test_a_grid_beyond_the_launch_is_counted(shapes):
    # 2^31 - 1 columns of 4,096 rows: 22 runs of 134,217,728 chunks
    (lg, nchunk, _, run, grid), = shapes([(4096, 2**31 - 1, 1, 148)])
    assert lg == 4 and nchunk == 2**27 and run == 192 and grid == 22 * 2**27 > 2**31 - 1
