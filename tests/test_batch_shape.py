"""How the multi-RHS kernels of the diagonal form cut their work
(batch_shape.cuh), compiled for the host: every (row, column) belongs to one
lane of one CTA, the grid is counted without overflow, so that the launch
can refuse one that does not fit, and the CSR kernels keep the products that
they are faster at."""
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
        const nm::CsrBatchShape c = nm::csr_batch_shape(k, vec);
        std::printf("%d %d %d %d %lld %d %d %lld", b.lg, b.nchunk, b.chunk_cols, b.run,
                    (long long)b.grid, c.tpr_log2, c.ch, (long long)c.slots);
        for (int nd : {3, 7, 9, 16})
            for (int f = 0; f < 3; ++f)  // ragged, full, full and constant
                std::printf(" %d", int(nm::dia_batch_takes(n, nd, f > 0, f > 1, k, vec, b)));
        std::printf("\n");
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
    for (n, k, vec, _), (lg, nchunk, cols, run, grid, *_) in zip(cases, shapes(cases)):
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
    (lg, nchunk, _, run, grid, *_), = shapes([(4096, 2**31 - 1, 1, 148)])
    assert lg == 4 and nchunk == 2**27 and run == 192 and grid == 22 * 2**27 > 2**31 - 1


def test_the_csr_kernels_shape(shapes):
    cases = [(5000, k, vec, 148) for k in range(1, 600) for vec in (1, 2) if k % vec == 0]
    for (_, k, vec, _), (*_, tpr, ch, slots) in zip(cases, (s[:8] for s in shapes(cases))):
        groups = -(-k // vec)
        assert (1 << tpr) >= min(groups, 32) and (tpr == 0 or (1 << tpr - 1) < groups)
        assert ch in (1, 2, 4) and slots % (ch << tpr) == 0
        assert slots >= groups > slots - (ch << tpr)


def _routes(shapes, n, k):
    vec = 2 if k % 2 == 0 else 1
    row, = shapes([(n, k, vec, 148)])
    took = np.array(row[8:], bool).reshape(4, 3)
    return {nd: dict(zip(("ragged", "full", "constant"), t)) for nd, t in zip((3, 7, 9, 16), took)}


def test_who_takes_a_product(shapes):
    # one chunk of the CSR kernels' columns, or many of their lanes idle
    for n in (1000, 30_000, 300_000):
        for k in (1, 2, 3, 16, 31, 32, 33, 48, 64, 65, 80):
            assert all(all(v.values()) for v in _routes(shapes, n, k).values())
    # full rows of constant values stay, whatever the width
    for k in (63, 100, 127, 128, 256, 500):
        assert all(v["constant"] for v in _routes(shapes, 30_000, k).values())
    # four chunks: only those
    for k in (113, 127, 256):
        for v in _routes(shapes, 300_000, k).values():
            assert not v["ragged"] and not v["full"]
    # two chunks, nearly all lanes busy
    small, large = _routes(shapes, 30_000, 128), _routes(shapes, 300_000, 128)
    assert [small[d]["ragged"] for d in (3, 7, 9, 16)] == [True, False, False, False]
    assert [large[d]["ragged"] for d in (3, 7, 9, 16)] == [True, True, True, False]
    assert [small[d]["full"] for d in (3, 7, 9, 16)] == [True, True, True, False]
