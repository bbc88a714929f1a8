"""The packed counter of a list's big part (entries and chunks) over the sizes
that the searches accept: more than 2^24 rows longer than a chunk in one list
keep their slots and chunk bases in order."""
from __future__ import annotations

import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "cuda-graph-traversal_b200", "csrc")

PROGRAM = """
#include "g5_frontier.cuh"
using namespace g5;
// `rows` rows of `chunks` chunks each, appended `step` at a time (one add for
// each, as a warp makes it): 0 when every append got the next slots and chunks.
int main(int argc, char **argv) {
    const unsigned long long rows = atoll(argv[1]), chunks = atoll(argv[2]), step = atoll(argv[3]);
    unsigned long long big = 0;
    for (unsigned long long i = 0; i < rows; i += step) {
        const unsigned long long k = rows - i < step ? rows - i : step;
        if (big_count(big) != i || big_chunks(big) != i * chunks) return 1;
        big += big_pack((unsigned)k, (unsigned)(k * chunks));
    }
    return !(big_count(big) == rows && big_chunks(big) == rows * chunks);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("packing")
    src, exe = d / "packing.cpp", d / "packing"
    src.write_text("#include <cstdlib>\n" + PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-w", f"-I{CSRC}", f"-I{REPO}/include", "-I/usr/local/cuda/include",
                    "-o", str(exe), str(src)], check=True)
    return exe


# 2^25 vertices of degree 64 in chunks of 32; the first count that 24 bits do
# not hold; every vertex of the largest graph with one chunk each; a hub.
@pytest.mark.parametrize("rows,chunks,step", [(1 << 25, 2, 1), ((1 << 24) + 1, 9, 32), (1 << 31, 1, 32),
                                              (1, (1 << 32) - 1, 1), ((1 << 31) - 1, 2, 31)])
def test_slots_and_chunks_in_order(program, rows, chunks, step):
    assert subprocess.run([str(program), str(rows), str(chunks), str(step)]).returncode == 0
