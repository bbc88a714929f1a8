"""The default grids of the searches, by the graph's size (a fake CUDA runtime,
fake_cuda.py, with four blocks an SM on 148 SMs)."""
from __future__ import annotations

import subprocess

import fake_cuda
import pytest

PROGRAM = r"""
#include "%s.cu"
#include <cstdlib>

extern "C" int on_occupancy(const char *) { return 4; }

namespace g5 {
int set_error(int code, const char *, ...) { return code; }
void clear_error() {}
int deverr_to_status(unsigned, const char *) { return G5_OK; }
int device_info(DeviceInfo *out) {
    *out = DeviceInfo{0, 148, 2048};
    return G5_OK;
}
unsigned long long wait_limit_ns() { return 1; }
int persistent_kernel_setup(const void *) { return G5_OK; }
int l2_persist_window(uint64_t, uint64_t *bytes) { return *bytes = 0, G5_OK; }
int scan_u32_to_u64(const unsigned *, uint64_t, uint64_t *, uint64_t *, cudaStream_t) { return G5_OK; }
}
extern "C" const char *g5_last_error(void) { return ""; }
"""

BFS = PROGRAM % "bfs" + r"""
extern "C" void on_launch(const char *, void **) {}
// argv: vertices ...  Prints the default grid of each.
int main(int argc, char **argv) {
    for (int i = 1; i < argc; ++i) {
        int32_t blocks = 0, most = 0;
        if (g5_bfs_grid(atoll(argv[i]), &blocks, &most)) return 1;
        printf("%d\n", blocks);
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def bfs(tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("bfs_grid"), BFS)


def test_bfs_grid_by_vertices(bfs):
    want = {1: 1, 255: 1, 4096: 16, 16384: 64, 148 * 256: 148, 500_000: 148, 850_000: 207, 1_000_000: 244,
            1_300_000: 296, 2_000_000: 296, 3_000_000: 366, 4_194_304: 512, 1 << 25: 592, 1 << 31: 592}
    out = subprocess.run([bfs, *map(str, want)], check=True, capture_output=True, text=True).stdout
    assert [int(x) for x in out.split()] == list(want.values())
