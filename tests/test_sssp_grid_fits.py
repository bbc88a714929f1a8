"""A search launches two cooperative kernels with one grid, so the largest grid
is the smaller of what fits of either: asked for both, here with a fake CUDA
runtime (fake_cuda.py) that answers differently for the two."""
from __future__ import annotations

import subprocess

import fake_cuda
import pytest

PROGRAM = r"""
#include "sssp.cu"
#include <cstdlib>
#include <cstring>

static int fits_buckets, fits_finish;
extern "C" void on_launch(const char *, void **) {}
extern "C" int on_occupancy(const char *name) { return strstr(name, "finish") ? fits_finish : fits_buckets; }

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
}
extern "C" const char *g5_last_error(void) { return ""; }

// argv: blocks an SM of the bucketed and of the finish kernel.  Prints the
// largest grid and the one for 2^22 vertices.
int main(int, char **argv) {
    fits_buckets = atoi(argv[1]), fits_finish = atoi(argv[2]);
    int32_t blocks = 0, most = 0;
    if (g5_sssp_grid(1ull << 22, &blocks, &most)) return 1;
    printf("%d %d\n", most, blocks);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("sssp_grid"), PROGRAM)


@pytest.mark.parametrize("buckets,finish", [(3, 3), (3, 2), (2, 4), (1, 1)])
def test_grid_fits_both_kernels(program, buckets, finish):
    out = subprocess.run([program, str(buckets), str(finish)], check=True, capture_output=True, text=True).stdout
    assert out.split() == [str(148 * min(buckets, finish))] * 2
