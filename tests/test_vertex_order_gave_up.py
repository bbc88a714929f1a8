"""The vertex order's radix passes end with an error word when a look-back
wait gives up, and then leave parts of the order unwritten: the host reads
the word and launches nothing that indexes by the order.  The host code of
csr_sort.cu runs here on a fake CUDA runtime (fake_cuda.py) whose radix passes
set the error word."""
from __future__ import annotations

import subprocess

import fake_cuda
import pytest

PROGRAM = r"""
#include "csr_sort.cu"
#include <cstdlib>

static bool give_up = false;

extern "C" void on_launch(const char *name, void **args) {
    if (give_up && strstr(name, "csr_radix_pass")) *((g5::RxPass *)args[0])->err |= g5::SORTERR_WAIT;
    printf("%s\n", name);
}

namespace g5 {
int set_error(int code, const char *, ...) { return code; }
void clear_error() {}
int device_info(DeviceInfo *out) {
    *out = DeviceInfo{0, 148, 2048};
    return G5_OK;
}
unsigned long long wait_limit_ns() { return 1; }
int scan_u32_to_u64(const unsigned *, uint64_t, uint64_t *, uint64_t *, cudaStream_t) { return G5_OK; }
}

// argv: degree_order | renumber, 0 | 1 (give up).  Prints every kernel
// launched, then the status.
int main(int, char **argv) {
    const uint64_t n = 5000, e = 20000;
    auto mem = [](uint64_t bytes) { return calloc(bytes, 1); };
    uint64_t *rs = (uint64_t *)mem((n + 1) * 8), *rs2 = (uint64_t *)mem((n + 1) * 8), need = 0;
    int *col = (int *)mem(e * 4), *out = (int *)mem(e * 4);
    float *w = (float *)mem(e * 4), *w2 = (float *)mem(e * 4);
    unsigned *v[6];
    for (auto &p : v) p = (unsigned *)mem(n * 4);
    give_up = argv[2][0] == '1';
    int rc;
    if (argv[1][0] == 'd') {
        g5_csr_degree_order_workspace_size(n, e, &need);
        rc = g5_csr_degree_order(rs, col, n, e, out, mem(need), need, nullptr);
    } else {
        g5_csr_sssp_renumber_workspace_size(n, &need);
        rc = g5_csr_sssp_renumber(rs, col, w, v[0], v[1], n, e, v[2], v[3], rs2, out, w2, v[4], v[5], mem(need), need,
                                  nullptr);
    }
    printf("%d\n", rc);
    return 0;
}
"""

G5_ERR_TIMEOUT = -4


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("vertex_order"), PROGRAM)


@pytest.mark.parametrize("what,reads", [("degree_order", "rank_rows_warp"), ("renumber", "renumber_entries")])
@pytest.mark.parametrize("give_up", [0, 1])
def test_nothing_reads_an_unfinished_order(program, what, reads, give_up):
    *names, rc = subprocess.run([str(program), what, str(give_up)], check=True, capture_output=True,
                                text=True).stdout.split()
    assert any("csr_radix_pass" in x for x in names)
    if give_up:
        assert int(rc) == G5_ERR_TIMEOUT
        assert "csr_radix_pass" in names[-1], names[-1]  # nothing is launched after the passes
    else:
        assert int(rc) == 0 and any(reads in x for x in names) and any("vertex_perm" in x for x in names)
