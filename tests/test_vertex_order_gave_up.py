"""The vertex order's radix passes end with an error word when a look-back
wait gives up, and then leave parts of the order unwritten: the host reads
the word and launches nothing that indexes by the order.  The host code of
csr_sort.cu runs here on a fake CUDA runtime whose kernels do nothing, whose
device memory is host memory, and whose radix passes set the error word."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "cuda-graph-traversal_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

# The fake runtime: what nvcc's launches and the library's host code call.
RUNTIME = r"""
#include <cuda_runtime_api.h>
#include <cstring>
#include <map>
#include <string>

extern "C" void on_launch(const char *name, void **args);

// Kernels register from static constructors, before a global would be made.
static std::map<const void *, std::string> &names() {
    static std::map<const void *, std::string> m;
    return m;
}
static dim3 grid_, block_;
static size_t smem_;
static void *stream_;

extern "C" {
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, void *st) {
    grid_ = g, block_ = b, smem_ = s, stream_ = st;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
    *g = grid_, *b = block_, *s = smem_, *(void **)st = stream_;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) {
    static void *h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *fun, char *, const char *name, int, void *, void *, void *, void *,
                            int *) {
    names()[fun] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
char __cudaInitModule(void **) { return 0; }
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fun) {
    *k = (cudaKernel_t)fun;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *fun, dim3, dim3, void **args, size_t, cudaStream_t) {
    on_launch(names()[fun].c_str(), args);
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void **args, size_t s, cudaStream_t st) {
    return cudaLaunchKernel((const void *)k, g, b, args, s, st);
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int x, size_t n, cudaStream_t) {
    memset(d, x, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return ""; }
}
"""

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
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("vertex_order")
    (d / "runtime.cpp").write_text(RUNTIME)
    (d / "order.cu").write_text(PROGRAM)
    exe = d / "order"
    subprocess.run([NVCC, "-O1", "-Xptxas", "-O0", "-std=c++17", "-w", "-cudart", "none", "-gencode",
                    "arch=compute_100a,code=sm_100a", f"-I{CSRC}", f"-I{REPO}/include", "-o", str(exe),
                    str(d / "order.cu"), str(d / "runtime.cpp")], check=True)
    return exe


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
