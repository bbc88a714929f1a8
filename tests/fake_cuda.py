"""A fake CUDA runtime for the host code of the library's sources, on a machine
without a GPU: launches are reported to the test and run nothing, device memory
is host memory, every call succeeds."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "cuda-graph-traversal_b200", "csrc")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"

# What nvcc's launches and the library's host code call.
RUNTIME = r"""
#include <cuda_runtime_api.h>
#include <cstring>
#include <map>
#include <string>

// What a test gives: called for every launch, and asked for a kernel's blocks an SM.
extern "C" void on_launch(const char *name, void **args);
extern "C" __attribute__((weak)) int on_occupancy(const char *) { return 1; }

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
cudaError_t cudaLaunchCooperativeKernel(const void *fun, dim3 g, dim3 b, void **args, size_t s, cudaStream_t st) {
    return cudaLaunchKernel(fun, g, b, args, s, st);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *fun, void **args) {
    return cudaLaunchKernel(fun, c->gridDim, c->blockDim, args, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *fun, int, size_t) {
    *n = on_occupancy(names()[fun].c_str());
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *fun, int b, size_t s, unsigned) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, fun, b, s);
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


def build(folder, program: str) -> str:
    """Builds `program` (CUDA C++ that includes the library sources under test
    and defines on_launch) against the fake runtime; returns the executable."""
    if not os.path.exists(NVCC):
        pytest.skip("no nvcc")
    (folder / "runtime.cpp").write_text(RUNTIME)
    (folder / "program.cu").write_text(program)
    exe = str(folder / "program")
    subprocess.run([NVCC, "-O0", "-Xcicc", "-O0", "-Xptxas", "-O0", "-std=c++17", "-w", "-cudart", "none", "-gencode",
                    "arch=compute_100a,code=sm_100a", f"-I{CSRC}", f"-I{REPO}/include", "-o", exe,
                    # what the program never calls need not be here
                    "-Xlinker", "--unresolved-symbols=ignore-all", str(folder / "program.cu"),
                    str(folder / "runtime.cpp")], check=True)
    return exe
