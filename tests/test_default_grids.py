"""The default grids and list tiles of the searches, by the graph's size (a fake
CUDA runtime, fake_cuda.py, with four blocks an SM on 148 SMs)."""
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

MSBFS = PROGRAM % "msbfs" + r"""
#include <cstring>
#include <sys/mman.h>
extern "C" void on_launch(const char *name, void **args) {
    if (strstr(name, "ms_persistent")) printf("%u\n", ((g5::MsArgs *)args[0])->nblocks);
}
// argv: vertices and CSR entries of a graph, ...  Prints the grid that a
// search of each is launched with.
int main(int argc, char **argv) {
    for (int i = 1; i + 1 < argc; i += 2) {
        const uint64_t n = atoll(argv[i]), e = atoll(argv[i + 1]), root = 0;
        uint64_t need = 0;
        if (g5_msbfs_workspace_size(n, e, 0, &need)) return 1;
        void *work = mmap(nullptr, need, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
        if (work == MAP_FAILED || g5_msbfs_run(n, e, 0, &root, 1, work, need, nullptr, nullptr, nullptr)) return 2;
        munmap(work, need);
    }
    return 0;
}
"""

SSSP = PROGRAM % "sssp" + r"""
#include <cstring>
#include <sys/mman.h>
extern "C" void on_launch(const char *name, void **args) {
    const g5::SsspArgs &a = *(g5::SsspArgs *)args[0];
    if (strstr(name, "sssp_persistent")) printf("%u %u\n", a.big_deg, a.chunk);
}
// argv: vertices, bucket width (rows split at 0.1) ...  Prints the tiles that
// a search of each is launched with.
int main(int argc, char **argv) {
    static uint64_t some[4];
    for (int i = 1; i + 1 < argc; i += 2) {
        const uint64_t n = atoll(argv[i]);
        uint64_t need = 0;
        if (g5_sssp_workspace_size(n, &need)) return 1;
        void *work = mmap(nullptr, need, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
        g5_sssp_params p = {};
        p.delta = (float)atof(argv[i + 1]);
        if (work == MAP_FAILED ||
            g5_sssp_traverse(some, (int32_t *)some, (float *)some, (uint32_t *)some, 0.1f, n, 0, (float *)some,
                             (int64_t *)some, work, need, &p, nullptr))
            return 2;
        munmap(work, need);
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


@pytest.fixture(scope="module")
def msbfs(tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("msbfs_grid"), MSBFS)


def test_batched_bfs_grid_by_entries_and_vertices(msbfs):
    want = [(2, 2, 148), (260_000, 33_280_000, 148), (600_000, 9_600_000, 148), (1_000_000, 32_000_000, 148),
            (4_000_000, 16_000_000, 296), (400_000, 51_200_000, 296), (4_000_000, 64_000_000, 296),
            (8_000_000, 64_000_000, 444), (1_000_000, 128_000_000, 592), (1 << 22, 1 << 27, 592)]
    out = subprocess.run([msbfs, *(str(x) for n, e, _ in want for x in (n, e))], check=True, capture_output=True,
                         text=True).stdout
    assert [int(x) for x in out.split()] == [b for _, _, b in want]


@pytest.fixture(scope="module")
def sssp(tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("sssp_tiles"), SSSP)


def test_sssp_tiles_by_vertices_and_rows(sssp):
    want = [(2000, 0.1, 64), (1 << 22, 0.1, 64), ((1 << 22) + 1, 0.1, 128), (1 << 24, 0.05, 128),
            ((1 << 24) + 1, 0.1, 256), (2000, 0.2, 256), (1 << 22, 0.11, 256), (1 << 25, 0.4, 256)]
    out = subprocess.run([sssp, *(str(x) for n, d, _ in want for x in (n, d))], check=True, capture_output=True,
                         text=True).stdout
    assert [int(x) for x in out.split()] == [t for _, _, t in want for _ in range(2)]
