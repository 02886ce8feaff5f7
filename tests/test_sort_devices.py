"""The cooperative sort's grid and count tables on each device of a process: csrc/k_sort_coop.cu, as the build left it,
linked to a runtime of two devices that only answers the queries it makes (no GPU)."""
import os
import shutil
import subprocess

import pytest

from splatter_gb300 import build

MAIN = r"""
#include <cstddef>
#include <cstdint>
#include <cstdio>

namespace spl {
int sort_coop_grid();
size_t sort_coop_table_words(uint64_t n_cap);
}

static int device = 0;
static const int sms[2] = {100, 152};
static bool opted_in[2];
static int queries[2];

extern "C" {
int cudaGetDevice(int* d) { return *d = device, 0; }
int cudaDeviceGetAttribute(int* v, int, int d) { return *v = sms[d], 0; }
int cudaFuncSetAttribute(const void*, int, int bytes) { return opted_in[device] = bytes > 48 * 1024, 0; }
// two blocks of that much shared memory on a multiprocessor, none where the kernel was not allowed to have it
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    ++queries[device];
    return *n = opted_in[device] ? 2 : 0, 0;
}
}

int main() {
    for (int round = 0; round < 2; ++round)
        for (device = 0; device < 2; ++device) {
            const int grid = spl::sort_coop_grid(), want = 2 * sms[device];
            const size_t words = spl::sort_coop_table_words(1u << 28), rows = want + (want + 15) / 16;
            std::printf("device %d: %d blocks, %zu words\n", device, grid, words);
            if (!opted_in[device] || grid != want || words != rows * 256 || queries[device] != 1) return 1;
        }
    return 0;
}
"""


def test_each_device_has_its_own_grid(tmp_path):
    lib, compiler = "/usr/local/cuda/lib64", shutil.which("g++")
    if compiler is None or not os.path.isdir(lib):
        pytest.skip("no g++ or no CUDA runtime library")
    build.build()
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run([compiler, "-std=c++17", str(tmp_path / "main.cpp"), os.path.join(build.OUT, "k_sort_coop.cu.o"), "-L" + lib,
                    "-lcudart", "-Wl,-rpath," + lib, "-o", str(tmp_path / "main")], check=True)
    run = subprocess.run([str(tmp_path / "main")], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout + run.stderr
