"""Failed allocations and launches while the compaction's tables are built (CPU): the next call builds them again, and no
pass runs on tables that are missing or not filled.  The program below compiles compact.cuh with an allocator that
fails on demand and runs without a device, so every launch and memset fails as well."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "compact.cuh"
bool fail = true;
namespace granite_b200 {
cudaError_t dev_alloc(void **p, size_t bytes) {
    if (fail) return cudaErrorMemoryAllocation;
    *p = malloc(bytes);
    return cudaSuccess;
}
void dev_free(void *p) { free(p); }
}
extern "C" int gr_host_free(void *) { return 0; }
using namespace granite_b200;
#define WANT(x) if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; }
int main() {
    int devices = 0;
    WANT(cudaGetDeviceCount(&devices) != cudaSuccess || devices == 0);
    Bricks b;
    WANT(b.build(3, 64, 64, 64, 0) == cudaErrorMemoryAllocation);
    WANT(b.nbins == 0);
    fail = false;
    for (int k = 0; k < 2; ++k) {   // memory, but no launch
        WANT(b.build(3, 64, 64, 64, 0) != cudaSuccess);
        WANT(b.nbins == 0);
    }
    CompactScratch s;
    fail = true;
    WANT(s.alloc(1000) == cudaErrorMemoryAllocation);
    fail = false;
    for (int k = 0; k < 2; ++k) WANT(s.alloc(1000) != cudaSuccess);   // memory, but not zeroed
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("nvcc") is None, reason="needs nvcc")
def test_tables_are_built_again_after_a_failure(tmp_path):
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(PROGRAM)
    csrc = os.path.join(ROOT, "pygranite_b200", "csrc")
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", csrc, str(src), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], env=dict(os.environ, CUDA_VISIBLE_DEVICES=""), capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
