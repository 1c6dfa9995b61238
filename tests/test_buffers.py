"""csrc/buffers.hpp against a fake CUDA runtime whose allocations fail on demand (host only)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"

SOURCE = r"""
#include "gpesolver_b200/csrc/buffers.hpp"
#include <cstdio>
#include <cstdlib>

static int allowed = 0; // allocations that still succeed
extern "C" {
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) {
    if (allowed-- <= 0)
        return cudaErrorMemoryAllocation;
    *p = std::malloc(bytes);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaMalloc(void **, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void *) { return cudaSuccess; }
cudaError_t cudaMemset(void *, int, size_t) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "out of memory"; }
}

int main() {
    gpe::MappedBuf<double> b;
    allowed = 1;
    b.alloc(5);
    int code = 0;
    try {
        b.alloc(50); // grows: fails
    } catch (const gpe::Error &e) {
        code = e.code;
    }
    // a buffer without memory holds nothing: a caller that asks for its size allocates again
    std::printf("%d %zu %d\n", code, b.n, b.p == nullptr);
    allowed = 1;
    b.alloc(7);
    std::printf("%zu %d %g\n", b.n, b.p != nullptr, b[6]);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="needs g++ and the CUDA headers")
def test_failed_growth_leaves_an_empty_mapped_buffer(tmp_path):
    src, exe = tmp_path / "buf.cpp", tmp_path / "buf"
    src.write_text(SOURCE)
    subprocess.check_call(["g++", "-std=c++17", "-I", ROOT, "-I", CUDA, "-o", str(exe), str(src)])
    out = subprocess.check_output([str(exe)], text=True).split("\n")
    assert out[0] == "6 0 1"  # GPE_ERR_NOMEM, no elements, no memory
    assert out[1] == "7 1 0"
