"""The kept dynamic shared memory limits (max_dynamic_smem_set, bats_gb300/csrc/abi_util.cu), compiled for the host with stand-ins for
the CUDA calls: nothing is thrown when memory is short (a C caller could not catch it), and a limit is never lowered, for more
kernels than are remembered, on two devices."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <new>
#include <utility>
static bool armed = false;
void* operator new(std::size_t n) { if (armed) throw std::bad_alloc(); return std::malloc(n); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
typedef int cudaError_t;
enum { cudaSuccess = 0, cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
struct cudaFuncAttributes { int maxDynamicSharedSizeBytes; };
static int device = 0, limit[2][700], calls = 0;
static char kernels[700];
static cudaError_t cudaGetDevice(int* d) { *d = device; return 0; }
static cudaError_t cudaFuncSetAttribute(const void* f, int, int bytes) {
    limit[device][(const char*)f - kernels] = bytes;
    ++calls;
    return 0;
}
static cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* f) {
    a->maxDynamicSharedSizeBytes = limit[device][(const char*)f - kernels];
    return 0;
}
namespace bats {
@SOURCE@
}
int main() {
    armed = true;
    for (int round = 0; round < 3; ++round)
        for (device = 0; device < 2; ++device)
            for (int k = 0; k < 700; ++k) {
                const int before = limit[device][k], ask = round == 1 ? 1000 : 2000 + round * 10 + k;
                if (bats::max_dynamic_smem_set(kernels + k, ask) != 0) return 1;
                const int now = limit[device][k];
                if (now < ask || now < before) return 2;
            }
    const int n = calls;  // asked again for what is set: no call
    device = 0;
    for (int k = 0; k < 300; ++k)
        if (bats::max_dynamic_smem_set(kernels + k, 500) != 0) return 3;
    return calls == n ? 0 : 4;
}
"""


def test_limits_are_kept_without_memory(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    text = open(os.path.join(ROOT, "bats_gb300", "csrc", "abi_util.cu")).read()
    body = text[text.index("int max_dynamic_smem_set("):text.index("bool pdl_enabled()")]
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(PROGRAM.replace("@SOURCE@", body))
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
