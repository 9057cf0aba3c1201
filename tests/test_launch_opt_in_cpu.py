"""Launch attributes are set once on every device that launches a kernel, whichever thread comes first (the CUDA calls
are stand-ins)."""

import os
import shutil
import subprocess

import pytest

SOURCE = r"""
#include <atomic>
#include <thread>
#include <vector>
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize };
enum { cudaSuccess = 0 };
static thread_local int device = 0;
static std::atomic<int> sets[4][2];
static bool refuse = false;
static int cudaGetDevice(int* d) { *d = device; return 0; }
static void first() {}
static void second() {}
static int cudaFuncSetAttribute(void (*k)(), cudaFuncAttribute, int) {
    if (refuse) return 1;
    ++sets[device][k == second];
    return 0;
}
#include "opt_in.cuh"
#define CHECK(x) do { if (!(x)) return __LINE__; } while (0)
int main() {
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    refuse = true;
    CHECK(!lme::opt_in<first>(attr, 1));
    refuse = false;
    for (int i = 0; i < 3; ++i)
        for (device = 0; device < 3; ++device) CHECK(lme::opt_in<first>(attr, 1));
    for (int d = 0; d < 3; ++d) CHECK(sets[d][0] == 1 && sets[d][1] == 0);
    std::vector<std::thread> ts;
    for (int i = 0; i < 8; ++i) ts.emplace_back([&, i] { device = i % 4; lme::opt_in<second>(attr, 1); });
    for (auto& t : ts) t.join();
    for (int d = 0; d < 4; ++d) CHECK(sets[d][1] >= 1);
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_every_device_is_opted_in(tmp_path):
    import lm_engine_b200

    kernels = os.path.join(os.path.dirname(lm_engine_b200.__file__), "csrc", "kernels")
    src, exe = tmp_path / "opt_in.cpp", tmp_path / "opt_in"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", kernels, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
