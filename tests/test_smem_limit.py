"""A kernel's shared-memory limit is raised once on every device that launches it (csrc/smem_limit.hpp), compiled here against
stand-ins for the two runtime calls."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <map>
#include <mutex>
#include <thread>
#include <vector>
#include "smem_limit.hpp"

static thread_local int t_device = 0;
static std::mutex g_mu;
static std::map<int, int> g_asked;          // device -> calls
static bool g_refuse = false;
extern "C" cudaError_t cudaGetDevice(int* dev) { *dev = t_device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int bytes) {
    std::lock_guard<std::mutex> lock(g_mu);
    ++g_asked[t_device];
    return g_refuse || bytes != 1000 ? cudaErrorInvalidValue : cudaSuccess;
}
static void kernel(int) {}

#define EXPECT(what) do { if (!(what)) { std::printf("line %d: %s\n", __LINE__, #what); return 1; } } while (0)
int main() {
    static simnets::SmemLimit limit;
    g_refuse = true;
    EXPECT(limit.raise(kernel, 1000) == cudaErrorInvalidValue);
    g_refuse = false;
    EXPECT(limit.raise(kernel, 1000) == cudaSuccess && g_asked[0] == 2);            // a refusal is not remembered
    EXPECT(limit.raise(kernel, 1000) == cudaSuccess && g_asked[0] == 2);
    for (int d : {1, 5, 63, 64, 127}) {
        t_device = d;
        EXPECT(limit.raise(kernel, 1000) == cudaSuccess && g_asked[d] == 1);
        EXPECT(limit.raise(kernel, 1000) == cudaSuccess && g_asked[d] == (d < 64 ? 1 : 2));
    }
    std::vector<std::thread> threads;
    for (int i = 0; i < 16; ++i)
        threads.emplace_back([i] { t_device = 10 + i % 4; for (int k = 0; k < 1000; ++k) limit.raise(kernel, 1000); });
    for (auto& t : threads) t.join();
    for (int d = 10; d < 14; ++d) EXPECT(g_asked[d] >= 1 && g_asked[d] <= 4);       // (threads that meet may each ask)
    return 0;
}
"""


def test_the_limit_is_raised_on_every_device(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", str(src), "-o", str(exe), "-isystem", include,
                           "-I", os.path.join(ROOT, "simnets_tf_b200", "csrc")])
    got = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert got.returncode == 0, got.stdout


def test_no_launcher_keeps_a_flag_for_all_devices():
    csrc = os.path.join(ROOT, "simnets_tf_b200", "csrc")
    for name in sorted(os.listdir(csrc)):
        assert not re.search(r"static\s+bool\s+\w+\s*(=|;)", open(os.path.join(csrc, name)).read()), name
