"""A kernel's shared-memory size is allowed on every device that launches it,
and a refusal is not kept (csrc/smem_limit.hpp): against a stand-in for the
CUDA runtime with two devices."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sycldb_gb300", "csrc")

PROGRAM = r"""
#include <cassert>
#include <cstdio>
#include <thread>
#include <vector>
#include "smem_limit.hpp"

static thread_local int device = 0;
static std::atomic<int> asked[2];   // per device
static std::atomic<bool> refuse{false};

extern "C" cudaError_t cudaGetDevice(int *d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute a, int bytes)
{
    assert(a == cudaFuncAttributeMaxDynamicSharedMemorySize && bytes == 61440);
    if (refuse) return cudaErrorInvalidValue;
    asked[device]++;
    return cudaSuccess;
}

static void k0(int) {}
static void k1(int) {}

int main()
{
    sdb::SmemLimit limit;
    refuse = true;
    assert(!limit.allow(61440, k0, k1));
    refuse = false;
    for (int i = 0; i < 3; i++) assert(limit.allow(61440, k0, k1));  // the refusal was not kept
    assert(asked[0] == 2 && asked[1] == 0);
    device = 1;
    for (int i = 0; i < 3; i++) assert(limit.allow(61440, k0, k1));  // another device of the process
    assert(asked[0] == 2 && asked[1] == 2);
    refuse = true;
    assert(limit.allow(61440, k0, k1));
    refuse = false;
    sdb::SmemLimit shared;  // several threads, a device each
    std::vector<std::thread> t;
    for (int d = 0; d < 8; d++)
        t.emplace_back([&, d] {
            device = d & 1;
            for (int i = 0; i < 1000; i++) assert(shared.allow(61440, k0));
        });
    for (auto &x : t) x.join();
    assert(asked[0] >= 3 && asked[1] >= 3);
    std::puts("ok");
}
"""


def test_every_device_and_no_kept_refusal(tmp_path):
    gxx = shutil.which("g++")
    inc = "/usr/local/cuda/include"
    if not gxx or not os.path.exists(os.path.join(inc, "cuda_runtime_api.h")):
        pytest.skip("no host compiler or CUDA headers")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", inc, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "ok\n"


def test_every_launch_site_goes_through_it():
    """No call site sets the attribute by itself."""
    for name in os.listdir(CSRC):
        if name.endswith((".cu", ".cuh", ".cpp")):
            text = open(os.path.join(CSRC, name)).read()
            assert not re.search(r"cudaFuncAttributeMaxDynamicSharedMemorySize", text), name
