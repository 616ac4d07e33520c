"""The shared-memory limit of the sweeps against a runtime of two devices that is made up here (no GPU)."""

import glob
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "subsetix_b200", "csrc")

RUNTIME = """
#pragma once
enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1 };
enum cudaFuncAttribute { cudaFuncAttributeMaxDynamicSharedMemorySize };
cudaError_t cudaGetDevice(int*);
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int);
"""

MAIN = """
#include "sx_smem_limit.h"
#include <thread>
#include <unistd.h>
thread_local int current = 0;
int limit[70], calls;
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int bytes)
{
    if (bytes > 232448) return cudaErrorInvalidValue;
    usleep(200);  // a window for another thread's smaller request
    limit[current] = bytes;
    ++calls;
    return cudaSuccess;
}
int launches(SxSmemLimit& l, int device, int bytes)  // whether a launch would be accepted
{
    current = device;
    return l.raise(&l, bytes) == cudaSuccess && bytes <= limit[device];
}
int main()
{
    static SxSmemLimit a;
    if (!launches(a, 0, 100000) || !launches(a, 1, 60000) || !launches(a, 1, 100000) || !launches(a, 0, 60000)) return 1;
    if (calls != 3 || launches(a, 0, 300000) || !launches(a, 0, 100000) || !launches(a, 69, 50000)) return 2;
    for (int round = 0; round < 50; ++round) {
        SxSmemLimit b;
        limit[0] = 0;
        int ok[2];
        std::thread t([&] { ok[0] = launches(b, 0, 50000 + round); });
        ok[1] = launches(b, 0, 90000);
        t.join();
        if (!ok[0] || !ok[1] || limit[0] != 90000) return 3;
    }
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_limit_per_device_and_thread(tmp_path):
    (tmp_path / "cuda_runtime_api.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "limit"
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", str(tmp_path), "-I", CSRC, str(tmp_path / "main.cpp"), "-o",
                    str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_sweeps_keep_no_limit_of_their_own():
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        src = open(path).read()
        assert "static int configured" not in src, path
