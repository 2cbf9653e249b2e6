"""A kernel's shared-memory limit is raised on every device (csrc/smem_limit.h): compiled
for the host against a CUDA runtime of two devices that only counts, and no other place
in the sources that sets a kernel's attributes."""
import glob
import os
import shutil
import subprocess

import pytest

from fug30v0kxc_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "fug30v0kxc_gb300", "csrc")
CHECK = r"""
#include <stdio.h>
#include <thread>
#include <vector>
#include "smem_limit.h"
static thread_local int dev;
static int fail;
static std::atomic<int> calls[80];
extern "C" cudaError_t cudaGetDevice(int *d) { *d = dev; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int)
{
    if (fail) return cudaErrorInvalidValue;
    calls[dev]++;
    return cudaSuccess;
}
static int bad;
#define IS(a, b) do { int x_ = (a), y_ = (b); if (x_ != y_) { printf("line %d: %d, not %d\n", __LINE__, x_, y_); bad = 1; } } while (0)
int main()
{
    static SmemLimit a, b;
    int kern = 0;
    for (int r = 0; r < 3; r++)
        for (dev = 0; dev < 2; dev++) IS(a.raise(&kern, 100000), cudaSuccess);
    IS(calls[0], 1);
    IS(calls[1], 1);
    dev = 1;
    fail = 1;
    IS(b.raise(&kern, 1), cudaErrorInvalidValue);      // reported, and tried again
    fail = 0;
    IS(b.raise(&kern, 1), cudaSuccess);
    IS(calls[1], 2);
    dev = 70;
    for (int r = 0; r < 3; r++) a.raise(&kern, 1);
    IS(calls[70], 3);
    static SmemLimit c;
    std::vector<std::thread> t;
    for (int i = 0; i < 8; i++)
        t.emplace_back([i, &kern] { dev = 2 + i % 2; for (int r = 0; r < 1000; r++) c.raise(&kern, 1); });
    for (auto &x : t) x.join();
    IS(calls[2] >= 1 && calls[2] <= 4 && calls[3] >= 1 && calls[3] <= 4, 1);
    return bad;
}
"""


def test_once_per_device(tmp_path):
    cc = shutil.which("g++")
    if cc is None:
        pytest.skip("no C++ compiler")
    include = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(CHECK)
    subprocess.run([cc, "-std=c++17", "-O1", "-I", CSRC, "-I", include, str(src), "-o", str(exe), "-lpthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_nowhere_else():
    for path in glob.glob(os.path.join(CSRC, "*")):
        with open(path) as f:
            if os.path.basename(path) != "smem_limit.h":
                assert "cudaFuncSetAttribute" not in f.read(), path
