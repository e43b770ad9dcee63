"""Kernel attributes belong to a device: they are set on each one of a process, by whichever thread comes first."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dcgan-cuda_b200", "csrc")

PROGRAM = r"""
#include "per_device.cuh"
#include <cstdio>
#include <thread>
#include <vector>
int main()
{
    dcg::OncePerDevice once;
    int runs[3] = {0, 0, 0};
    for (int pass = 0; pass < 3; ++pass)
        for (int dev = 0; dev < 3; ++dev)
            if (once(dev, [&] { return ++runs[dev] == 1 && dev == 2 ? 7 : 0; }) != (pass == 0 && dev == 2 ? 7 : 0)) return 1;
    if (runs[0] != 1 || runs[1] != 1 || runs[2] != 2) return 2;   // a failure is reported and tried again
    dcg::OncePerDevice shared;
    std::atomic<int> count{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t) threads.emplace_back([&, t] { for (int i = 0; i < 1000; ++i) shared((i + t) % 64, [&] { ++count; return 0; }); });
    for (auto& t : threads) t.join();
    if (count != 64) return 3;
    int beyond = 0;
    for (int i = 0; i < 2; ++i) shared(64 + i, [&] { ++beyond; return 0; }), shared(-1, [&] { ++beyond; return 0; });
    return beyond == 4 ? 0 : 4;
}
"""


def test_once_on_every_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", str(exe), str(src)])
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_attribute_is_set_once_per_process():
    for name in os.listdir(CSRC):
        if name.endswith((".cu", ".cuh")):
            text = open(os.path.join(CSRC, name)).read()
            for body in re.findall(r"call_once\((.*?)\n    \}\);", text, flags=re.S):
                assert "cudaFuncSetAttribute" not in body, name
