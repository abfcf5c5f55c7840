"""Values kept per CUDA device (csrc/sx_per_device.h): each device finds its own,
once, with several threads; and no kernel limit is raised once per process."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "starlab-physics_gb300", "csrc")

SOURCE = r"""
#include "sx_per_device.h"
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
int main() {
    static sx::PerDevice memo;
    std::atomic<int> found[4] = {};
    std::vector<std::thread> threads;
    std::atomic<int> wrong{0};
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] {
            for (int k = 0; k < 1000; ++k) {
                const int dev = (k + t) % 4;
                if (memo.get(dev, [&] { ++found[dev]; return dev == 2 ? 0 : 100 + dev; }) != (dev == 2 ? 0 : 100 + dev))
                    ++wrong;
            }
        });
    for (auto& t : threads) t.join();
    int far = 0;
    for (int k = 0; k < 3; ++k) memo.get(k == 0 ? -1 : 1000, [&] { return ++far; });
    std::printf("%d %d %d %d %d %d\n", (int)found[0], (int)found[1], (int)found[2], (int)found[3], (int)wrong, far);
}
"""


def test_each_device_has_its_own(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    (tmp_path / "t.cpp").write_text(SOURCE)
    subprocess.run([gxx, "-std=c++17", "-pthread", "-I", CSRC, str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")],
                   check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["1", "1", "1", "1", "0", "3"]


def test_no_attribute_is_set_once_per_process():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            src = open(os.path.join(CSRC, name)).read()
            for m in re.finditer(r"call_once\(", src):
                assert "cudaFuncSetAttribute" not in src[m.start():m.start() + 800], name
