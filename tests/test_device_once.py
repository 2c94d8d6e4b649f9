"""bg_deviceonce.h: an attribute set per device, once, also when several
threads meet there; a failed attempt is made again."""
import os
import subprocess

from brian_b200 import build as engine_build

SRC = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "bg_deviceonce.h"
int main() {
    DeviceOnce once;
    int a = 0, b = 0;
    std::atomic<int> sets[3][2] = {};
    std::vector<std::thread> th;
    for (int t = 0; t < 16; ++t)
        th.emplace_back([&] {
            for (int r = 0; r < 1000; ++r)
                for (int dev = 0; dev < 3; ++dev)
                    for (int k = 0; k < 2; ++k)
                        if (!once(dev, k ? (const void *)&a : (const void *)&b, [&] { ++sets[dev][k]; return true; })) return;
        });
    for (auto &t : th) t.join();
    for (auto &d : sets) for (auto &n : d) if (n != 1) return 1;
    DeviceOnce again;
    int tries = 0;
    if (again(0, &a, [&] { ++tries; return false; })) return 2;
    if (!again(0, &a, [&] { ++tries; return true; }) || !again(0, &a, [&] { ++tries; return true; }) || tries != 2) return 3;
    std::puts("ok");
    return 0;
}
"""


def test_once_per_device(tmp_path):
    src = tmp_path / "once.cpp"
    src.write_text(SRC)
    exe = str(tmp_path / "once")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I", engine_build.CSRC, str(src), "-o", exe])
    assert subprocess.run([exe], capture_output=True, text=True, timeout=60).stdout.strip() == "ok"


def test_no_process_wide_flag_in_the_training_launches():
    """The attributes of the training kernels belong to a device: no launch
    keeps whether it has set them in a flag of the whole process."""
    with open(os.path.join(engine_build.CSRC, "bg_mlp.cu")) as f:
        assert "static bool" not in f.read()
