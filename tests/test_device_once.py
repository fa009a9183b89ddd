"""csrc/device_once.h on the CPU: what belongs to a device is set on every device of the process."""
import os
import subprocess

from conftest import ROOT

PROGRAM = r"""
#include "device_once.h"
#include <cstdio>
#include <thread>
#include <vector>
int main()
{
    DeviceOnce once;
    int sets[70] = {}, fail = 1;
    auto set_on = [&](int d) { return once.run(d, [&]() { sets[d]++; return 0; }); };
    // a failure is handed on and tried again
    if (once.run(3, [&]() { sets[3]++; return fail; }) != 1) return 1;
    for (int round = 0; round < 3; round++)
        for (int d : {0, 1, 3, 63, 64})
            if (set_on(d)) return 2;
    if (sets[0] != 1 || sets[1] != 1 || sets[3] != 2 || sets[63] != 1 || sets[64] != 3) return 3;
    // threads that meet: nobody passes before a set() of its device has returned
    DeviceOnce shared;
    std::atomic<int> ready[8] = {}, early{0};
    std::vector<std::thread> all;
    for (int t = 0; t < 32; t++)
        all.emplace_back([&, t]() {
            shared.run(t % 8, [&]() { std::this_thread::yield(); ready[t % 8] = 1; return 0; });
            early += ready[t % 8] == 0;
        });
    for (auto &t : all) t.join();
    return early ? 4 : 0;
}
"""


def test_set_once_on_each_device(tmp_path):
    (tmp_path / "once.cc").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "nncp-metal_b200", "csrc"), "-o", str(tmp_path / "once"),
                    str(tmp_path / "once.cc")], check=True)
    assert subprocess.run([str(tmp_path / "once")]).returncode == 0
