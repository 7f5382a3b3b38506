"""What a process does once per device (opt-ins to shared memory belong to a device): device_once.h against a counting step, and that no
launcher keeps such an opt-in for the whole process."""
import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "jasmine_b200" / "csrc"

PROGRAM = r"""
#include "device_once.h"
#include <cstdio>
#include <thread>
#include <vector>
int main() {
    jsm::DeviceOnce once;
    int set[70] = {0};
    auto step = [&](int dev) { return once.run(dev, [&] { ++set[dev]; return 0; }); };
    for (int round = 0; round < 3; ++round)
        for (int dev : {0, 1, 63, 64}) if (step(dev) != 0) return 1;
    if (set[0] != 1 || set[1] != 1 || set[63] != 1 || set[64] != 3) return 2;  // beyond 63: every time
    jsm::DeviceOnce failing;
    int calls = 0;
    if (failing.run(2, [&] { ++calls; return 7; }) != 7 || failing.run(2, [&] { ++calls; return 0; }) != 0 || failing.run(2, [&] { ++calls; return 7; }) != 0 || calls != 2) return 3;
    jsm::DeviceOnce shared;
    std::atomic<int> ran[8];
    for (auto& r : ran) r = 0;
    std::vector<std::thread> threads;
    for (int i = 0; i < 8; ++i)
        threads.emplace_back([&, i] { for (int k = 0; k < 1000; ++k) shared.run((i + k) % 8, [&] { ran[(i + k) % 8]++; return 0; }); });
    for (auto& t : threads) t.join();
    for (auto& r : ran) if (r < 1 || r > 8) return 4;
    std::puts("ok");
    return 0;
}
"""


def test_steps_run_once_per_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.returncode


def test_every_opt_in_to_shared_memory_is_per_device():
    for f in sorted(CSRC.glob("*.cu*")):
        text = f.read_text()
        if f.name != "common.cuh":  # (allow_shared)
            assert "cudaFuncSetAttribute" not in text, f.name
        for line in re.findall(r".*allow_shared\((\w+),", text):
            assert re.search(r"static DeviceOnce [\w, ]*\b" + line + r"\b", text), (f.name, line)
