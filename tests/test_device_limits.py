"""What a process remembers of a kernel's limits belongs to one device: csrc/device_limits.h, compiled with the host compiler and driven by made-up
devices, and a look at the sources for limits that are raised past it."""

from __future__ import annotations

import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "borrowed_compute_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "device_limits.h"
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main() {
    static BcDeviceLimits a, b;
    int calls = 0, had[66] = {}, fail = 0;
    auto on = [&](BcDeviceLimits& l, int device, int value) { return l.at_least(device, value, [&](int v) { calls++; if (fail) return fail; had[device] = v; return 0; }); };
    CHECK(on(a, 0, 100) == 0 && calls == 1 && had[0] == 100);
    CHECK(on(a, 0, 100) == 0 && on(a, 0, 60) == 0 && calls == 1);           // as much and less: nothing to do
    CHECK(on(a, 1, 100) == 0 && calls == 2 && had[1] == 100);               // another device has had nothing yet
    CHECK(on(a, 0, 200) == 0 && calls == 3 && had[0] == 200);               // more
    CHECK(on(b, 0, 50) == 0 && calls == 4);                                 // another kernel
    fail = 7;
    CHECK(on(a, 1, 300) == 7 && calls == 5);                                // what failed is not remembered
    fail = 0;
    CHECK(on(a, 1, 300) == 0 && calls == 6 && had[1] == 300);
    CHECK(on(a, 64, 10) == 0 && on(a, 64, 10) == 0 && calls == 8);          // beyond the known devices: asked anew
    static BcDeviceLimits shared;
    int most[8] = {};                                                       // threads with growing needs: the last word on a device is the largest
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; t++)
        threads.emplace_back([&, t] {
            for (int i = 1; i <= 2000; i++) shared.at_least(i % 8, 10 * i + t, [&](int v) { most[i % 8] = v; return 0; });
        });
    for (auto& t : threads) t.join();
    for (int d = 0; d < 8; d++) CHECK(most[d] >= 10 * (1993 + (d == 0 ? 7 : d - 1)) && shared.at_least(d, most[d], [](int) { return 9; }) == 0);
    return 0;
}
"""


def test_limits_are_kept_by_device(tmp_path):
    compiler = shutil.which("g++") or shutil.which("c++")
    if compiler is None:
        pytest.skip("no host compiler")
    source, program = tmp_path / "limits.cpp", tmp_path / "limits"
    source.write_text(PROGRAM)
    subprocess.run([compiler, "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(source), "-o", str(program)], check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout


def test_no_launcher_raises_a_limit_past_them():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")) and name != "common.cuh":
            with open(os.path.join(CSRC, name)) as f:
                text = f.read()
            assert "cudaFuncAttributeMaxDynamicSharedMemorySize" not in text, name
            assert not re.search(r"static (bool|int|size_t) (configured|raised|sixteen)\b", text), name
