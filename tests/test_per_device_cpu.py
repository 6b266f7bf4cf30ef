"""What the step kernel's launches remember per device (csrc/mpm_per_device.h),
in a small host program: worked out once for each device, asked again while it
is not known, never taken from another device, from several threads too.  The
step kernel keeps no attribute of a launch in a plain static: a process that
steps handles on two devices has to set the shared-memory size on both."""
from __future__ import annotations

import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "edegpredict-engine-rotary_b200" / "csrc"

PROG = r"""
#include <cassert>
#include <cstdio>
#include <thread>
#include <vector>
#include "mpm_per_device.h"
using mpmb::PerDevice;

int main() {
    static PerDevice fit;
    int calls = 0;
    auto f = [&](int v) { return [&calls, v] { ++calls; return v; }; };
    assert(fit.get(0, f(3)) == 3 && calls == 1);
    assert(fit.get(0, f(9)) == 3 && calls == 1);    // known
    assert(fit.get(1, f(0)) == 0 && calls == 2);    // the query failed: asked again
    assert(fit.get(1, f(2)) == 2 && calls == 3);
    assert(fit.get(0, f(9)) == 3 && fit.get(1, f(9)) == 2 && calls == 3);
    assert(fit.get(PerDevice::kMaxDevices, f(5)) == 5 && fit.get(-1, f(6)) == 6 && calls == 5);   // not kept
    assert(fit.get(PerDevice::kMaxDevices, f(7)) == 7);
    static PerDevice shared;
    std::vector<std::thread> t;
    std::atomic<int> bad{0};
    for (int k = 0; k < 8; ++k)
        t.emplace_back([&, k] {
            for (int q = 0; q < 10000; ++q)
                if (shared.get((k + q) % 4, [&] { return 10 + (k + q) % 4; }) != 10 + (k + q) % 4) ++bad;
        });
    for (auto& x : t) x.join();
    assert(bad == 0);
    std::puts("OK");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_once_per_device(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROG)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", str(CSRC), str(src), "-o", str(exe), "-pthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stderr


def test_the_launches_keep_nothing_for_the_whole_process():
    src = (CSRC / "mpm_step.cu").read_text()
    assert not re.search(r"\bstatic (bool|int|size_t) \w+ *(=|;)", src)
