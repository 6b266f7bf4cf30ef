"""The bound below which the step skips the flow stress (csrc/mpm_flow_bound.h)
never skips a particle that the flow stress itself would let yield: for every
temperature -- next to the melting point above all, where 1 - Ts^m is a few
roundings of 1 -- it lies below ylo times the smallest factor 1 - pow(Ts, m)
that a power within CUDA's error bounds (4 ulp in FP32, 2 ulp in FP64) gives.
A small host program walks the temperatures in both precisions."""
from __future__ import annotations

import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = ROOT / "edegpredict-engine-rotary_b200" / "csrc"

PROG = r"""
#include <cassert>
#include <cmath>
#include <cstdio>
#include <type_traits>
#include "mpm_flow_bound.h"
using namespace mpmb;

template <typename R> long check(double m, R ylo) {
    const R scale = flow_scale<R>(ylo, m);
    const int ulps = std::is_same<R, float>::value ? 4 : 2;
    long bad = 0, used = 0;
    auto at = [&](R Ts) {
        const long double p = powl((long double)Ts, (long double)(R)m);
        R pw = (R)p;
        for (int k = 0; k < ulps; ++k) pw = std::nextafter(pw, R(2));   // the largest power allowed
        const R tt = R(1) - pw;                                         // the smallest factor computed
        const R lim = flow_bound(scale, Ts);
        used += lim > R(0);
        if (lim > R(0) && lim > ylo * tt) ++bad;
    };
    R T = R(1);
    for (int k = 0; k < 4000; ++k) { at(T); T = std::nextafter(T, R(0)); }      // the last roundings below 1
    for (int k = 1; k < 32000; ++k) at((R)(1.0 - std::pow(10.0, -16.0 * k / 32000.0)));
    for (int k = 0; k <= 16000; ++k) at((R)(k / 16000.0));
    assert(used > 16000);
    return bad;
}

int main() {
    const double ms[] = {1.0 / 32.0, 0.05, 0.1, 0.3, 0.5, 0.8, 0.9, 0.999, 1.0, 1.001, 1.03, 1.1, 1.4, 2.0, 5.0};
    for (double m : ms)
        for (double y : {1.098e9, 3.0}) {
            const long f = check<float>(m, (float)y), d = check<double>(m, y);
            if (f || d) { std::printf("m %g ylo %g: %ld FP32, %ld FP64 temperatures above\n", m, y, f, d); return 1; }
        }
    for (double m : {0.0, -1.0, 0.01}) assert(flow_scale<float>(1e9f, m) == 0.0f && flow_scale<double>(1e9, m) == 0.0);
    // what it gives up is small: an unheated particle's bound is within 2e-4 of ylo
    assert(flow_bound(flow_scale<float>(1e9f, 1.03), 0.0f) > 0.9998e9f);
    std::puts("OK");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_the_bound_is_below_every_flow_stress(tmp_path):
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROG)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-ffp-contract=off", "-I", str(CSRC), str(src), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout + out.stderr
