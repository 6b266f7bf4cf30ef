"""A scratch buffer whose growth failed (out of device memory) is gone: the next
call allocates it again instead of taking the freed one's size for it.  Read
from the source, since running out of device memory disturbs the GPU's other
users."""
from __future__ import annotations

import re

from conftest import ROOT

ENGINE = ROOT / "edegpredict-engine-rotary_b200" / "csrc" / "mpm_engine.cu"


def test_a_failed_growth_leaves_no_size_behind():
    src = ENGINE.read_text()
    grow = src[src.index("mpm_status grow("):src.index("static constexpr bool kPosLo")]
    assert grow.index("cudaFree(p)") < grow.index("have = 0") < grow.index("cudaMalloc(&p")
    for buf in ("gen", "stage"):
        tests = re.findall(r"if \(([^;{]*\b%s_bytes < need)\)" % buf, src)
        assert tests and all(t.startswith(f"!d_{buf} || ") for t in tests), (buf, tests)
