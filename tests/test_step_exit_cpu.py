"""Every CTA of the step kernel leaves through the kernel's end, where it
counts itself out of the work-item tickets: the launch's last CTA zeroes them
for the next launch.  A CTA that returned early (after a bounded wait ran out)
would leave the tickets of its launch behind, and later launches would skip
work items or hand one to two CTAs.  The wait itself cannot be made to run out
without damaging a copy in flight, so the source is read."""
from __future__ import annotations

import re

from conftest import ROOT

STEP = ROOT / "edegpredict-engine-rotary_b200" / "csrc" / "mpm_step.cu"


def block(src: str, start: int) -> str:
    """The text from the brace at `start` to the one that closes it."""
    depth = 0
    for i in range(start, len(src)):
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[start:i + 1]
    raise AssertionError("unbalanced braces")


def body_of(name: str) -> str:
    """The body of kernel `name` without its comments, strings and lambdas."""
    src = re.sub(r'//[^\n]*|/\*.*?\*/|"(?:\\.|[^"\\])*"', "", STEP.read_text(), flags=re.S)
    at = re.search(r"__global__[^;{]*\b" + name + r"\s*\(", src).end()
    body = block(src, src.index("{", at))
    while (lam := re.search(r"\[&\]\s*\([^)]*\)[^{;]*(?=\{)", body)):
        body = body[:lam.start()] + body[lam.end() + len(block(body, lam.end())):]
    return body


def test_every_cta_counts_itself_out():
    body = body_of("k_step")
    assert not re.search(r"\breturn\s*;", body)
    assert not re.search(r"\b(exit|__trap)\b", body)
    loop, tail = body.index("blockIdx.x; wi < nw"), body.index("atomicAdd(&ticket[1], 1u)")
    assert loop < tail and body.count("ticket[1], 1u") == 1


def test_the_scatter_does_not_promise_its_tile_to_itself():
    """The lanes of a warp add to the same nodes in turns, ordered by
    __syncwarp alone: a __restrict__ on the tile would let a compiler move a
    load over another lane's store."""
    src = re.sub(r"//[^\n]*", "", STEP.read_text())
    body = block(src, src.index("{", src.index("void warp_scatter(")))
    assert "Sm.acc[wid]" in body and "__restrict__" not in body
