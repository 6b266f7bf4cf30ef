"""The step kernel's scatter at the edges of its warps: bins whose particles fill
a warp partly, exactly or by one more; several particles in one cell (lanes
that share a cell take turns); particles of both halves of a bin in one warp
(fewer than 64 particles); particles that change cells between re-bins.  FP64
against the oracle to 1e-9; FP32 within the parity tests' tolerances; the same
bits on a second run."""
from __future__ import annotations

import numpy as np
import pytest

from mpm_b200 import capi as A, workpiece as W
from test_gpu_parity import field_errors, run_ours

pytestmark = pytest.mark.gpu


def layout(name):
    """Positions in cells (grid units) for a layout of one or a few bins."""
    rng = np.random.default_rng(5)
    bin0 = np.array([8.5, 8.5, 8.5])          # stencil base (8, 8, 8): first cell of a bin
    grid = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    if name.startswith("n"):                  # n particles spread over one bin
        return bin0 + rng.uniform(0.0, 4.0, (int(name[1:]), 3))
    if name == "one_cell":                    # seven turns of a warp
        return bin0 + rng.uniform(0.0, 1.0, (200, 3))
    if name == "two_layers":                  # every warp holds cells of both halves
        return np.concatenate([bin0 + [x, y, z] + rng.uniform(0, 1, 3) for x in range(4) for y in range(4)
                               for z in (0, 3)]).reshape(-1, 3)
    if name == "ppc8":                        # full columns
        return np.repeat(bin0 + grid, 8, 0) + rng.uniform(0, 1, (512, 3))
    if name == "ppc5_tail":                   # five rows, then a tail
        return np.concatenate([np.repeat(bin0 + grid, 5, 0), bin0 + grid[:17]]) + rng.uniform(0, 1, (337, 3))
    raise KeyError(name)


@pytest.mark.parametrize("name", ["n1", "n31", "n32", "n33", "n63", "n65", "n129", "one_cell", "two_layers", "ppc8",
                                  "ppc5_tail"])
def test_scatter_edges(oracle, name):
    case = W.config1(cells=(16, 12, 12), tool_mode=A.TOOL_NONE)
    p = case["params"]
    pos = layout(name)
    n = len(pos)
    rng = np.random.default_rng(6)
    xyz = np.asarray(p["origin"]) + pos * p["dx"]
    st = W.full_state(dict(x=xyz[:, 0].copy(), y=xyz[:, 1].copy(), z=xyz[:, 2].copy(),
                           status=np.zeros(n, np.int32), id=np.arange(n, dtype=np.int32)), case)
    for k in ("vx", "vy", "vz"):
        st[k] = rng.normal(0, 40.0, n)        # up to 0.01 cell a step: cells change between re-bins
    st["F"] = st["F"] + rng.normal(0, 1e-4, (n, 9))
    steps = 12
    ref, rc = oracle.step(case, st, steps)
    assert rc == 0
    out = run_ours(case, st, steps, prec=A.PREC_F64)
    assert (out["status"] == ref["status"]).all()
    err = field_errors(out, ref, case)
    assert max(err.values()) < 1e-9, err
    a = run_ours(case, st, steps, prec=A.PREC_F32)
    b = run_ours(case, st, steps, prec=A.PREC_F32)
    err = field_errors(a, ref, case)
    tol = dict(x=2e-4, y=2e-4, z=2e-4, vx=1e-3, vy=1e-3, vz=1e-3)
    bad = {k: v for k, v in err.items() if v > tol.get(k, 2e-3)}
    assert not bad, (bad, err)
    for k in ("x", "vx", "F", "C", "stress"):
        assert np.array_equal(a[k], b[k]), k
