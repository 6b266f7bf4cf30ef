"""Particles whose stencil left their bin's tile (a re-bin cadence longer than
the run): the warp's lanes share such a particle's 27 nodes.  Few lanes (fewer
than 27, so that each takes several nodes), full warps and several such
particles in one warp; the tool boundary; heat conduction.  FP64 against the
oracle to 1e-9 in both node-sum modes; FP32 within the parity tests'
tolerances."""
from __future__ import annotations

import numpy as np
import pytest

from mpm_b200 import Solver, capi as A, workpiece as W
from test_gpu_parity import field_errors

pytestmark = pytest.mark.gpu


def run(case, st, steps, precision, deterministic=True):
    with Solver(W.to_mpm_params(case, precision=precision), len(st["x"])) as s:
        s.set_launch_config(sort_every=1024, deterministic=deterministic)
        s.set_tool(case["tool"])
        s.upload(st)
        s.step(case["dt"], steps)
        out = s.download()
        out["metrics"] = s.metrics()
    return out


def crossing(case, n, seed, speed):
    """n particles close to the faces of a bin, moving across them."""
    p = case["params"]
    rng = np.random.default_rng(seed)
    pos = 8.5 + rng.uniform(0.0, 4.0, (n, 3))
    axis, side = rng.integers(0, 3, n), rng.integers(0, 2, n)
    r = np.arange(n)
    pos[r, axis] = 8.5 + 4.0 * side + np.where(side, -1, 1) * rng.uniform(1e-4, 0.02, n)
    vel = rng.normal(0, 0.1 * speed, (n, 3))
    vel[r, axis] = np.where(side, 1, -1) * speed
    xyz = np.asarray(p["origin"]) + pos * p["dx"]
    st = W.full_state(dict(x=xyz[:, 0].copy(), y=xyz[:, 1].copy(), z=xyz[:, 2].copy(),
                           status=np.zeros(n, np.int32), id=np.arange(n, dtype=np.int32)), case)
    for a, k in enumerate(("vx", "vy", "vz")):
        st[k] = vel[:, a].copy()
    return st


@pytest.mark.parametrize("deterministic", [True, False])
@pytest.mark.parametrize("mode", [A.TOOL_NONE, A.TOOL_SDF_SLIP])
@pytest.mark.parametrize("n", [1, 5, 26, 33, 300])
def test_crossing_particles(oracle, n, mode, deterministic):
    case = W.config1(cells=(16, 12, 12), tool_mode=mode)
    st = crossing(case, n, 7 + n, 60.0)
    steps = 16
    ref, rc = oracle.step(case, st, steps)
    assert rc == 0
    out = run(case, st, steps, A.PREC_F64, deterministic)
    assert n == 1 or out["metrics"]["n_escaped"] > 0
    assert (out["status"] == ref["status"]).all()
    err = field_errors(out, ref, case)
    assert max(err.values()) < 1e-9, err
    err = field_errors(run(case, st, steps, A.PREC_F32, deterministic), ref, case)
    tol = dict(x=2e-4, y=2e-4, z=2e-4, vx=1e-3, vy=1e-3, vz=1e-3)
    bad = {k: v for k, v in err.items() if v > tol.get(k, 2e-3)}
    assert not bad, (bad, err)


@pytest.mark.parametrize("deterministic", [True, False])
@pytest.mark.parametrize("mode", [A.TOOL_NONE, A.TOOL_SDF_SLIP])
@pytest.mark.parametrize("n", [33, 300])
def test_crossing_particles_between_others(oracle, n, mode, deterministic):
    """Warps whose lanes off the tile lie between FIXED and INACTIVE ones, which take no part in the gather (the
    lanes that share the nodes have gaps), and CHIP ones, which keep their C."""
    case = W.config1(cells=(16, 12, 12), tool_mode=mode)
    st = crossing(case, n, 11 + n, 60.0)
    status = np.array([A.ACTIVE, A.FIXED, A.ACTIVE, A.CHIP, A.INACTIVE], np.int32)
    st["status"] = status[np.random.default_rng(n).integers(0, len(status), n)]
    for k in ("vx", "vy", "vz"):
        st[k][st["status"] == A.FIXED] = 0.0
    steps = 16
    ref, rc = oracle.step(case, st, steps)
    assert rc == 0
    out = run(case, st, steps, A.PREC_F64, deterministic)
    assert out["metrics"]["n_escaped"] > 0 and len(set(out["status"])) > 2
    assert (out["status"] == ref["status"]).all()
    err = field_errors(out, ref, case)
    assert max(err.values()) < 1e-9, err
    err = field_errors(run(case, st, steps, A.PREC_F32, deterministic), ref, case)
    tol = dict(x=2e-4, y=2e-4, z=2e-4, vx=1e-3, vy=1e-3, vz=1e-3)
    bad = {k: v for k, v in err.items() if v > tol.get(k, 2e-3)}
    assert not bad, (bad, err)


@pytest.mark.parametrize("deterministic", [True, False])
def test_heat_of_crossing_particles(oracle, deterministic):
    """Particles crossing at a grazing offset put about 2^-42 of their mass on
    the nodes they just reached: less than the fixed-point unit of the
    deterministic node sums (2^-40), where heat without mass would be a node
    temperature without bound."""
    case = W.config1(cells=(16, 12, 12), tool_mode=A.TOOL_NONE)
    p = case["params"]
    p.update(heat_conduction=1, thermal_conductivity=0.05 * p["dx"] ** 2 / case["dt"] * p["rho_phys"] * p["cp"])
    st = crossing(case, 400, 3, 0.0)
    rng = np.random.default_rng(4)
    # base cell one beyond the bin's last, offset within 2e-6 of its lower edge after the first step
    pos = np.stack([12.5 + rng.uniform(-1.0, 1.0, 400) * 2e-6, 8.5 + np.floor(rng.uniform(0, 4, 400)),
                    8.5 + np.floor(rng.uniform(0, 4, 400))], 1)
    pos[:, 1:] += rng.uniform(0.0, 2e-6, (400, 2))
    for a, k in enumerate(("x", "y", "z")):
        st[k] = p["origin"][a] + pos[:, a] * p["dx"]
        st["v" + k] = np.zeros(400)
    st["vx"] = np.full(400, 2e-6 * p["dx"] / case["dt"])
    st["temperature"] = p["Tamb"] + rng.uniform(100.0, 600.0, 400)
    p["gravity_z"] = 0.0
    ref, rc = oracle.step(case, st, 6)
    assert rc == 0
    out = run(case, st, 6, A.PREC_F64, deterministic)
    assert out["metrics"]["n_escaped"] > 0
    # In the deterministic sums T m is a whole number of units too: a node of one unit
    # is up to 0.5 K off, and a heavy neighbour takes 0.05 of that a step, so at most
    # 6 x 0.05 x 0.5 = 0.15 K from each light neighbour (0.04 K seen; heat without
    # mass there: 58 K).
    tol = 0.15 if deterministic else 1e-6 * np.abs(ref["temperature"] - p["Tamb"]).max()
    assert np.abs(out["temperature"] - ref["temperature"]).max() <= tol
