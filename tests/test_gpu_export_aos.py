"""Particle records (mpm_export_aos) against the field download, at the edges of
the export's 32-particle warps and 64/128-particle CTAs: every field of every
record is the downloaded double, bit for bit, and the constant fields are the
workpiece's."""
from __future__ import annotations

import numpy as np
import pytest

from mpm_b200 import Solver, capi as A, workpiece as W

pytestmark = pytest.mark.gpu


def state(case, n, seed=3):
    rng = np.random.default_rng(seed)
    st = W.full_state({k: v[:n] for k, v in W.generate_box(case).items()}, case)
    for k in ("vx", "vy", "vz", "plastic_strain", "strain_rate", "damage", "residual_stress"):
        st[k] = rng.uniform(-1.0, 1.0, n)
    st["temperature"] = 293.0 + rng.uniform(0, 500, n)
    for k in ("F", "Fp"):
        st[k] = st[k] + rng.normal(0, 1e-3, (n, 9))
    st["C"] = rng.normal(0, 1e3, (n, 9))
    st["stress"], st["backstress"] = rng.normal(0, 1e8, (n, 6)), rng.normal(0, 1e7, (n, 6))
    st["id"] = rng.permutation(n).astype(np.int32)
    st["vx"][0] = -0.0
    return st


@pytest.mark.parametrize("precision", [A.PREC_F32, A.PREC_F64])
@pytest.mark.parametrize("hkin", [0.0, 1e9])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 65, 127, 129, 1000])
def test_records_equal_download(precision, hkin, n):
    case = W.config1(cells=(8, 6, 6), tool_mode=A.TOOL_NONE)
    case["params"]["H_kin"] = hkin
    with Solver(W.to_mpm_params(case, precision=precision), n) as s:
        s.upload(state(case, n))
        rec = s.export_aos().view(A.MPM_PARTICLE)
        ref = s.download()
    assert len(rec) == n
    for a in ("x", "y", "z", "vx", "vy", "vz", "F", "C", "temperature", "damage", "id", "status"):
        assert np.array_equal(rec[a], ref[a]), a
    assert np.signbit(rec["vx"][0])
    for a, b in (("F_p", "Fp"), ("plasticStrain", "plastic_strain"), ("strainRate", "strain_rate"),
                 ("residualStress", "residual_stress")):
        assert np.array_equal(rec[a], ref[b]), a
    assert np.array_equal(rec["stress"], ref["stress"]) and np.array_equal(rec["backstress"], ref["backstress"])
    p = case["params"]
    R = np.float32 if precision == A.PREC_F32 else np.float64
    assert (rec["mass"] == float(R(p["particle_mass"]))).all()
    assert (rec["volume"] == float(R(p["particle_volume"]))).all()
    assert (rec["density"] == p["rho_phys"]).all()
    for a in ("fx", "fy", "fz", "ext_fx", "ext_fy", "ext_fz", "pressure", "cellHash", "lodZone", "lastUpdateStep",
              "asbCounter"):
        assert not rec[a].any(), a
