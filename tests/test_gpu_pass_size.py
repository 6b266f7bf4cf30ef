"""The launch config's pass_size, accepted and without effect, and the
persistent grid's clamp to the CTAs that fit on an SM.

- 128, 256 and 512 are accepted and returned (0: 128); another value is
  refused and leaves the configuration as it was.
- A workpiece of more bins than the grid has CTAs gives the same bits at one
  CTA per SM, at two, and at eight, more than the three (FP64: two) that fit,
  where the launch clamps the grid; and with another pass_size.
"""
from __future__ import annotations

import numpy as np
import pytest

from mpm_b200 import Solver, capi as A, workpiece as W

pytestmark = pytest.mark.gpu

STATE = ("x", "y", "z", "vx", "vy", "vz", "F", "Fp", "C", "stress", "plastic_strain", "strain_rate",
         "temperature", "damage", "residual_stress", "status")


def run(case, precision, ctas=4, pass_size=0):
    b = case["box"]
    with Solver(W.to_mpm_params(case, precision=precision), 64 * 32 * 32 * 8) as s:
        s.set_launch_config(ctas_per_sm=ctas, pass_size=pass_size)
        assert s.launch_config()["pass_size"] == (pass_size or 128)
        s.init_box(b["c0"], b["c1"], b["ppc"], b["seed"], 0, b["fixed_layers"], b["T0"], tool=case["tool"])
        s.step(case["dt"], 20)
        return s.download(STATE)


@pytest.mark.parametrize("precision", [A.PREC_F32, A.PREC_F64])
def test_any_cta_count_gives_the_same_bits(precision):
    case = W.config1()   # 16 x 8 x 8 bins: more than 148 SMs x 3 CTAs
    a = run(case, precision)
    for kw in (dict(ctas=1), dict(ctas=2), dict(ctas=8), dict(pass_size=256), dict(pass_size=512)):
        b = run(case, precision, **kw)
        for k in STATE:
            assert np.array_equal(a[k], b[k], equal_nan=True), (kw, k)


def test_unknown_pass_size_is_refused():
    case = W.config1(cells=(8, 8, 8))
    with Solver(W.to_mpm_params(case, precision=A.PREC_F32), 4096) as s:
        s.set_launch_config(pass_size=512)
        before = s.launch_config()
        with pytest.raises(A.MpmError) as e:
            s.set_launch_config(ctas_per_sm=2, pass_size=384)
        assert e.value.status == A.MPM_INVALID_ARG
        assert s.launch_config() == before
