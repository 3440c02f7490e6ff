"""FP64 transfer at frequencies to the ends of the double range, where nu / g and
nu / nu_s overflow or vanish, against the oracle."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu", [math.inf, 1.79e308, 1e305, 1e290, 1e40, 1e-3, 1e-150])
def test_matches_oracle(cuda, oracle, nu):
    from blackhole_b200 import kerr, rt

    med, lut, prm = rt.Medium(n_r=40, n_theta=24, n_phi=20), rt.Lut(), rt.rt_defaults(nu_hz=nu)
    s = kerr.scene(width=9, height=7, spin=0.94, theta_obs=math.radians(50.0), integrator=1, precision=0,
                   max_steps=2000, alpha_min=-16, alpha_max=16, beta_min=-16, beta_max=16)
    got = {k: v.cpu().numpy() for k, v in rt.trace(s, med, lut, prm).items()}
    d = lut.desc
    with np.errstate(all="ignore"):
        ref = oracle.trace_rt(s, med.cells.cpu().numpy(), (2.0, 50.0), lut.table.cpu().numpy(),
                              (d.log_theta_min, d.log_theta_max), (d.log_x_min, d.log_x_max), nu, prm.length_cm,
                              prm.ds_max, prm.min_transmit)
    np.testing.assert_array_equal(got["cls"], ref["cls"])
    np.testing.assert_array_equal(got["steps"], ref["steps"])
    np.testing.assert_allclose(got["tau"], ref["tau"], rtol=1e-9, atol=1e-300)  # the tolerance of test_gpu_rt_warp.py
    np.testing.assert_allclose(got["i_nu"], ref["i_nu"], rtol=1e-9, atol=1e-300)
