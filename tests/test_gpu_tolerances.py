"""Tolerances at and beyond the ends of the range a scene may have: infinite ones accept
every step, a vanishing atol leaves the decision to rtol, as in the oracle."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

TOLS = [(math.inf, 1e-10), (1e-8, math.inf), (1.7e308, 1e-10), (1e-8, 1.7e308), (1e-8, 1e-290), (1e-8, 1e-310),
        (1e-8, 5e-324)]


@pytest.mark.parametrize("rtol,atol", TOLS)
@pytest.mark.parametrize("spin", [0.9, 0.0])
def test_fp64_frame_matches_oracle(cuda, oracle, rtol, atol, spin):
    from blackhole_b200 import kerr

    s = kerr.scene(width=18, height=9, integrator=1, max_steps=1500, max_crossings=2, spin=spin, rtol=rtol, atol=atol)
    outs = kerr.trace_image(s)
    torch.cuda.synchronize()
    ref = oracle.trace_pixels(s)
    for k in ("cls", "steps", "n_cross", "r_hit", "g"):
        got = outs[k].cpu().numpy()
        np.testing.assert_array_equal(got, ref[k].reshape(got.shape), err_msg=k)


@pytest.mark.parametrize("rtol,atol", [(math.inf, 1e-10), (1e-8, math.inf), (1e-8, 5e-324)])
def test_fp64_transfer_takes_them(cuda, oracle, rtol, atol):
    from blackhole_b200 import kerr, rt

    med, lut, prm = rt.Medium(n_r=40, n_theta=24, n_phi=20), rt.Lut(), rt.rt_defaults()
    s = kerr.scene(width=6, height=5, spin=0.94, theta_obs=math.radians(50.0), integrator=1, precision=0,
                   max_steps=2000, alpha_min=-16, alpha_max=16, beta_min=-16, beta_max=16, rtol=rtol, atol=atol)
    got = {k: v.cpu().numpy() for k, v in rt.trace(s, med, lut, prm).items()}
    d = lut.desc
    ref = oracle.trace_rt(s, med.cells.cpu().numpy(), (2.0, 50.0), lut.table.cpu().numpy(),
                          (d.log_theta_min, d.log_theta_max), (d.log_x_min, d.log_x_max), prm.nu_hz, prm.length_cm,
                          prm.ds_max, prm.min_transmit)
    np.testing.assert_array_equal(got["cls"], ref["cls"])
    np.testing.assert_array_equal(got["steps"], ref["steps"])
