"""Sample spacings of the transfer at and beyond the ends of the range: one sample a
step for an infinite one, 64 for a vanishing one, in both precisions."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SPACINGS = [math.inf, 1.7e308, 1e290, 1e-290, 1e-310, 5e-324]


def _scene(kerr, precision):
    return kerr.scene(width=9, height=7, spin=0.94, theta_obs=math.radians(50.0), integrator=1, precision=precision,
                      max_steps=2000, alpha_min=-16, alpha_max=16, beta_min=-16, beta_max=16)


@pytest.mark.parametrize("ds", SPACINGS)
def test_fp64_matches_oracle(cuda, oracle, ds):
    from blackhole_b200 import kerr, rt

    med, lut, prm = rt.Medium(n_r=40, n_theta=24, n_phi=20), rt.Lut(), rt.rt_defaults(ds_max=ds)
    s = _scene(kerr, 0)
    got = {k: v.cpu().numpy() for k, v in rt.trace(s, med, lut, prm).items()}
    d = lut.desc
    ref = oracle.trace_rt(s, med.cells.cpu().numpy(), (2.0, 50.0), lut.table.cpu().numpy(),
                          (d.log_theta_min, d.log_theta_max), (d.log_x_min, d.log_x_max), prm.nu_hz, prm.length_cm,
                          ds, prm.min_transmit)
    np.testing.assert_array_equal(got["cls"], ref["cls"])
    np.testing.assert_array_equal(got["steps"], ref["steps"])
    np.testing.assert_allclose(got["tau"], ref["tau"], rtol=1e-9, atol=1e-300)  # the tolerance of test_gpu_rt_warp.py
    np.testing.assert_allclose(got["i_nu"], ref["i_nu"], rtol=1e-9, atol=1e-300)
    assert (got["i_nu"] > 0).any()


@pytest.mark.parametrize("ds,same", [(math.inf, 1e30), (5e-324, 1e-30)])
def test_mixed_takes_the_ends_of_the_range(cuda, ds, same):
    from blackhole_b200 import kerr, rt

    med, lut = rt.Medium(n_r=40, n_theta=24, n_phi=20), rt.Lut()
    a = rt.trace(_scene(kerr, 1), med, lut, rt.rt_defaults(ds_max=ds))
    b = rt.trace(_scene(kerr, 1), med, lut, rt.rt_defaults(ds_max=same))
    torch.cuda.synchronize()
    for k in a:
        assert torch.equal(a[k], b[k]), k
    assert float(a["i_nu"].max()) > 0.0
