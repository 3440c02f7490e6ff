"""The transfer kernels that sample the medium warp by warp: frames at the edges of
a warp's rays, of a tile and of the one-wave rule, against the oracle (FP64) and
against the same frame traced by the per-lane kernel as part of a larger window
(mixed)."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _scene(kerr, w, h, precision, **kw):
    return kerr.scene(width=w, height=h, spin=0.94, theta_obs=math.radians(50.0), integrator=1, precision=precision,
                      max_steps=2000, **{**dict(alpha_min=-16, alpha_max=16, beta_min=-16, beta_max=16), **kw})


@pytest.mark.parametrize("w,h", [(1, 1), (3, 1), (5, 3), (9, 5), (33, 4)])
def test_fp64_edges_match_oracle(cuda, oracle, w, h):
    from blackhole_b200 import kerr, rt

    med, lut, prm = rt.Medium(n_r=40, n_theta=24, n_phi=20), rt.Lut(), rt.rt_defaults()
    s = _scene(kerr, w, h, 0)
    got = {k: v.cpu().numpy() for k, v in rt.trace(s, med, lut, prm).items()}
    d = lut.desc
    ref = oracle.trace_rt(s, med.cells.cpu().numpy(), (2.0, 50.0), lut.table.cpu().numpy(),
                          (d.log_theta_min, d.log_theta_max), (d.log_x_min, d.log_x_max), prm.nu_hz, prm.length_cm,
                          prm.ds_max, prm.min_transmit)
    np.testing.assert_array_equal(got["cls"], ref["cls"])
    np.testing.assert_array_equal(got["steps"], ref["steps"])
    np.testing.assert_allclose(got["tau"], ref["tau"], rtol=1e-9, atol=1e-300)
    np.testing.assert_allclose(got["i_nu"], ref["i_nu"], rtol=1e-9, atol=1e-300)


@pytest.mark.parametrize("w,h", [(1, 1), (5, 4), (32, 32), (256, 37)])
def test_mixed_few_rays_equal_many(cuda, w, h):
    """The first rows of a tall frame (past one wave: the per-lane kernel) are the
    short frame's rays: pixel (i, j) of both has the same alpha and beta."""
    from blackhole_b200 import kerr, rt

    med, lut = rt.Medium(n_r=40, n_theta=24, n_phi=20), rt.Lut()
    tall = max(1, -(-100000 // w))
    scale = 2.0 ** math.ceil(math.log2(tall / h))  # a power of two: the pixel pitch is the same number
    H = int(h * scale)
    few = _scene(kerr, w, h, 1, beta_min=0.0, beta_max=16.0)
    many = _scene(kerr, w, H, 1, beta_min=0.0, beta_max=16.0 * scale)
    a, b = rt.trace(few, med, lut), rt.trace(many, med, lut)
    torch.cuda.synchronize()
    for k in a:
        assert torch.equal(a[k], b[k][:w * h]), k
