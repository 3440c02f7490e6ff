"""Rays that start within a rounding of a polar turning point: the branch-free step and
the one with CUDA's operators, which takes lengths beyond 2^200, see the same sign of
the polar potential and so turn the same rays."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

GEOM = 2.99792458e10**2 / 6.67430e-8  # G m / c^2 = 1 cm


@pytest.mark.parametrize("a", [0.0, 0.5])
def test_both_steps_turn_the_same_rays(cuda, a):
    """In units of 2^205 cm every operation rounds as in cm (r^4 stays below 2^860), so
    the traces agree bit for bit."""
    from blackhole_b200 import kerr

    n = 20000
    rng = np.random.default_rng(7)
    r, th, lz = rng.uniform(8, 30, n), rng.uniform(0.4, 2.7, n), rng.uniform(1, 4, n)
    # Theta(theta) = 0 up to rounding
    q = lz * lz / np.sin(th) ** 2 - a * a * np.cos(th) ** 2
    out = []
    for k in (1.0, 2.0**205):
        dev = lambda v: torch.as_tensor(np.ascontiguousarray(v), device="cuda")  # noqa: E731
        one = np.ones(n)
        st = {"r": r * k, "theta": th, "phi": 0 * one, "t": 0 * one, "sign_r": -one, "sign_theta": one}
        tr = kerr.KerrRaytracer(GEOM * k, a * k)
        tr.set_step_size(1e-3 / k)
        tr.set_max_steps(3)
        res = tr.trace({f: dev(v) for f, v in st.items()}, dev(one), dev(lz * k), dev(q * k * k))
        torch.cuda.synchronize()
        out.append(res)
    assert torch.equal(out[0].steps_taken, out[1].steps_taken)
    assert torch.equal(out[0].final_theta, out[1].final_theta)
    assert torch.equal(out[0].final_phi, out[1].final_phi)
    assert torch.equal(out[0].final_r * 2.0**205, out[1].final_r)
