"""The batched Mino step away from ordinary magnitudes: the branch-free step and the
one with CUDA's operators take over from each other at the ends of their range, and
neither may change a ray that the other would have traced."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

GEOM = 2.99792458e10**2 / 6.67430e-8  # G m / c^2 = 1 cm


def dev(x):
    return torch.as_tensor(np.atleast_1d(np.asarray(x, np.float64)), device="cuda")


def _state(r, theta):
    r, theta = np.broadcast_arrays(np.atleast_1d(r), np.atleast_1d(theta))
    one = np.ones(r.shape)
    return {"r": dev(r), "theta": dev(theta), "phi": dev(0 * one), "t": dev(0 * one), "sign_r": dev(-one),
            "sign_theta": dev(one)}


@pytest.mark.parametrize("scale", [1.0, 1e30, 2.0**180, 2.0**230])
@pytest.mark.parametrize("n", [1, 31, 33])
def test_step_scales_exactly(cuda, scale, n):
    """With a power of two between them, lengths in other units give the same step
    bit for bit: r and lambda scale, angles do not (e = 1, l ~ length, q ~ length^2,
    dlam ~ 1 / length), as long as Delta stays above the 1e-12 cm^2 at which the
    reference clamps it."""
    from blackhole_b200 import kerr

    s = 2.0 ** round(math.log2(scale))
    rng = np.random.default_rng(n)
    r, th = rng.uniform(6, 40, n), rng.uniform(0.7, 2.4, n)
    lz = rng.uniform(-4, 4, n)
    q = lz**2 / np.sin(th) ** 2 + rng.uniform(1, 9, n)
    out = []
    for k in (1.0, s):
        st = _state(r * k, th)
        kerr.kerr_step_mino(st, GEOM * k, 0.5 * k, dev(np.ones(n)), dev(lz * k), dev(q * k * k), 1e-3 / k)
        out.append({f: v.cpu().numpy() for f, v in st.items()})
    np.testing.assert_array_equal(out[1]["theta"], out[0]["theta"])
    np.testing.assert_array_equal(out[1]["phi"], out[0]["phi"])
    if scale < 2.0**190:  # beyond, r^4 leaves the range on the way
        np.testing.assert_array_equal(out[1]["r"], out[0]["r"] * s)


@pytest.mark.parametrize("step", [1e-3, 1e10, 1e60, 1e200])
def test_extreme_steps_end_as_the_oracles(cuda, oracle, step):
    """Steps whose stages leave the double range (infinities and NaN on the way) end
    with the oracle's status after the oracle's number of steps."""
    from blackhole_b200 import kerr

    n = 6
    r = np.array([20.0, 3.0, 1e3, 1e70, 1e-3, 50.0])
    host = {"r": r, "theta": np.full(n, 1.2), "phi": np.zeros(n), "t": np.zeros(n),
            "sign_r": np.array([1.0, -1, 1, 1, -1, -1]), "sign_theta": np.ones(n)}
    e, lz, q = np.ones(n), np.full(n, 2.0), np.full(n, 5.0)
    tr = kerr.KerrRaytracer(GEOM, 0.3)
    tr.set_step_size(step)
    tr.set_max_steps(7)
    p = tr.params
    ref = oracle.trace_rays(host, e, lz, q, GEOM, 0.3, p.r_horizon, p.r_escape, step, 7)
    res = tr.trace({k: dev(v) for k, v in host.items()}, dev(e), dev(lz), dev(q))
    assert res.status.tolist() == ref["status"].tolist()
    assert res.steps_taken.tolist() == ref["steps"].tolist()
