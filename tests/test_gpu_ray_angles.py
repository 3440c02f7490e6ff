"""The polar angles of the batched Mino step: reduction by pi / 2 in two parts below
1024, CUDA's sincos beyond, the poles and the equator, against 128 bits."""
from __future__ import annotations

import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

GEOM = 2.99792458e10**2 / 6.67430e-8  # G m / c^2 = 1 cm
EPS = 2.0**-53


def _angles(kind):
    if kind == "multiples":  # of pi / 4 and beside them, both sides of each change of quadrant
        k = np.arange(1, 40) * (math.pi / 4)
        return np.concatenate([k, np.nextafter(k, 0), k * (1 + 1e-9), k * (1 - 1e-5)])
    if kind == "poles":
        return np.array([1e-6, 1e-5, 1e-3, math.pi - 1e-6, math.pi - 1e-4, 0.1, 3.0])
    if kind == "edge":  # of the reduction's range
        return np.array([1023.5, np.nextafter(1024.0, 0), 1024.0, 1024.5, -1023.0, -1025.0, 3e4])
    return np.random.default_rng(3).uniform(-6, 8, 257)


@pytest.mark.parametrize("kind", ["multiples", "poles", "edge", "random"])
def test_azimuth_of_one_step(cuda, oracle, kind):
    """phi' = lz / sin^2 - a e + a A / Delta: sin^2 is within 2 x 1 ulp and its own
    rounding, each of the terms within 2 more; four stages and the step's sum add 6
    roundings of the largest term, taken at the smallest sin^2 of the step."""
    from blackhole_b200 import kerr

    th = _angles(kind)
    n = th.size
    r, a, lz, dlam = np.full(n, 12.0), 0.4, 0.7, 1e-16
    sin2 = np.array([float(np.sin(np.longdouble(t)) ** 2) for t in th])
    q = lz * lz / np.maximum(sin2, 1e-12) + 50.0  # far from a polar turning point
    one = np.ones(n)
    host = {"r": r, "theta": th.copy(), "phi": 0 * one, "t": 0 * one, "sign_r": -one, "sign_theta": one}
    st = {k: torch.as_tensor(v.copy(), device="cuda") for k, v in host.items()}
    dev = lambda v: torch.as_tensor(v, device="cuda")  # noqa: E731
    kerr.kerr_step_mino(st, GEOM, a, dev(one), dev(lz * one), dev(q), dlam)
    ref = oracle.step_mino_f128(host, GEOM, a, one, lz * one, q, dlam)
    # the angle moves by up to dlam sqrt(q) in the step, which sin^2 follows
    moved = dlam * np.sqrt(q + 1.0)
    small = np.maximum(np.maximum(np.abs(np.sqrt(sin2)) - moved, 0.0) ** 2, 1e-12)
    A = r * r + a * a - a * lz
    size = lz / small + a + a * A / (r * r - 2 * r + a * a)
    # a stage's angle is rounded to 64 bits, which sin^2 follows near the poles
    cond = 2 * np.spacing(np.abs(th)) / np.sqrt(small)
    assert np.all(np.abs(st["phi"].cpu().numpy() - ref["phi"]) <= (16 * EPS + cond) * dlam * size)
    assert np.array_equal(st["sign_theta"].cpu().numpy(), one)
