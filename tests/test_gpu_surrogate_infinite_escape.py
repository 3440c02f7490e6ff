"""The surrogate's refinement takes an infinite escape radius, which a scene may have:
its escape directions are those at infinity, the limit of large radii."""
from __future__ import annotations

from pathlib import Path

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

WEIGHTS = Path(__file__).resolve().parents[1] / "blackhole_b200" / "data" / "surrogate_c4.npz"


@pytest.mark.parametrize("refine_fp64", [False, True])
@pytest.mark.parametrize("fields", ["all", "no azimuths"])
def test_directions_at_infinity(cuda, refine_fp64, fields):
    from blackhole_b200 import kerr
    from blackhole_b200 import surrogate as S

    net = S.Surrogate(max_batch=128)
    net.load(WEIGHTS)

    def frame(escape_factor):
        s = kerr.scene(width=49, height=33, integrator=1, precision=1, spin=0.9, max_steps=3000,
                       escape_factor=escape_factor)
        outs = kerr.alloc_image_outputs(s)
        if fields != "all":
            outs = {k: outs[k] for k in ("cls", "steps", "theta_inf")}
        # the refinement decides every pixel: those it leaves to the closed form, which has no
        # direction at infinity, are not what is tested
        net.trace_image(s, outs, refine_fp64=refine_fp64, min_confidence=0.0, verify=3, critical_band=0.0)
        torch.cuda.synchronize()
        return {k: v.cpu().numpy() for k, v in outs.items()}

    far, inf = frame(1e12), frame(float("inf"))
    np.testing.assert_array_equal(inf["cls"], far["cls"])
    out = inf["cls"] == 2
    assert out.sum() > 50
    # 1 / r moves by 1e-15, far below the rounding of the variable; the FP32 quadrature's noise is 1e-6 (1e-12 in FP64)
    tol = 1e-9 if refine_fp64 else 2e-5
    np.testing.assert_allclose(inf["theta_inf"][out], far["theta_inf"][out], rtol=0, atol=tol)
    if fields == "all":
        np.testing.assert_allclose(inf["phi_inf"][out], far["phi_inf"][out], rtol=0, atol=tol)
