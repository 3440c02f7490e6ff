"""Media that vary with azimuth on both sides of the line between 32- and 64-bit offsets
of the mixed transfer (2^28 cells of 16 bytes), against the same field on fewer
azimuths."""
from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _medium(rt, n_ph, amplitude=1.0):
    m = rt.Medium(64, 64, n_ph, r_min=2.0, r_max=50.0, synthetic=False)
    i = torch.arange(64, device="cuda", dtype=torch.float64)
    r = 2.0 * 25.0 ** (i / 63)
    th = (i + 0.5) / 64 * math.pi
    ph = torch.arange(n_ph, device="cuda", dtype=torch.float64) * (2 * math.pi / n_ph)
    n = 3e5 * torch.exp(-((torch.cos(th)[None, :] / 0.5) ** 2)) * (r[:, None] / 10) ** -1.1
    wave = (1.0 + amplitude * (0.6 * torch.sin(ph) + 0.25 * torch.cos(2 * ph))).float()
    for k, v in enumerate((n, (8.0 / r[:, None]).expand(64, 64), (30.0 / r[:, None]).expand(64, 64))):
        m.cells[..., k] = v.float()[:, :, None]
    m.cells[..., 0] *= wave
    m.cells[..., 3] = 0.0
    return m


@pytest.mark.parametrize("side", [48, 320])  # few rays a warp; whole warps
@pytest.mark.parametrize("n_ph", [65536, 65537])
def test_a_wave_in_azimuth(cuda, n_ph, side):
    """Linear interpolation on 4096 azimuths is off by at most (2 pi / 4096)^2 / 8 times
    the second derivative, 1.6: 5e-7 of a density of at least 0.15; and a sample's
    azimuth, known to 2^-24 of a turn times its few turns in FP32, moves the density by
    2e-6 of itself. With the roundings of test_gpu_rt_wide.py: 5e-5 of the intensity."""
    from blackhole_b200 import kerr, rt

    if torch.cuda.mem_get_info()[0] < 16 << 30:
        pytest.skip("needs 16 GB")
    lut = rt.Lut()
    sc = kerr.scene(width=side, height=side, spin=0.9, theta_obs=math.radians(50.0), alpha_min=-15.0, alpha_max=15.0,
                    beta_min=-15.0, beta_max=15.0, precision=1, integrator=1, max_steps=2000)
    outs = []
    for k, amplitude in ((4096, 1.0), (n_ph, 1.0), (16, 0.0)):
        m = _medium(rt, k, amplitude)
        o = rt.trace(sc, m, lut)
        torch.cuda.synchronize()
        outs.append({f: v.clone() for f, v in o.items()})
        del m, o
        torch.cuda.empty_cache()
    i0 = outs[0]["i_nu"]
    assert float(i0.max()) > 0.0
    assert float((outs[2]["i_nu"] - i0).abs().max()) > 0.05 * float(i0.max())  # the wave is seen
    torch.testing.assert_close(outs[1]["i_nu"], i0, rtol=5e-5, atol=5e-5 * float(i0.max()))
