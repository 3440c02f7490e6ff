"""Media on both sides of the line between 32- and 64-bit offsets of the mixed transfer
(2^28 cells of 16 bytes), against the same medium with few azimuths."""
from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _medium(rt, n_ph):
    m = rt.Medium(64, 64, n_ph, r_min=2.0, r_max=50.0, synthetic=False)
    i = torch.arange(64, device="cuda", dtype=torch.float32)
    r = 2.0 * 25.0 ** (i / 63)
    th = (i + 0.5) / 64 * math.pi
    n = 3e5 * torch.exp(-((torch.cos(th)[None, :] / 0.5) ** 2)) * (r[:, None] / 10) ** -1.1
    for k, v in enumerate((n, (8.0 / r[:, None]).expand(64, 64), (30.0 / r[:, None]).expand(64, 64))):
        m.cells[..., k] = v[:, :, None]
    m.cells[..., 3] = 0.0
    return m


@pytest.mark.parametrize("side", [48, 320])  # few rays a warp; whole warps
@pytest.mark.parametrize("n_ph", [65536, 65537])
def test_axisymmetric_medium(cuda, n_ph, side):
    """The cells do not depend on the azimuth, so the number of azimuths may only move
    the roundings of the 8 products of a sample: 8 x 2^-24 relative in density, field
    and temperature, of which ln j takes 1, 1 + d and 2 d times (d = 1.89 / 3 x^(1/3)
    <= 14 on the table), the source function about 1 more: 3e-5 of the intensity."""
    from blackhole_b200 import kerr, rt

    if torch.cuda.mem_get_info()[0] < 12 << 30:
        pytest.skip("needs 12 GB")
    lut = rt.Lut()
    sc = kerr.scene(width=side, height=side, spin=0.9, theta_obs=math.radians(50.0), alpha_min=-15.0, alpha_max=15.0,
                    beta_min=-15.0, beta_max=15.0, precision=1, integrator=1, max_steps=2000)
    outs = []
    for k in (16, n_ph):
        m = _medium(rt, k)
        o = rt.trace(sc, m, lut)
        torch.cuda.synchronize()
        outs.append({f: v.clone() for f, v in o.items()})
        del m, o
        torch.cuda.empty_cache()
    assert torch.equal(outs[0]["cls"], outs[1]["cls"]) and torch.equal(outs[0]["steps"], outs[1]["steps"])
    assert float(outs[0]["i_nu"].max()) > 0.0
    torch.testing.assert_close(outs[1]["i_nu"], outs[0]["i_nu"], rtol=3e-5, atol=3e-5 * float(outs[0]["i_nu"].max()))
