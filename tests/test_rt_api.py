"""bh_kerr_trace_rt refuses grids and emission tables that have no interval to
interpolate in (on the host, before any device work)."""
from __future__ import annotations

import ctypes as C

import pytest


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("field,value", [("n_r", 1), ("n_r", 0), ("n_theta", 1), ("n_phi", 0), ("n_phi", -1),
                                         ("lut_theta", 1), ("lut_x", 0)])
def test_bad_grids_are_refused(lib, precision, field, value):
    from blackhole_b200 import _abi, rt

    L = rt._lib()
    dims = {**dict(n_r=8, n_theta=6, n_phi=4, lut_theta=16, lut_x=16), field: value}
    s = _abi.default_scene(width=4, height=4, integrator=1, precision=precision)
    grid = rt.GrmhdGrid(4096, dims["n_r"], dims["n_theta"], dims["n_phi"], 0, 2.0, 50.0)  # never read
    lut = rt.SynchrotronLut(4096, dims["lut_theta"], dims["lut_x"], -2.0, 7.0, -9.0, 9.0)
    assert L.bh_kerr_trace_rt(C.byref(s), C.byref(grid), C.byref(lut), None, None, None, None, None, None) == -1
    assert b"nodes" in L.bh_last_error()
