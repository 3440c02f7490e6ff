"""The tracers' pixel order (csrc/device/tile_order.h), compiled for the host: a
bijection of the frame at the edges of a tile and a band, and at the widths where a
band of four rows leaves 32 bits."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = tmp_path_factory.mktemp("tile_order") / "tile_order_main"
    cmd = ["g++", "-std=c++20", "-O2", "-Wall", "-Wextra", "-Werror", f"-I{ROOT / 'blackhole_b200/csrc/device'}",
           str(ROOT / "tests/cpp/tile_order_main.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("frames", [
    [(1, 1), (1, 7), (7, 1), (7, 5), (8, 4), (8, 5), (9, 3), (33, 17), (640, 360), (2048, 2048)],
    [(2**30 - 1, 1), (2**30 - 1, 2), (2**29, 3), (2**28 + 1, 7), (1, 2**31 - 1), (46340, 46340)],
    [(2**30, 1), (2**30 + 1, 1), (2**30 + 1000, 1), (1430000000, 1), (2**31 - 1, 1), (2**30, 2)],
])
def test_every_pixel_once_and_inside(program, frames):
    r = subprocess.run([str(program), *(str(v) for f in frames for v in f)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
