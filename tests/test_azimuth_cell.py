"""The azimuthal cell of a medium (csrc/device/azimuth_cell.h), compiled for the host:
the exact remainder, also where an azimuth is past the whole numbers of its type."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_cells_are_the_exact_remainder(tmp_path):
    exe = tmp_path / "azimuth_cell_main"
    cmd = ["g++", "-std=c++20", "-O2", "-Wall", "-Wextra", "-Werror", f"-I{ROOT / 'blackhole_b200/csrc/device'}",
           str(ROOT / "tests/cpp/azimuth_cell_main.cpp"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
