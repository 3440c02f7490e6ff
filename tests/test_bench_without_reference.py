"""bench.py where the reference's CPU library is not built: its arm says so in one line
and ends well, and the GPU's own line is printed without a CPU baseline."""
from __future__ import annotations

import json
import subprocess
import sys
from pathlib import Path

from oracle import pyoracle

ROOT = Path(__file__).resolve().parents[1]


def _absent(monkeypatch, tmp_path):
    monkeypatch.setattr(pyoracle.RefLib.__init__, "__defaults__", (tmp_path / "libbh_ref.so",))


def test_no_cpu_baseline_is_none(monkeypatch, tmp_path, capsys):
    import bench

    _absent(monkeypatch, tmp_path)
    assert bench.cpu_baseline(None, "c0_256", 0.1) is None
    assert "not built" in capsys.readouterr().err


def test_reference_arm_says_unavailable(monkeypatch, tmp_path, capsys):
    import bench

    _absent(monkeypatch, tmp_path)
    monkeypatch.setattr(sys, "argv", ["bench.py", "--impl", "reference", "--workload", "c0_256"])
    bench.main()
    line = json.loads(capsys.readouterr().out)
    assert line["impl"] == "reference" and "not built" in line["unavailable"]


def test_reference_arm_exits_0(tmp_path):
    if pyoracle.RefLib.available():
        import pytest

        pytest.skip("the reference's library is built here")
    r = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--impl", "reference", "--steps", "1", "--warmup", "0"],
                       capture_output=True, text=True, cwd=ROOT)
    assert r.returncode == 0, r.stderr
    assert json.loads(r.stdout)["unavailable"]
