"""The branch-free FP32 root over every float, and the FP64 quotients and root over
2^28 operands, against CUDA's IEEE operations, bit for bit."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
NVCC = Path("/usr/local/cuda/bin/nvcc")


def test_equal_ieee(cuda, tmp_path):
    if not NVCC.exists():
        pytest.skip("no nvcc here")
    exe = tmp_path / "exact_ops"
    # -fmad=false as the FP64 tracers, whose quotients round as the CPU's do
    cmd = [str(NVCC), "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
           f"-I{ROOT / 'blackhole_b200/csrc/device'}", str(ROOT / "tests/cpp/exact_ops_main.cu"), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    counts = dict(zip(("sqrt_rn_f", "div_rn", "sqrt_rn", "div_5", "div_6"), map(int, r.stdout.split())))
    assert counts == dict.fromkeys(counts, 0)
