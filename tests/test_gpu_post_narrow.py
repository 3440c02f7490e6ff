"""Post-processing of narrow images: every width about the paddings of the blurs'
planes against the float64 restatement, and the scratch that a long thin image takes."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import legacy_oracle as LO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [*range(1, 50), 64, 65, 68, 69, 100, 119, 120, 121, 239, 240, 241, 300, 471, 480, 481, 944, 945])
def test_widths(cuda, w):
    from blackhole_b200 import legacy

    h = 19
    rng = np.random.default_rng(w)
    img = np.exp(rng.normal(-1.0, 1.3, (h, w, 4))).astype(np.float32)
    fb = torch.from_numpy(img.copy()).cuda()
    legacy.postprocess(fb, w, h, bloom_threshold=1.0, bloom_strength=0.7, exposure_gain=3.0)
    want = LO.postprocess(img, 1.0, 0.7, 3.0)
    # 124 products of a bloomed value, then the tone curve: a few FP32 roundings of values <= 1
    np.testing.assert_allclose(fb.cpu().numpy(), want, rtol=2e-5, atol=2e-6)


@pytest.mark.parametrize("w,strength,floats_a_pixel", [(1, 0.0, 4), (1, 0.7, 60), (2, 0.7, 30), (4, 0.7, 16), (46, 0.7, 16)])
def test_scratch_of_a_thin_image(cuda, w, strength, floats_a_pixel):
    from blackhole_b200 import _abi, legacy

    h = 2_000_000 // w
    lib = _abi.load_library()
    fb = torch.full((h, w, 4), 0.5, device="cuda")
    legacy.postprocess(fb, w, h, bloom_strength=strength)  # kernels loaded
    assert lib.bhbCudaResetDevice() == 0  # gives the scratch back
    before = torch.cuda.mem_get_info()[0]
    legacy.postprocess(fb, w, h, bloom_strength=strength)
    taken = before - torch.cuda.mem_get_info()[0]
    # cudaMalloc takes whole pieces of 2 MiB
    assert taken <= 4 * floats_a_pixel * w * h + (4 << 20), (taken, w * h)
    assert lib.bhbCudaResetDevice() == 0
