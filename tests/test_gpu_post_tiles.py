"""Post-processing frames at the edges of its tiles (64 x 16 rows pass, 32 x 64 columns
pass, 64 x 16 tone map) and with more rows of tiles than a grid's second dimension
holds, against the float64 restatement."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import legacy_oracle as LO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(15, 17), (16, 16), (31, 15), (32, 47), (33, 63), (95, 1), (128, 65), (701, 499), (2, 1048577)])
@pytest.mark.parametrize("strength", [0.0, 0.7])
def test_postprocess_tiles(cuda, w, h, strength):
    from blackhole_b200 import legacy

    rng = np.random.default_rng(w * 1000 + h)
    img = np.exp(rng.normal(-1.0, 1.3, (h, w, 4))).astype(np.float32)
    fb = torch.from_numpy(img.copy()).cuda()
    legacy.postprocess(fb, w, h, bloom_threshold=1.0, bloom_strength=strength, exposure_gain=3.0)
    want = LO.postprocess(img, 1.0, strength, 3.0)
    # 124 products of a bloomed value, then the tone curve: a few FP32 roundings of values <= 1
    np.testing.assert_allclose(fb.cpu().numpy(), want, rtol=2e-5, atol=2e-6)
