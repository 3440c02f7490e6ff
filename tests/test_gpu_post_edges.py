"""Post-processing frames at the edges of the blur kernels' tiles (128 x 32 and 64 x 64),
of a row pair and of the padded planes, against the float64 restatement."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import legacy_oracle as LO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (2, 1), (63, 31), (64, 64), (65, 33), (127, 2), (129, 65), (200, 97)])
@pytest.mark.parametrize("strength", [0.0, 0.7])
def test_postprocess_tile_edges(cuda, w, h, strength):
    from blackhole_b200 import legacy

    rng = np.random.default_rng(w * 1000 + h)
    img = np.exp(rng.normal(-1.0, 1.3, (h, w, 4))).astype(np.float32)
    fb = torch.from_numpy(img.copy()).cuda()
    legacy.postprocess(fb, w, h, bloom_threshold=1.0, bloom_strength=strength, exposure_gain=3.0)
    want = LO.postprocess(img, 1.0, strength, 3.0)
    # 124 products of a bloomed value, then the tone curve: a few FP32 roundings of values <= 1
    np.testing.assert_allclose(fb.cpu().numpy(), want, rtol=2e-5, atol=2e-6)
