"""The tone map's rows per thread change with the image's size, not its values: a pixel
at the same place (u, v) of a uniform image has the same bits on both sides of one
wave of threads."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strength", [0.0, 0.5])
@pytest.mark.parametrize("colour", [(0.3, 0.7, 0.1), (0.04, 0.02, 0.9)])
def test_same_bits_on_both_sides_of_a_wave(cuda, colour, strength):
    from blackhole_b200 import legacy

    p = torch.cuda.get_device_properties(0)
    side = int((p.multi_processor_count * p.max_threads_per_multi_processor) ** 0.5)
    images = []
    for k in (1, 2):  # side^2 pixels are one wave, (2 side)^2 are four
        fb = torch.tensor((*colour, 1.0), device="cuda").repeat((k * side) ** 2, 1)
        legacy.postprocess(fb, k * side, k * side, bloom_strength=strength)
        images.append(fb.view(k * side, k * side, 4))
    torch.cuda.synchronize()
    assert torch.equal(images[0], images[1][::2, ::2])
