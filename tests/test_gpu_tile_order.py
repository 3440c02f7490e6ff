"""The persistent tracers take a frame's pixels in 8 x 4 tiles and serve crossings
and finished rays for a whole warp at a time: every pixel of frames at the edges
of a tile, of a band and of a warp is traced once, bit for bit as the oracle's."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (1, 5), (7, 3), (8, 4), (9, 5), (17, 9), (33, 2), (40, 13)])
@pytest.mark.parametrize("integrator", [0, 1])
def test_frame_edges_match_oracle(cuda, oracle, w, h, integrator):
    from blackhole_b200 import kerr

    s = kerr.scene(width=w, height=h, integrator=integrator, max_crossings=1 + 2 * integrator, spin=0.9)
    outs = kerr.alloc_image_outputs(s)
    for v in outs.values():
        v.fill_(-7)
    kerr.trace_image(s, outs)
    torch.cuda.synchronize()
    ref = oracle.trace_pixels(s)
    for k in ("cls", "steps", "n_cross", "r_hit", "g", "flux", "intensity"):
        got = outs[k].cpu().numpy()
        np.testing.assert_array_equal(got, ref[k].reshape(got.shape), err_msg=k)


def test_mixed_frame_in_a_batch_equals_it_alone(cuda):
    from blackhole_b200 import kerr

    scenes = [kerr.scene(width=w, height=h, integrator=1, precision=1, max_crossings=3, spin=0.7)
              for w, h in ((9, 5), (1, 3), (31, 33), (64, 4))]
    batch = kerr.TraceBatch(scenes)
    batch.trace()
    for s, o in zip(scenes, batch.outs):
        alone = kerr.trace_image(s)
        torch.cuda.synchronize()
        for k, v in alone.items():
            assert torch.equal(v, o[k]), k
