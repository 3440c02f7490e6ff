"""Training batches of more than one 128-row tile per SM, where a CTA of the training
pass carries its barriers, accumulators and buffers from tile to tile, against the
oracle's backward pass (the tolerance of test_gpu_surrogate.py's gradient test)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import surrogate_oracle as so
from test_gpu_surrogate import rand_inputs, synthetic_targets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles_per_sm,more", [(1, 1), (2, 0), (2, 5)])
def test_gradients_of_several_tiles_a_cta(cuda, tiles_per_sm, more):
    from blackhole_b200 import surrogate as S

    B = 128 * (tiles_per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more)
    net = S.Surrogate(max_batch=B, seed=9)
    x = rand_inputs(B, B).cuda()
    t = synthetic_targets(B, B + 1)
    grad, loss = net.gradients(x, torch.from_numpy(t).cuda())
    grad, loss = grad.double().cpu().numpy(), loss.cpu().numpy()
    assert net.device_error() == 0
    params = net.get_params().astype(np.float64)
    F = S.features(x).float().cpu().numpy().astype(np.float64)
    out, cache = so.forward(params, F, emulate=True)
    loss_ref, dout = so.loss_and_grad(out, t.astype(np.float64))
    ref = so.backward(params, cache, dout, emulate=True)
    np.testing.assert_allclose(loss, loss_ref, rtol=2e-3)
    for l, (ws, bs) in enumerate(S.weight_slices()):
        for name, sl in (("W", ws), ("b", bs)):
            rel = np.linalg.norm(grad[sl] - ref[sl]) / max(np.linalg.norm(ref[sl]), 1e-30)
            assert rel < 1e-2, (l, name, rel)
