"""Training batches at the edges of the kernels' splits (128-row tiles, 512-row weight-
gradient splits, 1024 for the head), with one handle used at several batch sizes in
turn, against the oracle's backward pass (BF16 rounding emulated at the same points;
the tolerance of test_gpu_surrogate.py's gradient test)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import surrogate_oracle as so
from test_gpu_surrogate import rand_inputs, synthetic_targets

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net():
    from blackhole_b200 import surrogate as S

    return S.Surrogate(max_batch=2176, seed=9)


@pytest.mark.parametrize("B", [128, 2176, 512, 640, 1024, 1152, 128])
def test_gradients_at_split_edges(cuda, net, B):
    from blackhole_b200 import surrogate as S

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
    used = grad[S.weight_slices()[0][0]].reshape(256, 192)
    assert not used[:, S.N_FEATURES_USED:].any()  # the padded feature columns have no gradient
