"""Training batches whose targets start anywhere in a flat buffer (a float array has no
other alignment than 4 bytes) give the gradients of an aligned copy; inputs off 16
bytes are refused before anything is launched."""
from __future__ import annotations

import pytest
import torch

from test_gpu_surrogate import rand_inputs, synthetic_targets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [1, 2, 3])
def test_targets_at_any_float(cuda, off):
    from blackhole_b200 import surrogate as S

    B = 256
    net = S.Surrogate(max_batch=B, seed=4)
    x, t = rand_inputs(B, 1).cuda(), torch.from_numpy(synthetic_targets(B, 2)).cuda()
    want, loss_want = net.gradients(x, t)
    flat = torch.empty(off + 16 * B, device="cuda")
    view = flat[off:].view(B, 16)
    view.copy_(t)
    assert view.data_ptr() % 16 == 4 * off
    got, loss = net.gradients(x, view)
    assert torch.equal(got, want)
    # the loss is a sum of 8 warps' sums by atomics, in any order: 7 roundings
    torch.testing.assert_close(loss, loss_want, rtol=7 * 2.0**-23, atol=0.0)
    assert net.device_error() == 0


def test_inputs_off_16_bytes_are_refused(cuda):
    from blackhole_b200 import surrogate as S

    net = S.Surrogate(max_batch=128, seed=4)
    x = torch.zeros(4 * 128 + 1, device="cuda")[1:].view(128, 4)
    t = torch.from_numpy(synthetic_targets(128, 2)).cuda()
    with pytest.raises(RuntimeError, match="16 bytes"):
        net.gradients(x, t)
    before = net.get_params()
    with pytest.raises(RuntimeError, match="16 bytes"):
        net.train_step(x, t, 1e-3)
    assert (net.get_params() == before).all() and net.device_error() == 0
