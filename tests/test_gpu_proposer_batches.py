"""The proposer's gradient passes at batches whose row counts are not whole
64-row tiles (160 and 480 rows of the last convolution's gradient, 8 and 24 of
the linear layers') and at one that is, against the oracle with BF16 rounding at
the same points; tolerances as for the batch of 16 (FP32 accumulation order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [8, 24, 64])
def test_gradients_match_oracle(gpu, batch):
    import torch
    from merge_fusion_gb300 import proposer as mp
    from oracle import proposer as op
    rng = np.random.default_rng(40 + batch)
    pr = mp.PoseProposer(max_batch=batch + 8)
    p = mp.init_params(7)
    p = (p + 0.02 * rng.normal(size=p.shape).astype(np.float32) * op.trainable_mask()).astype(np.float32)
    pr.set_params(p)
    x = rng.uniform(0.4, 4.0, (batch, 60, 80, 2)).astype(np.float16)
    x[rng.uniform(size=x.shape) < 0.1] = 0
    t = rng.normal(size=(batch, 6)).astype(np.float32)
    _, cache = op.forward(p.astype(np.float64), x.astype(np.float64), quantize=True)
    loss_o, g_o = op.backward(cache, t)
    loss, g = pr.gradients(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda())
    assert abs(loss - loss_o) <= 2e-3 * loss_o
    for i, (off, shp) in enumerate(op.layout()[0]):
        n = int(np.prod(shp))
        a, b = g[off:off + n], g_o[off:off + n]
        assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b), i
    assert np.all(g[~op.trainable_mask()] == 0)
