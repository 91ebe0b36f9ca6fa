"""Bias gradients are sums in a fixed order: the same bits on every call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [8, 72, 256])
def test_bias_gradients_repeat(gpu, batch):
    import torch
    from merge_fusion_gb300 import proposer as mp
    from oracle import proposer as op
    rng = np.random.default_rng(batch)
    pr = mp.PoseProposer(max_batch=batch)
    pr.set_params(mp.init_params(7))
    x = torch.from_numpy(rng.uniform(0.4, 4.0, (batch, 60, 80, 2)).astype(np.float16)).cuda()
    # targets whose sums cancel: the order of the additions shows
    t = torch.from_numpy((rng.normal(size=(batch, 6)) * 10.0 ** rng.integers(-3, 4, (batch, 6))).astype(np.float32)).cuda()
    biases = [(off, int(np.prod(shp))) for off, shp in op.layout()[0]][1::2]
    first = pr.gradients(x, t)[1]
    for _ in range(10):
        again = pr.gradients(x, t)[1]
        for off, n in biases:
            assert np.array_equal(first[off:off + n].view(np.uint32), again[off:off + n].view(np.uint32)), off
