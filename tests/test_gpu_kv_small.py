"""QuantizedKVCache calls on short lists (one launch, mapped host memory) against the same calls on long ones."""
import numpy as np
import pytest
import torch

import turboquant_b200 as tq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("dim,n", [(32, 1), (64, 9), (128, 300), (256, 33), (128, 3840), (128, 3841)])
def test_short_lists_equal_the_batch_calls(dim, n, bits):
    # 3,840 entries are the last that go through the mapped page; query projections, scores and sums as the device calls give them
    rng = np.random.default_rng(dim + n)
    cfg = tq.TurboQuantConfig(bits, dim).with_seed(5)
    cache = tq.QuantizedKVCache(cfg, 2, 5)
    k, v = (rng.standard_normal((n, dim), dtype=np.float32) for _ in range(2))
    cache.push_batch(1, k, v)
    for step in range(3):                                   # the ticket and the page are used again
        q = rng.standard_normal(dim, dtype=np.float32)
        w = rng.random(n, dtype=np.float32)
        qd = torch.from_numpy(q).cuda()
        want = tq.qjl_attention_scores(cfg, qd, tq.query_projections(qd, dim, 5)[0], *tq.qjl_quantize_batch(cfg, torch.from_numpy(k).cuda(), 5))
        assert np.array_equal(cache.attention_scores(1, q), want.cpu().numpy())
        packed, scales = tq.qjl_quantize_batch(cfg, torch.from_numpy(v).cuda(), 5)[:2]
        want = tq.weighted_values(cfg, torch.from_numpy(w).cuda(), packed, scales).cpu().numpy()
        assert np.array_equal(cache.weighted_values(1, w), want)
