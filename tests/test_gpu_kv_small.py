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


@pytest.mark.parametrize("scores_first", [False, True])
def test_first_calls_on_a_stream_of_their_own(scores_first):
    # a non-blocking stream does not wait for what the default stream still has queued
    rng = np.random.default_rng(3)
    cfg = tq.TurboQuantConfig(3, 128).with_seed(5)
    caches = [tq.QuantizedKVCache(cfg, 1, 5) for _ in range(4)]
    k, v = (rng.standard_normal((700, 128), dtype=np.float32) for _ in range(2))
    q, w = rng.standard_normal(128, dtype=np.float32), rng.random(700, dtype=np.float32)
    for c in caches:
        c.push_batch(0, k, v)
    want = caches[0].attention_scores(0, q), caches[0].weighted_values(0, w)
    for c in caches[1:]:
        torch.cuda._sleep(20_000_000)                       # about 10 ms of work on the default stream
        for _ in range(2):
            with torch.cuda.stream(torch.cuda.Stream()):
                if scores_first:
                    assert np.array_equal(c.attention_scores(0, q), want[0])
                assert np.array_equal(c.weighted_values(0, w), want[1])
        torch.cuda.synchronize()
        assert np.array_equal(c.weighted_values(0, w), want[1])
