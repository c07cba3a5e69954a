"""The caches' device memory across growth and reset: blocks that a cache takes again hold what fresh ones would."""

import threading

import pytest
import torch

import turboquant_b200 as tq

pytestmark = pytest.mark.gpu


def _fill(cache, sizes, seed, sketch):
    g = torch.Generator(device="cuda").manual_seed(seed)
    cfg, out = cache.config, []
    for layer in range(cfg.num_layers):
        for n in sizes:
            k, v = (torch.randn((cfg.batch, cfg.num_kv_heads, n, cfg.head_dim), generator=g, device="cuda") for _ in range(2))
            q = torch.randn((cfg.batch, 2 * cfg.num_kv_heads, 1, cfg.head_dim), generator=g, device="cuda")
            r = cache.prefill(layer, k, v, q) if sketch else cache.prefill(layer, k, v)
            out += [r.k, r.v] + ([r.logit_bias] if sketch else [])
        step = (k[:, :, :1].contiguous(), v[:, :, :1].contiguous(), q, tq.AttendConfig(0.1, 2))
        out.append((cache.decode_fused if sketch else cache.decode)(layer, *step).fused)
    return out


@pytest.mark.parametrize("sketch", [False, True])
@pytest.mark.parametrize("first,second", [((100, 300), (100, 300)), ((700,), (30, 500)), ((40,), (900, 1)), ((5, 5), (1,))])
def test_reset_cache_equals_fresh_cache(first, second, sketch):
    cfg = tq.CacheConfig(bits=3, head_dim=128, num_kv_heads=2, num_layers=3, batch=2, outlier_blocks=0 if sketch else tq.ALL_BLOCKS)
    make = tq.TqCache if sketch else tq.PqoCache
    used, fresh = make(cfg), make(cfg)
    for seed in (1, 2):
        _fill(used, first, seed, sketch)
        used.reset()
        assert used.memory_usage() == 0 and used.seq_len(0) == 0
        if not sketch:
            assert used.capacity(0) == 0 and used.layer_ptrs(0) == [None] * 4
    for a, b in zip(_fill(used, second, 9, sketch), _fill(fresh, second, 9, sketch)):
        assert torch.equal(a, b)
    assert used.memory_usage() == fresh.memory_usage()


def test_reset_gives_large_blocks_back():
    # 2 GB of rows, of which a cache keeps at most 512 MB
    cache = tq.PqoCache(tq.CacheConfig(bits=4, head_dim=128, num_kv_heads=8, num_layers=8, batch=16))
    x = torch.zeros((16, 8, 16384, 128), dtype=torch.bfloat16, device="cuda")
    free0 = torch.cuda.mem_get_info()[0]
    for layer in range(8):
        cache.prefill(layer, x, x)
    cache.reset()
    assert free0 - torch.cuda.mem_get_info()[0] <= (512 + 64) << 20


@pytest.mark.parametrize("sketch", [False, True])
def test_growth_beside_a_capture(sketch):
    # a cache may grow on its stream while another thread has a graph of its own under capture
    cfg = tq.CacheConfig(bits=3, head_dim=128, num_kv_heads=2, num_layers=1, batch=1, outlier_blocks=0 if sketch else tq.ALL_BLOCKS)
    cache = (tq.TqCache if sketch else tq.PqoCache)(cfg)
    rows = torch.randn((1, 2, 200, 128), device="cuda")
    y, s1, s2, failed = torch.zeros(8, device="cuda"), torch.cuda.Stream(), torch.cuda.Stream(), []
    torch.cuda.synchronize()

    def fill():
        try:
            with torch.cuda.stream(s2):
                for _ in range(4):
                    cache.prefill(0, rows, rows, rows[:, :, :1].contiguous()) if sketch else cache.prefill(0, rows, rows)
        except Exception as e:
            failed.append(e)

    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s1):
        graph.capture_begin(capture_error_mode="thread_local")
        y.add_(1.0)
        t = threading.Thread(target=fill)
        t.start()
        t.join()
        y.add_(1.0)
        graph.capture_end()
    graph.replay()
    torch.cuda.synchronize()
    assert not failed and cache.seq_len(0) == 800 and y[0].item() == 2.0


def test_one_layer_of_many():
    # the growths of one layer of 80: its first allocation may hold blocks for all, the later ones two each
    cache = tq.PqoCache(tq.CacheConfig(bits=4, head_dim=128, num_kv_heads=8, num_layers=80, batch=1))
    x = torch.zeros((1, 8, 64, 128), dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    free0, caps = torch.cuda.mem_get_info()[0], set()
    for _ in range(200):
        cache.prefill(79, x, x)
        caps.add(cache.capacity(79))
    block = lambda cap: 8 * cap * (2 * 64 + 2 * 8) + 1024
    bound = 80 * block(min(caps)) + sum(2 * block(c) for c in caps)
    assert free0 - torch.cuda.mem_get_info()[0] <= bound + len(caps) * (4 << 20)      # 2 MB granules of the driver
    assert len(caps) > 10
