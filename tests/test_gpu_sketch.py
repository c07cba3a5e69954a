"""GPU kernels of the sign sketch at the edges of their tiles and on awkward vectors."""
import ctypes

import numpy as np
import pytest
import torch

import turboquant_b200 as tq
from turboquant_b200._lib import lib

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("dim", [32, 64, 96, 128, 256])
@pytest.mark.parametrize("group,q_len,kv_len", [(1, 1, 1), (4, 1, 33), (3, 5, 127), (1, 16, 128), (1, 65, 129), (4, 25, 300), (8, 2, 97)])
def test_logit_bias_at_tile_edges(dim, group, q_len, kv_len):
    # rows 1 .. 100 around the 16-row and 64-row tiles, tokens around the 8-, 32- and 128-token tiles
    hkv, stride = 2, kv_len + 3
    g = torch.Generator(device="cuda").manual_seed(dim + kv_len)
    rq = torch.randn((hkv * group, q_len, dim), generator=g, device="cuda") * torch.exp(2 * torch.randn((hkv * group, q_len, 1), generator=g, device="cuda"))
    signs = torch.randint(0, 256, (hkv, stride, dim // 8), generator=g, device="cuda", dtype=torch.uint8)
    norms = torch.rand((hkv, stride), generator=g, device="cuda").to(torch.float16)
    bias = torch.full((hkv * group, q_len, kv_len), 7.0, device="cuda")
    assert lib.tqb_qjl_logit_bias(dim, _p(rq), _p(signs), _p(norms), _p(bias), 0, hkv * group, hkv, q_len, kv_len, stride,
                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    bits = torch.stack([(signs >> b) & 1 for b in range(8)], -1).reshape(hkv, stride, dim)[:, :kv_len].double() * 2 - 1
    c = (norms[:, :kv_len].double() * float(np.float32(np.sqrt(np.pi / 2)) / np.sqrt(np.float32(dim)))).repeat_interleave(group, 0)
    want = torch.einsum("hid,htd->hit", rq.double(), bits.repeat_interleave(group, 0)) * c[:, None]
    # every product is exact (three bf16 terms of rq, +-1): only the f32 sum of 3 dim terms rounds, at most 2^-23 of
    # the running magnitude per addition, and the final scaling twice
    bound = (3 * dim + 4) * 2.0 ** -23 * rq.double().abs().sum(-1)[..., None] * c[:, None] + 1e-30
    assert bool(((bias.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("spread", [0.0, 1.0, 2.0, 4.0])
@pytest.mark.parametrize("dim", [32, 64, 128, 256])
def test_logit_bias_is_no_less_exact_than_the_sequential_sum(dim, spread):
    # against 64 bits, beside f32 additions from the first element to the last; log-normal spread over the elements
    hq, hkv, q_len, kv_len = 8, 2, 37, 300
    g = torch.Generator(device="cuda").manual_seed(dim)
    rq = torch.randn((hq, q_len, dim), generator=g, device="cuda") * torch.exp(spread * torch.randn((hq, q_len, dim), generator=g, device="cuda"))
    signs = torch.randint(0, 256, (hkv, kv_len, dim // 8), generator=g, device="cuda", dtype=torch.uint8)
    norms = (torch.rand((hkv, kv_len), generator=g, device="cuda") + 0.5).to(torch.float16)
    bias = torch.empty((hq, q_len, kv_len), device="cuda")
    assert lib.tqb_qjl_logit_bias(dim, _p(rq), _p(signs), _p(norms), _p(bias), 0, hq, hkv, q_len, kv_len, kv_len, _stream()) == 0
    pm = (torch.stack([(signs >> b) & 1 for b in range(8)], -1).reshape(hkv, kv_len, dim).float() * 2 - 1).repeat_interleave(hq // hkv, 0)
    c = (norms.float() * float(np.float32(np.sqrt(np.pi / 2)) / np.sqrt(np.float32(dim)))).repeat_interleave(hq // hkv, 0)[:, None]
    want = torch.einsum("hid,htd->hit", rq.double(), pm.double()) * c.double()
    seq = torch.zeros_like(bias)
    for d in range(dim):
        seq = seq + rq[:, :, d, None] * pm[:, None, :, d]
    err, err_seq = ((t.double() - want).norm().item() for t in (bias, seq * c))
    assert err <= err_seq, (err, err_seq)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dim", [32, 64, 128, 256])
@pytest.mark.parametrize("group,q_len,kv_len", [(1, 1, 1), (1, 1, 128), (1, 1, 1000), (2, 1, 129), (1, 2, 300), (3, 1, 257)])
def test_logit_bias_of_few_rows(dim, group, q_len, kv_len, dtype):
    # one row, and two from 128 dims on, are summed from the first element to the last; beyond that on the tensor cores
    hkv, stride, rows = 3, kv_len + 1, group * q_len
    g = torch.Generator(device="cuda").manual_seed(dim + kv_len)
    rq = torch.randn((hkv * group, q_len, dim), generator=g, device="cuda")
    signs = torch.randint(0, 256, (hkv, stride, dim // 8), generator=g, device="cuda", dtype=torch.uint8)
    norms = torch.rand((hkv, stride), generator=g, device="cuda").to(torch.float16)
    bias = torch.empty((hkv * group, q_len, kv_len), device="cuda", dtype=dtype)
    assert lib.tqb_qjl_logit_bias(dim, _p(rq), _p(signs), _p(norms), _p(bias), 0 if dtype == torch.float32 else 2, hkv * group, hkv, q_len, kv_len,
                                  stride, _stream()) == 0
    pm = (torch.stack([(signs >> b) & 1 for b in range(8)], -1).reshape(hkv, stride, dim)[:, :kv_len].float() * 2 - 1).repeat_interleave(group, 0)
    factor = np.float32(np.sqrt(np.pi / 2)) / np.sqrt(np.float32(dim))
    c = (norms[:, :kv_len].float() * float(factor)).repeat_interleave(group, 0)[:, None]
    seq = torch.zeros((hkv * group, q_len, kv_len), device="cuda")
    for d in range(dim):
        seq = seq + rq[:, :, d, None] * pm[:, None, :, d]
    if rows == 1 or (rows == 2 and dim >= 128):
        assert torch.equal(bias, (seq * c).to(dtype))
    else:   # the additions of both sums: dim roundings of 2^-24 each, and the output's own
        bound = rq.double().abs().sum(-1)[..., None] * c.double() * dim * 2.0 ** -23 + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23) * (seq * c).abs()
        assert ((bias.double() - (seq * c).double()).abs() <= bound).all()


@pytest.mark.parametrize("dim", [32, 64, 96, 128, 256])
def test_logit_bias_of_infinities_and_nan(dim):
    # a NaN whose bits are all in the low half of the word is none the less one; rows without any are untouched
    rq = torch.randn((8, 5, dim), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    bits = rq.view(torch.int32)
    bits[0, 0, 3], bits[0, 1, dim - 1], bits[3, 2, 7] = 0x7F800001, 0x7FC00000, -0x7FFF8000     # NaN; the last one 0x80008000: a denormal
    bits[4, 4, 0] = 0x7F7F8001                                                                   # the finite end of the range
    rq[5, 1, 2] = float("inf")
    rq[6, 2, 5], rq[6, 2, 9] = float("inf"), float("-inf")
    signs = torch.zeros((2, 40, dim // 8), dtype=torch.uint8, device="cuda")                     # every sign -1
    norms = torch.ones((2, 40), dtype=torch.float16, device="cuda")
    bias = torch.empty((8, 5, 40), device="cuda")
    assert lib.tqb_qjl_logit_bias(dim, _p(rq), _p(signs), _p(norms), _p(bias), 0, 8, 2, 5, 40, 40, _stream()) == 0
    nan = torch.zeros((8, 5), dtype=torch.bool, device="cuda")
    nan[0, 0] = nan[0, 1] = nan[6, 2] = True
    assert torch.equal(bias.isnan(), nan[..., None].expand_as(bias))
    assert torch.equal(bias[5, 1], torch.full((40,), float("-inf"), device="cuda"))
    nan[5, 1] = True
    want = -rq.double().sum(-1) * float(np.float32(np.sqrt(np.pi / 2)) / np.sqrt(np.float32(dim)))
    err = (bias.double() - want[..., None]).abs() / rq.double().abs().sum(-1)[..., None]
    assert (err[~nan] < 1e-6).all()


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _awkward(n, dim, seed):
    """Vectors with sums that tie or nearly cancel, all-zero ones, denormal and huge ones, infinities and NaN among ordinary ones."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((n, dim), generator=g, device="cuda")
    kind = torch.arange(n, device="cuda") % 9
    x[kind == 1] = 0.0
    x[kind == 2] = x[kind == 2].sign()                        # +-1: many sums are exactly zero in some order
    x[kind == 3] = x[kind == 3] * 1e-30
    x[kind == 4] = x[kind == 4] * 1e30
    x[kind == 5] = torch.round(x[kind == 5] * 4)              # small integers
    if n > 60:
        x[7, 3], x[16, dim - 1], x[25, 0] = float("inf"), float("nan"), float("-inf")
    return x


@pytest.mark.parametrize("bits", [3, 4])
@pytest.mark.parametrize("dim,n", [(32, 16), (32, 1000), (64, 33), (64, 700), (128, 17), (128, 31), (128, 2500), (256, 20), (256, 900)])
def test_qjl_quantize_batches_equal_single_vectors(dim, n, bits):
    # the bytes of a batch on the tensor cores are those of the sequential sums, which calls of a few vectors take
    cfg = tq.TurboQuantConfig(bits, dim).with_seed(7)
    x = _awkward(n, dim, dim + n)
    got = tq.qjl_quantize_batch(cfg, x, 5)
    pieces = [tq.qjl_quantize_batch(cfg, x[a:a + 15], 5) for a in range(0, n, 15)]
    for i, name in enumerate(("packed", "scales", "signs", "rnorms")):
        assert torch.equal(got[i], torch.cat([p[i] for p in pieces])), name


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("dim", [32, 64, 128, 256])
def test_residual_sketch_tiles_equal_single_vectors(dim, dtype):
    n, rpg, gs, off = 2048 + 37, 139, 200, 11                 # 15 groups of 139 rows at rows 11.. of 200
    x = _awkward(n, dim, dim).to(dtype)
    xhat = (x.float() * 0.9 + 0.02).nan_to_num(1.0, 2.0, -2.0)
    rb = tq.api.rademacher_bits(dim, 9, x.device)
    code = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}[dtype]
    outs = []
    for step in (n, rpg):                                     # one call on the tensor cores; one per group, sequential sums
        signs = torch.zeros((15 * gs, dim // 8), dtype=torch.uint8, device="cuda")
        norms = torch.zeros((15 * gs,), dtype=torch.int16, device="cuda")
        for a in range(0, n, step):
            assert lib.tqb_residual_sketch(dim, _p(rb), _p(x[a:]), code, _p(xhat[a:]), step, _p(signs[a // rpg * gs:]), _p(norms[a // rpg * gs:]),
                                           rpg, gs, off, _stream()) == 0
        outs.append((signs, norms))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("dim", [32, 64, 128, 256])
def test_projections_of_many_queries_equal_single_ones(dim):
    q = _awkward(2048 + 13, dim, 3)
    many = tq.query_projections(q, dim, 21)
    few = torch.cat([tq.query_projections(q[a:a + 100], dim, 21) for a in range(0, len(q), 100)])
    assert torch.equal(many.nan_to_num(7.0, 8.0, -8.0), few.nan_to_num(7.0, 8.0, -8.0))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("bits,dim,batch,group", [(3, 128, 1, 1), (3, 128, 5, 4), (4, 128, 3, 8), (3, 64, 2, 2), (4, 32, 1, 3), (3, 256, 2, 4)])
def test_decode_input_in_one_launch_equals_separate_kernels(bits, dim, batch, group, dtype):
    # a query that starts off a 16-byte boundary takes the separate kernels
    hkv, steps = 2, 3
    cfg = tq.CacheConfig(bits=bits, head_dim=dim, num_kv_heads=hkv, num_layers=1, batch=batch, outlier_blocks=0)
    att, outs = tq.AttendConfig(dim ** -0.5, group), []
    for shift in (0, 1):
        g = torch.Generator(device="cuda").manual_seed(dim + batch)
        cache = tq.TqCache(cfg)
        got = []
        for step in range(steps):
            k, v = (torch.randn((batch, hkv, 1, dim), generator=g, device="cuda").to(dtype) for _ in range(2))
            q = torch.randn((batch, hkv * group, 1, dim), generator=g, device="cuda").to(dtype)
            if step == 1:
                k[0, 0] = 0
                k[-1, -1, 0, 3] = 1e4
            hold = torch.zeros(q.numel() + shift, dtype=dtype, device="cuda")
            hold[shift:] = q.reshape(-1)
            got.append(cache.decode_fused(0, k, v, hold[shift:].view(q.shape), att).fused)
        r = cache.decode(0, k, v, q).dequantized
        outs.append(got + [r.k, r.v, r.logit_bias])
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype,ulp", [(torch.float32, 2.0 ** -22), (torch.float16, 2.0 ** -10), (torch.bfloat16, 2.0 ** -7)])
@pytest.mark.parametrize("dim,q_len,batch", [(32, 70, 2), (64, 65, 2), (128, 64, 2), (256, 45, 3)])
def test_bias_of_many_queries_equals_few(dim, q_len, batch, dtype, ulp):
    # from 2,048 queries on (2 x 16 x 64) 16-bit ones are projected on the tensor cores; pieces take the sequential sums.  Both
    # sums are exact to f32 rounding, so the bias differs by its own last place at most
    g = torch.Generator(device="cuda").manual_seed(dim)
    cfg = tq.CacheConfig(bits=3, head_dim=dim, num_kv_heads=4, num_layers=1, batch=batch, outlier_blocks=0)
    k, v = (torch.randn((batch, 4, 50, dim), generator=g, device="cuda").to(dtype) for _ in range(2))
    q = torch.randn((batch, 16, q_len, dim), generator=g, device="cuda").to(dtype)
    many = tq.TqCache(cfg).prefill(0, k, v, q).logit_bias
    few = torch.cat([tq.TqCache(cfg).prefill(0, k, v, q[:, :, a:a + 33].contiguous()).logit_bias for a in range(0, q_len, 33)], dim=2)
    scale = few.float().abs().max()
    assert ((many.float() - few.float()).abs() <= ulp * few.float().abs() + 2.0 ** -20 * scale).all()
