"""GPU kernels of the sign sketch at the edges of their tiles: the logit bias on the tensor cores."""
import ctypes

import numpy as np
import pytest
import torch

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
