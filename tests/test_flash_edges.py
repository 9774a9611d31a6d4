"""bf16 tensor-core attention at the edges of its tiles: query rows at and around 128 and 256 (a second query tile that is empty,
one row long, full), the diagonal tile, and the last rows' stores, which must not reach behind the output."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("S", [127, 128, 129, 255, 257, 384])
@pytest.mark.parametrize("causal", [False, True])
def test_flash_tile_edges(lib_built, device, D, S, causal):
    import torch
    from importlib import import_module
    _lib = import_module("luminal_jl_b200._lib")
    B, H, pad = 2, 3, 512
    n = B * H * S * D
    gen = torch.Generator().manual_seed(S * 1000 + D)
    q, k, v = (torch.randn(B, H, S, D, generator=gen).to(torch.bfloat16).cuda() for _ in range(3))
    buf = torch.full((n + 2 * pad,), 7.0, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    scale = 1.0 / D ** 0.5
    _lib.call("lmb200_flash_attention", device.handle, C.c_void_p(buf.data_ptr() + 2 * pad), C.c_void_p(q.data_ptr()),
              C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()), _lib.BF16, B, H, S, D, scale, int(causal))
    device.sync()
    s = q.double() @ k.double().transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    ref = s.softmax(-1) @ v.double()
    got = buf[pad:pad + n].view(B, H, S, D).double()
    # weights and result are each rounded to bf16 (2^-9 of a value): 2^-8 of the largest |v| bounds the weighted mean
    assert (got - ref).abs().max() <= 2.0 ** -8 * v.double().abs().max()
    assert bool((buf[:pad] == 7).all()) and bool((buf[pad + n:] == 7).all())
