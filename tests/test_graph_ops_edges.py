"""The float32 graph matmul at the edges of its 32 x 32 tiles and 128-wide k steps, and the value sum of the float32 decode attention
at head dimensions whose threads do not divide evenly."""
import ctypes

import numpy as np
import pytest
import torch

from luminal_jl_b200 import _lib

import luminal_oracle as O
from test_decode_parity import LOGIT_TOL, make_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,M,K,N", [(0, 1, 1, 1), (0, 32, 128, 32), (0, 33, 129, 31), (0, 5, 15, 70), (0, 64, 127, 33), (0, 31, 688, 256), (3, 17, 257, 65)])
def test_matmul_edges(lib_built, device, batch, M, K, N):
    g = torch.Generator(device="cuda").manual_seed(M * 1000 + K)
    lead = (batch,) if batch else ()
    a, b = torch.randn(*lead, M, K, device="cuda", generator=g), torch.randn(*lead, K, N, device="cuda", generator=g)
    out = torch.full((*lead, M, N), float("nan"), device="cuda")
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(t.data_ptr()) for t in (out, a, b)]
    _lib.call("lmb200_matmul", device.handle, p[0], p[1], a.dim(), _lib.dims(a.shape), p[2], b.dim(), _lib.dims(b.shape))
    device.sync()
    exact = a.double() @ b.double()
    # K roundings of a sum whose terms add up to at most |a| |b|
    bound = (K + 8) * 2.0 ** -24 * (a.double().abs() @ b.double().abs())
    assert ((out.double() - exact).abs() <= bound + 1e-30).all()


@pytest.mark.parametrize("heads,hidden", [(4, 64), (4, 192), (2, 192), (2, 256), (2, 288)])       # head dimensions 16, 48, 96, 128, 144
def test_f32_attention_head_dims(lib_built, device, heads, hidden):
    L = lib_built
    cfg = dict(n_layers=2, hidden=hidden, n_heads=heads, n_kv_heads=heads, intermediate=64, vocab=128, eps=1e-5, rope_base=10000.0)
    w = O.synth_llama_weights(cfg, seed=5)
    prompt = O.synth_tokens(5, 1000, (2, 70), cfg["vocab"])
    ref_tok, ref_log = O.CachedLlama(w, cfg, 2, 96).greedy(prompt, 4)
    model = make_model(L, device, cfg, w, "f32")
    sess = L.Session(model, 2, 96)
    tok, log = L.greedy_generate(sess, prompt, 4, want_logits=True)
    assert np.abs(log - ref_log).max() <= LOGIT_TOL and np.array_equal(tok, ref_tok)
    sess.close(); model.close()


@pytest.mark.parametrize("dims,perm", [((96, 100, 4000), (2, 1, 0)), ((96, 1000, 400), (2, 1, 0)), ((16, 1500, 1500), (1, 2, 0)), ((7, 33, 65), (2, 0, 1))])
def test_permute_routes(lib_built, device, dims, perm):
    """Either index width, around the rule on the distance between a warp's reads (1.6 MB, 1.6 MB, too few lanes, small)."""
    a = torch.arange(int(np.prod(dims)), device="cuda", dtype=torch.int32).view(torch.float32).view(dims)        # bit patterns, all different
    out = torch.empty([dims[p] for p in perm], device="cuda")
    torch.cuda.synchronize()
    _lib.call("lmb200_permute", device.handle, ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(a.data_ptr()), len(dims), _lib.dims(dims), (ctypes.c_int32 * len(dims))(*perm))
    device.sync()
    assert torch.equal(out.view(torch.int32), a.view(torch.int32).permute(perm))
