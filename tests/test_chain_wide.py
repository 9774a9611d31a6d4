"""Chained residual projections of more row groups than the chip has clusters (several tiles per cluster, a partly empty last round), with a
reduction so short that any other GEMV of it would be launched by itself: the norm that follows must see every slot of the sums of squares and
no stale one."""
import numpy as np
import pytest

import gibutar_oracle as G
import luminal_oracle as O
from test_decode_parity import BF16_REL_TOL, make_model, rel_err
from test_layered import agree, retention

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,heads,kv,batch", [(4352, 34, 17, 3), (8192, 64, 8, 17)])
def test_wide_residual_short_reduction(lib_built, device, hidden, heads, kv, batch):
    L = lib_built
    cfg = dict(n_layers=2, hidden=hidden, n_heads=heads, n_kv_heads=kv, intermediate=1024, vocab=300, eps=1e-5, rope_base=10000.0)
    rng = np.random.default_rng(hidden)
    w = {}
    for name in O.synth_llama_weights(dict(cfg, hidden=heads, n_kv_heads=kv, intermediate=8, vocab=8), seed=1):
        part = name.split(".")[-2]
        rows = dict(q_proj=hidden, k_proj=128 * kv, v_proj=128 * kv, o_proj=hidden, gate_proj=1024, up_proj=1024, down_proj=hidden, embed_tokens=300, lm_head=300).get(part)
        if rows is None:
            w[name] = (1.0 + 0.02 * rng.standard_normal(hidden)).astype(np.float32)
        else:
            w[name] = 0.02 * rng.standard_normal((rows, 1024 if part == "down_proj" else hidden), dtype=np.float32)
    tokens = rng.integers(0, 300, (batch, 3)).astype(np.int32)
    ref = O.CachedLlama(w, cfg, batch, 16)
    model = make_model(L, device, cfg, w, "bf16")
    sess = L.Session(model, batch, 16)
    sess.set_capture(True)
    for i in range(3):
        ref_logits, ref_hidden = ref.forward(tokens[:, i:i + 1], return_hidden=True)
        _, logits = sess.decode_step(np.ascontiguousarray(tokens[:, i]), want_logits=True)
        for l in range(2):
            assert rel_err(sess.layer_output(l), ref_hidden[l][:, -1, :]) <= BF16_REL_TOL, (i, l)
        assert rel_err(logits, ref_logits[:, -1, :]) <= 2 * BF16_REL_TOL, i
    sess.close(); model.close()


def test_wide_layered_short_reduction(lib_built, device):
    L = lib_built
    cfg = dict(architecture="Gibutar", width=4352, vocab=131, norm=dict(eps=3e-5), logit_softcap=9.0,
               layers=[retention(heads=2, dim=64, vdim=128, dims=64, ff=512, decay=[0.9, 0.97]) for _ in range(2)])
    w = G.random_weights(cfg, seed=11)
    ids = [int(t) for t in np.random.default_rng(4).integers(0, 131, 6)]
    want = G.forward(cfg, w, ids)
    model = L.models.build_model(device, cfg, "bf16")
    model.set_weights(w)
    sess = L.Session(model, 1, 16)
    got = [sess.decode_step(np.array([t], np.int32), want_logits=True)[1][0] for t in ids]
    assert agree(np.stack(got), want, "bf16")
    sess.close(); model.close()
