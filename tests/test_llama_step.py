"""The small float32 Llama's step as one launch, against the oracle: row groups that do not fill 16 rows, k that does not fill 32, grouped heads, contexts around its
16-key blocks and one round of its warps, several sequences, unequal positions, end of text."""
import numpy as np
import pytest

import luminal_oracle as O
from test_decode_parity import LOGIT_TOL, make_model

pytestmark = pytest.mark.gpu


def config(hidden, heads, kv, ffn, vocab, layers=2):
    return dict(n_layers=layers, hidden=hidden, n_heads=heads, n_kv_heads=kv, intermediate=ffn, vocab=vocab, eps=1e-5, rope_base=10000.0)


@pytest.mark.parametrize("cfg,batch,prompt_len,capacity", [
    (config(32, 1, 1, 8, 16), 1, 1, 16), (config(64, 2, 1, 88, 203), 2, 14, 48), (config(256, 8, 8, 688, 1024, 4), 1, 120, 144), (config(96, 3, 3, 104, 50), 3, 31, 64),
    (config(512, 8, 2, 1408, 3001), 4, 126, 160), (config(1024, 8, 4, 4096, 600), 4, 5, 32), (config(384, 3, 1, 1000, 130), 1, 290, 320)])
def test_step_against_oracle(lib_built, device, cfg, batch, prompt_len, capacity):
    L = lib_built
    w = O.synth_llama_weights(cfg, seed=5)
    prompt = O.synth_tokens(5, 1000, (batch, prompt_len), cfg["vocab"])
    n = 8
    ref_tok, ref_log = O.CachedLlama(w, cfg, batch, capacity).greedy(prompt, n)
    model = make_model(L, device, cfg, w, "f32")
    sess = L.Session(model, batch, capacity)
    before = device.launch_count()
    logits = sess.prefill(prompt)
    assert device.launch_count() - before == prompt_len            # one launch a token
    tok, log = L.greedy_generate(L.Session(model, batch, capacity), prompt, n, want_logits=True)
    assert np.abs(log - ref_log).max() <= LOGIT_TOL and np.array_equal(tok, ref_tok)
    assert np.abs(logits - ref_log[:, 0]).max() <= LOGIT_TOL
    assert np.array_equal(sess.decode_n(ref_tok[:, 0].astype(np.int32), n - 1).T, ref_tok[:, 1:])
    sess.close(); model.close()


def test_layer_outputs_and_unequal_positions(lib_built, device):
    L = lib_built
    cfg = config(128, 4, 2, 200, 97, layers=3)
    w = O.synth_llama_weights(cfg, seed=8)
    model = make_model(L, device, cfg, w, "f32")
    prompts = [O.synth_tokens(9, 100 + b, (1, n), cfg["vocab"])[0] for b, n in enumerate((19, 3, 40))]
    sess = L.Session(model, 3, 64)
    got = sess.prefill_ragged([p.astype(np.int32) for p in prompts])
    refs = []
    for b, p in enumerate(prompts):
        one = O.CachedLlama(w, cfg, 1, 64)
        tok, log = one.greedy(p[None], 5)
        refs.append((tok[0], log[0]))
        assert np.abs(got[b] - log[0, 0]).max() <= LOGIT_TOL
    toks = sess.decode_n(np.array([r[0][0] for r in refs], np.int32), 4)
    assert np.array_equal(toks.T, np.stack([r[0][1:] for r in refs]))
    sess.close()
    sess = L.Session(model, 1, 64)
    sess.set_capture(True)
    ref = O.CachedLlama(w, cfg, 1, 64)
    for t in prompts[1]:
        _, hidden = ref.forward(np.array([[t]]), return_hidden=True)
        sess.decode_step(np.array([t], np.int32))
        for l in range(cfg["n_layers"]):
            assert np.abs(sess.layer_output(l) - np.asarray(hidden[l]).reshape(1, -1)).max() <= 1e-4 * np.abs(hidden[l]).max()
    sess.close(); model.close()


@pytest.mark.parametrize("heads,kv", [(8, 8), (4, 2), (2, 1)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_values_behind_the_context_do_not_count(lib_built, device, heads, kv, bad):
    """A request that left infinities or NaN in the cache: after a reset, or a step back, what lies behind the context reaches nothing."""
    L = lib_built
    cfg = config(256, heads, kv, 200, 97)
    w = O.synth_llama_weights(cfg, seed=4)
    model = make_model(L, device, cfg, w, "f32")
    prompt = O.synth_tokens(4, 1000, (2, 40), cfg["vocab"])
    sess, clean = L.Session(model, 2, 48), L.Session(model, 2, 48)
    want = [clean.decode_step(np.ascontiguousarray(prompt[:, i]), want_logits=True)[1] for i in range(40)]
    for name in ("model.layers.0.self_attn.k_proj.weight", "model.layers.1.self_attn.v_proj.weight"):
        model.set_weight(name, np.full_like(w[name], bad))
    assert not np.isfinite(sess.prefill(prompt)).any()
    model.set_weights(w)
    sess.reset()
    for i in range(40):
        assert np.array_equal(sess.decode_step(np.ascontiguousarray(prompt[:, i]), want_logits=True)[1], want[i]), i
    sess.close(); clean.close(); model.close()


@pytest.mark.parametrize("vocab,layers,batch,one_launch", [(16384, 1, 1, True), (16385, 1, 1, False), (16384, 1, 2, False), (6553, 1, 4, True), (6554, 1, 4, False),
                                                           (32768, 8, 3, True), (32769, 8, 3, False)])
def test_vocabulary_at_the_rule(lib_built, device, vocab, layers, batch, one_launch):
    L = lib_built
    cfg = config(64, 2, 2, 40, vocab, layers)
    w = O.synth_llama_weights(cfg, seed=2)
    prompt = O.synth_tokens(2, 1000, (batch, 4), vocab)
    ref = O.CachedLlama(w, cfg, batch, 16).greedy(prompt, 2)[1]
    model = make_model(L, device, cfg, w, "f32")
    sess = L.Session(model, batch, 16)
    before = device.launch_count()
    logits = sess.prefill(prompt)
    assert (device.launch_count() - before == 4) is one_launch
    assert np.abs(logits - ref[:, 0]).max() <= LOGIT_TOL
    sess.close(); model.close()
