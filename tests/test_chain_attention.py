"""Decode attention as a link of the chained step against the step that launches it: head dimensions, groups, contexts around the 16-key blocks and 64-key stages,
one part or several per head, the newest key alone in its stage, unequal positions, several steps on the same counters; and the chain's limit of links."""
import numpy as np
import pytest

import luminal_oracle as O
from test_decode_parity import BF16_REL_TOL, make_model, rel_err

pytestmark = pytest.mark.gpu


def both(L, model, monkeypatch, batch, capacity, contexts, steps, seed):
    """(logits, tokens) of `steps` forced steps behind random caches, with the attention in the chain and launched."""
    out = []
    for env in ("1", "0"):                                         # 1: also where the library launches it because that is faster
        monkeypatch.setenv("LMB200_CHAIN_ATTENTION", env)
        sess = L.Session(model, batch, capacity)
        rng = np.random.default_rng(seed)
        sess.fill_kv_random(max(contexts), seed)
        sess.set_positions(np.array(contexts, np.int32)) if len(set(contexts)) > 1 else sess.set_position(contexts[0])
        got = []
        for _ in range(steps):
            _, lg = sess.decode_step(rng.integers(0, 500, batch).astype(np.int32), want_logits=True)
            got.append(lg)
        out.append(np.stack(got))
        sess.close()
    return out


@pytest.mark.parametrize("hidden,heads,kv", [(2048, 16, 4), (2048, 32, 8), (2304, 24, 6), (2048, 16, 16), (2048, 16, 8)])
@pytest.mark.parametrize("batch,contexts", [(1, [0]), (1, [1030]), (3, [15]), (2, [63]), (2, [64, 700]), (17, [127]), (5, [16, 0, 255, 64, 128]), (32, [400])])
def test_against_launched_attention(lib_built, device, monkeypatch, hidden, heads, kv, batch, contexts):
    L = lib_built
    model = L.Model(device, dtype="bf16", n_layers=2, hidden=hidden, n_heads=heads, n_kv_heads=kv, intermediate=512, vocab=500, eps=1e-5, rope_base=10000.0)
    model.init_random(seed=5, sigma=0.02)
    contexts = contexts if len(contexts) == batch else contexts * batch
    chain, launched = both(L, model, monkeypatch, batch, max(contexts) + 4, contexts, 4, batch)
    # the same products and sums but for the order of the keys' parts: differences of a bf16 rounding of the attention's outputs
    assert rel_err(chain, launched) <= BF16_REL_TOL / 2
    model.close()


@pytest.mark.parametrize("hidden,heads,kv", [(2048, 16, 4), (3072, 32, 8), (2048, 32, 8), (2048, 16, 16)])
@pytest.mark.parametrize("batch,contexts", [(1, [8100]), (1, [20000]), (3, [8100, 63, 4095]), (17, [8000]), (32, [8000])])
def test_long_contexts_against_launched_attention(lib_built, device, monkeypatch, hidden, heads, kv, batch, contexts):
    """Hundreds of stages in a link, which go round the ring many times, up to 64 parts a head, units of a second and later round; the steps cross a 64-key stage."""
    L = lib_built
    model = L.Model(device, dtype="bf16", n_layers=2, hidden=hidden, n_heads=heads, n_kv_heads=kv, intermediate=512, vocab=500, eps=1e-5, rope_base=10000.0)
    model.init_random(seed=6, sigma=0.02)
    contexts = contexts if len(contexts) == batch else contexts * batch
    chain, launched = both(L, model, monkeypatch, batch, max(contexts) + 70, contexts, 68, batch)
    # as above; the sums run over more keys, whose weights are the same bf16 values on both sides up to the maximum they are taken against
    assert np.isfinite(chain).all() and rel_err(chain, launched) <= BF16_REL_TOL / 2
    model.close()


@pytest.mark.parametrize("batch,capacity,link", [(16, 1024, True), (17, 128, True), (17, 4096, False), (20, 8192, False), (32, 8192, True), (1, 8192, True)])
def test_launched_where_whole_heads_spread_badly(lib_built, device, batch, capacity, link):
    L = lib_built
    model = L.Model(device, dtype="bf16", n_layers=4, hidden=2048, n_heads=32 if batch == 20 else 16, n_kv_heads=8, intermediate=512, vocab=300, eps=1e-5, rope_base=10000.0)
    model.init_random(seed=6, sigma=0.02)
    sess = L.Session(model, batch, capacity)
    tok = np.zeros(batch, np.int32)
    sess.decode_step(tok)
    before = device.launch_count()
    sess.decode_step(tok)
    assert (device.launch_count() - before == 4) is link           # embedding, one chain, token, position; launched: an attention and a chain per layer
    sess.close(); model.close()


def test_unequal_positions_choose_anew(lib_built, device, monkeypatch):
    """One long sequence among short ones launches its attention, positions close to one another keep it in the chain, back and forth in one session; the same
    results as with the attention launched throughout."""
    L = lib_built
    model = L.Model(device, dtype="bf16", n_layers=4, hidden=2048, n_heads=16, n_kv_heads=4, intermediate=512, vocab=300, eps=1e-5, rope_base=10000.0)
    model.init_random(seed=6, sigma=0.02)
    batch, capacity = 16, 4096
    places = [([4000] + [60] * 15, False), (list(range(3000, 3016)), True), ([100] * 16, True), ([60] * 15 + [4000], False), ([2000] * 16, True)]
    got = {}
    for env in (None, "0"):
        monkeypatch.delenv("LMB200_CHAIN_ATTENTION", raising=False)
        if env:
            monkeypatch.setenv("LMB200_CHAIN_ATTENTION", env)
        sess = L.Session(model, batch, capacity)
        sess.fill_kv_random(4000, 7)
        got[env] = []
        for pos, link in places:
            sess.set_positions(np.array(pos, np.int32))
            tok = O.synth_tokens(8, 1, (batch,), 300).astype(np.int32)
            for _ in range(3):
                before = device.launch_count()
                tok, lg = sess.decode_step(tok, want_logits=True)
                assert (device.launch_count() - before == 4) is (link and env is None), pos[:2]
                got[env].append(lg)
                tok = O.synth_tokens(8, len(got[env]), (batch,), 300).astype(np.int32)
        sess.close()
    assert rel_err(np.stack(got[None]), np.stack(got["0"])) <= BF16_REL_TOL / 2
    model.close()


def test_deep_model_against_oracle(lib_built, device):
    """More links than one launch takes (nine layers: 46), from an empty cache."""
    L = lib_built
    cfg = dict(n_layers=9, hidden=2048, n_heads=16, n_kv_heads=4, intermediate=256, vocab=300, eps=1e-5, rope_base=10000.0)
    model = L.Model(device, dtype="bf16", **cfg)
    model.init_random(seed=3, sigma=0.02)
    w = O.synth_llama_weights(cfg, seed=3)
    batch = 2
    tokens = O.synth_tokens(31, 1000, (batch, 5), cfg["vocab"])
    ref = O.CachedLlama(w, cfg, batch, 16)
    sess = L.Session(model, batch, 16)
    sess.set_capture(True)
    for i in range(5):
        ref_logits, ref_hidden = ref.forward(tokens[:, i:i + 1], return_hidden=True)
        before = device.launch_count()
        _, logits = sess.decode_step(np.ascontiguousarray(tokens[:, i]), want_logits=True)
        assert device.launch_count() - before == 5                 # embedding, two chains, token, position
        for l in range(cfg["n_layers"]):
            assert rel_err(sess.layer_output(l), ref_hidden[l][:, -1, :]) <= BF16_REL_TOL, (i, l)
        assert rel_err(logits, ref_logits[:, -1, :]) <= 2 * BF16_REL_TOL, i
    sess.close(); model.close()
