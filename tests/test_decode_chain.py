"""The chained decode GEMVs (one launch for o_proj, gate/up, down and the next q/k/v or the head) against the oracle, at the
sizes where the split can go wrong."""
import numpy as np
import pytest

import luminal_oracle as O
from test_decode_parity import BF16_REL_TOL, make_model, rel_err

pytestmark = pytest.mark.gpu

BASE = dict(n_layers=3, eps=1e-5, rope_base=10000.0)
SIZES = {
    # two units of k: two of a cluster's four CTAs have nothing to multiply
    "short_k": dict(hidden=256, n_heads=4, n_kv_heads=2, intermediate=200, vocab=300),
    # ragged last row group and k unit everywhere, k units that four does not divide
    "ragged": dict(hidden=640, n_heads=5, n_kv_heads=1, intermediate=1000, vocab=1111),
    # more row groups than clusters at K 512: gate/up and the head leave the chain and are launched by themselves
    "diverted": dict(hidden=512, n_heads=4, n_kv_heads=4, intermediate=5000, vocab=8200),
}


@pytest.mark.parametrize("size,batch", [("short_k", 1), ("short_k", 17), ("ragged", 16), ("ragged", 32), ("diverted", 3), ("diverted", 31)])
def test_chained_step_matches_oracle(lib_built, device, monkeypatch, size, batch):
    monkeypatch.setenv("LMB200_GEMV_CHAIN", "1")            # by default widths of 4 to 15 row groups are not chained
    L = lib_built
    cfg = dict(BASE, **SIZES[size])
    w = O.synth_llama_weights(cfg, seed=31)
    tokens = O.synth_tokens(31, 1000, (batch, 4), cfg["vocab"])
    ref = O.CachedLlama(w, cfg, batch, 16)
    model = make_model(L, device, cfg, w, "bf16")
    sess = L.Session(model, batch, 16)
    sess.set_capture(True)
    for i in range(4):                       # the counters have to be empty again for every launch of every step
        ref_logits, ref_hidden = ref.forward(tokens[:, i:i + 1], return_hidden=True)
        _, logits = sess.decode_step(np.ascontiguousarray(tokens[:, i]), want_logits=True)
        for l in range(cfg["n_layers"]):
            assert rel_err(sess.layer_output(l), ref_hidden[l][:, -1, :]) <= BF16_REL_TOL, (i, l)
        assert rel_err(logits, ref_logits[:, -1, :]) <= 2 * BF16_REL_TOL, i
    sess.close(); model.close()


def launches_per_step(L, device, model, batch):
    sess = L.Session(model, batch, 16)
    t = np.zeros(batch, np.int32)
    sess.decode_n(t, 1)
    before = device.launch_count()
    sess.decode_n(t, 1)
    n = device.launch_count() - before
    sess.close()
    return n


@pytest.mark.parametrize("batch", [2, 17])
def test_rounds_match_oracle(lib_built, device, monkeypatch, batch):
    """GEMVs of several tiles per cluster inside the chain: gate/up 74 row groups, the head 70, so with 33 clusters three rounds whose last one is partly
    empty; 14 units of k, which four CTAs share unevenly.  The launch counts show that nothing left the chain."""
    L = lib_built
    cfg = dict(BASE, n_layers=2, hidden=1792, n_heads=14, n_kv_heads=7, intermediate=4736, vocab=8900)
    rng = np.random.default_rng(batch)
    w = O.synth_llama_weights(dict(cfg, hidden=14, n_heads=14, n_kv_heads=7, intermediate=8, vocab=8), seed=1)
    for name in w:
        part = name.split(".")[-2]
        rows = dict(q_proj=1792, k_proj=896, v_proj=896, o_proj=1792, gate_proj=4736, up_proj=4736, down_proj=1792, embed_tokens=8900, lm_head=8900).get(part)
        w[name] = 0.02 * rng.standard_normal((rows, 4736 if part == "down_proj" else 1792), dtype=np.float32) if rows else np.ones(1792, np.float32)
    tokens = rng.integers(0, 8900, (batch, 3)).astype(np.int32)
    ref = O.CachedLlama(w, cfg, batch, 16)
    model = make_model(L, device, cfg, w, "bf16")
    count = {}
    for chain in "01":
        monkeypatch.setenv("LMB200_GEMV_CHAIN", chain)
        count[chain] = launches_per_step(L, device, model, batch)
    assert count["0"] - count["1"] == 3 * cfg["n_layers"]        # o_proj, gate/up, down_proj and the next q/k/v or the head are one launch
    sess = L.Session(model, batch, 16)
    sess.set_capture(True)
    for i in range(3):
        ref_logits, ref_hidden = ref.forward(tokens[:, i:i + 1], return_hidden=True)
        _, logits = sess.decode_step(np.ascontiguousarray(tokens[:, i]), want_logits=True)
        for l in range(2):
            assert rel_err(sess.layer_output(l), ref_hidden[l][:, -1, :]) <= BF16_REL_TOL, (i, l)
        assert rel_err(logits, ref_logits[:, -1, :]) <= 2 * BF16_REL_TOL, i
    sess.close(); model.close()


@pytest.mark.parametrize("hidden,heads,chained", [(384, 6, True), (512, 8, False), (1920, 15, False), (2048, 16, True)])
def test_widths_that_are_chained(lib_built, device, monkeypatch, hidden, heads, chained):
    """The rule on the residual width, and the same tokens either way."""
    L = lib_built
    model = L.Model(device, dtype="bf16", **dict(BASE, n_layers=2, hidden=hidden, n_heads=heads, n_kv_heads=heads, intermediate=1536, vocab=500))
    model.init_random(seed=5, sigma=0.02)
    count, logits = {}, {}
    for chain in ("0", "1", None):
        monkeypatch.delenv("LMB200_GEMV_CHAIN", raising=False)
        if chain:
            monkeypatch.setenv("LMB200_GEMV_CHAIN", chain)
        count[chain] = launches_per_step(L, device, model, 3)
        sess = L.Session(model, 3, 16)
        logits[chain] = [sess.decode_step(np.array(t, np.int32), want_logits=True)[1] for t in ((1, 2, 3), (77, 8, 9))][-1]
        sess.close()
    assert count["1"] < count["0"] and count[None] == count["1" if chained else "0"]
    assert np.array_equal(logits[None], logits["1" if chained else "0"])
    assert rel_err(logits["1"], logits["0"]) <= 2 * BF16_REL_TOL
    model.close()
