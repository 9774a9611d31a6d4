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
    # more row groups than clusters: gate/up in three rounds, the head in two, the last one partly empty
    "rounds": dict(hidden=512, n_heads=4, n_kv_heads=4, intermediate=5000, vocab=8200),
}


@pytest.mark.parametrize("size,batch", [("short_k", 1), ("short_k", 17), ("ragged", 16), ("ragged", 32), ("rounds", 3), ("rounds", 31)])
def test_chained_step_matches_oracle(lib_built, device, size, batch):
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
