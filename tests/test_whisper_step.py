"""The bf16 Whisper decoder's step of two launches (head dimension 64, up to 16 sequences) against the oracle, at the edges of its work split: widths whose 64-k units do
not divide among eight warps, one head, key counts around its 16-key blocks and its parts, a second column tile, end-of-text and ragged positions."""
import numpy as np
import pytest

import luminal_oracle as O
import whisper_oracle as W

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def wherever_it_can_be(monkeypatch):
    """Also at the sizes the library launches instead: these tests are about what the kernels compute."""
    monkeypatch.setenv("LMB200_WHISPER_STEP", "1")


def config(heads, ffn, layers=2, vocab=203, positions=40):
    return dict(d_model=64 * heads, heads=heads, enc_layers=1, dec_layers=layers, ffn=ffn, vocab=vocab, n_mels=8, max_positions=positions)


def decoder(L, device, cfg, batch, T, seed):
    w = {n: a for n, a in W.synth_weights(cfg, seed=seed).items() if n.startswith("model.decoder.")}
    rng = np.random.default_rng(seed)
    D = 64
    kv = [tuple(rng.standard_normal((batch, cfg["heads"], T, D)).astype(np.float32) for _ in range(2)) for _ in range(cfg["dec_layers"])]
    model = L.WhisperDecoderModel(device, d_model=cfg["d_model"], heads=cfg["heads"], layers=cfg["dec_layers"], ffn=cfg["ffn"], vocab=cfg["vocab"],
                                  max_positions=cfg["max_positions"], cross_len=T, dtype="bf16")
    for n, a in w.items():
        model.set_weight(n, a)
    sess = L.Session(model, batch, cfg["max_positions"])
    for i, (k, v) in enumerate(kv):
        sess.set_cross_kv(i, k, v)
    return w, kv, model, sess


@pytest.mark.parametrize("heads,ffn,batch,T", [(1, 64, 1, 1), (2, 192, 3, 15), (6, 1536, 2, 130), (8, 2048, 8, 1500), (9, 576, 9, 129), (16, 4096, 16, 257), (16, 64, 1, 1500)])
def test_step_against_oracle(lib_built, device, heads, ffn, batch, T):
    cfg = config(heads, ffn)
    w, kv, model, sess = decoder(lib_built, device, cfg, batch, T, heads + T)
    ref = W.CachedDecoder(w, cfg, batch, kv)
    sess.set_capture(True)
    tok = O.synth_tokens(4, 6, (batch,), cfg["vocab"])
    for step in range(20):                                         # past one block of the self-attention cache
        ref_logits, ref_hidden = ref.step(tok, return_hidden=True)
        before = device.launch_count()
        chosen, logits = sess.decode_step(tok, want_logits=True)
        assert step == 0 or device.launch_count() - before == 2    # (the first step also folds the norms into the weights)
        for l in range(cfg["dec_layers"]):                         # bf16 operands: as the launched step's bound
            got = sess.layer_output(l)
            assert np.linalg.norm(got - ref_hidden[l]) <= 2e-2 * np.linalg.norm(ref_hidden[l]), (step, l)
        assert np.linalg.norm(logits - ref_logits) <= 4e-2 * np.linalg.norm(ref_logits), step
        assert np.array_equal(chosen, logits.argmax(-1))           # the first of equals
        tok = ref_logits.argmax(-1)
    sess.close(); model.close()


def test_decode_n_and_end_of_text(lib_built, device):
    """The device-resident loop: the same tokens as single steps, repeats behind the end-of-text token, and steps without a head (a prompt)."""
    cfg = config(8, 512, vocab=60)
    _, _, model, sess = decoder(lib_built, device, cfg, 5, 70, 1)
    first = O.synth_tokens(4, 6, (5,), cfg["vocab"])
    n = 24
    toks, tok = [], first.astype(np.int32)
    for _ in range(n):
        tok, _ = sess.decode_step(tok, want_logits=True)
        toks.append(tok.copy())
    toks = np.stack(toks)
    sess.reset()
    assert np.array_equal(sess.decode_n(first, n), toks)
    prompt = np.concatenate([first[:, None], toks[:7].T], 1)
    sess.reset()
    logits = sess.prefill(prompt)
    assert np.array_equal(logits.argmax(-1), toks[7]) and sess.position() == 8
    assert np.array_equal(sess.decode_n(toks[7], n - 8), toks[8:])
    sess.close(); model.close()


def test_larger_batches_keep_the_launched_step(lib_built, device):
    cfg = config(2, 128)
    _, _, model, sess = decoder(lib_built, device, cfg, 17, 20, 2)
    before = device.launch_count()
    sess.decode_step(O.synth_tokens(4, 6, (17,), cfg["vocab"]))
    assert device.launch_count() - before > 8
    sess.close(); model.close()


@pytest.mark.parametrize("heads,batch,two_launches", [(12, 16, True), (13, 9, False), (16, 8, True), (16, 16, False)])
def test_wide_decoders_at_the_rule(lib_built, device, monkeypatch, heads, batch, two_launches):
    monkeypatch.delenv("LMB200_WHISPER_STEP")
    cfg = config(heads, 128)
    w, kv, model, sess = decoder(lib_built, device, cfg, batch, 20, heads)
    tok = O.synth_tokens(4, 6, (batch,), cfg["vocab"])
    ref = W.CachedDecoder(w, cfg, batch, kv).step(tok)
    chosen, logits = sess.decode_step(tok, want_logits=True)
    assert np.linalg.norm(logits - ref) <= 4e-2 * np.linalg.norm(ref)
    before = device.launch_count()
    sess.decode_step(tok)
    assert (device.launch_count() - before == 2) is two_launches
    sess.close(); model.close()
