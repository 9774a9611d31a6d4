"""The work that this library's users have it do, as cases that can be timed: calls of the public Python layer (and, for the
flash-attention operation on bf16 tensors, of the C entry it has no wrapper for) at the model sizes of bench.py and of the tests.

A case is a dict of plain values.  `kind` says which path it takes:
  decode   one or more cached steps of a Llama / Phi-3 session behind a given context, tokens forced as a replayed trace's are
  prompt   a whole prompt (or a batch of unequal ones) on a fresh session, the logits of every sequence's last position
  layered  a request on a decoder described layer by layer: reset, prompt, then forced steps
  whisper  mel -> encoder -> cross K/V -> greedy steps
  flash    the FlashAttentionOp alone
  graph    the reference's own route: a traced NN.Llama graph through compile() and called with new tokens
"""
import ctypes
import math

import numpy as np
import torch

import luminal_jl_b200 as L
from luminal_jl_b200 import _lib

# decoder sizes (bench.py, the tests' configurations)
LLAMA = {
    "small_llama": dict(n_layers=4, hidden=256, n_heads=8, n_kv_heads=8, intermediate=688, vocab=1024, eps=1e-5, rope_base=10000.0),
    "mid_gqa": dict(n_layers=2, hidden=1024, n_heads=8, n_kv_heads=2, intermediate=2816, vocab=4096, eps=1e-5, rope_base=500000.0),
    "phi3_mini": dict(n_layers=32, hidden=3072, n_heads=32, n_kv_heads=8, intermediate=8192, vocab=32064, eps=1e-5, rope_base=10000.0),
    "llama3_8b": dict(n_layers=32, hidden=4096, n_heads=32, n_kv_heads=8, intermediate=14336, vocab=128256, eps=1e-5, rope_base=500000.0),
}
WHISPER_BASE = dict(d_model=512, heads=8, enc_layers=6, dec_layers=6, ffn=2048, vocab=51865, n_mels=80, max_positions=448)
SIGMA = 0.02
# Gains of the norms in front of attention and feed-forward.  Trained decoders' are well below one; here these keep the embedding, attention and
# feed-forward contributions of one size, so that all of them show in the logits and 32 random layers do not amplify rounding.
ATTENTION_GAIN, FEED_FORWARD_GAIN = 0.25, 0.05


def gibutar(width, heads, ff, kv_rank, q_rank, layers=8, vocab=32064):
    """One latent-attention layer to three retention layers, the second latent layer of a pair reading the first one's cache."""
    dim, out = width // heads, []
    for i in range(layers):
        if i % 4 == 0:
            mx = dict(heads=heads, dim=dim, rot_dim=64, vdim=dim, kv_rank=kv_rank, q_rank=q_rank, scale=(dim + 64) ** -0.5, rot=dict(base=500000.0, dims=64))
            if i % 8 == 4:
                mx["kv_from"] = i - 4
            out.append(dict(type="latent_attention", mixer=mx, mlp=dict(kind="dense", ff=ff)))
        else:
            mx = dict(heads=heads, dim=dim, vdim=dim, rot=dict(base=10000.0, dims=dim), decay=[1.0 - 2.0 ** -(5 + 4 * h / heads) for h in range(heads)])
            out.append(dict(type="retention", mixer=mx, mlp=dict(kind="dense", ff=ff)))
    return dict(architecture="Gibutar", width=width, vocab=vocab, norm=dict(eps=1e-5), logit_softcap=30.0, layers=out)


def kevatar(width, heads, kv_heads, ff, side, window, layers=8, vocab=32064):
    """Of eight layers two windowed attention (the second reading the first one's cache), two channel delta and four lightning."""
    dim, out = width // heads, []
    for i in range(layers):
        if i % 4 == 0:
            mx, kind = dict(heads=heads, kv_heads=kv_heads, dim=dim, vdim=dim, scale=dim ** -0.5, softcap=30.0, mask=dict(size=window),
                            rot=dict(base=500000.0, dims=dim // 2, scaling=dict(factor=4.0, original=8192, fast=32.0, slow=1.0))), "attention"
            if i % 8 == 4:
                mx["kv_from"] = i - 4
        elif i % 4 == 2:
            mx, kind = dict(heads=heads, kv_heads=heads // 2, dim=dim, vdim=dim, conv=4), "channel_delta"
        else:
            mx, kind = dict(heads=heads, dim=dim, vdim=dim, decay=[1.0 - 2.0 ** -(5 + 4 * h / heads) for h in range(heads)]), "lightning"
        out.append(dict(type=kind, mixer=mx, mlp=dict(kind="dense", ff=ff)))
    return dict(architecture="Kevatar", width=width, vocab=vocab, norm=dict(eps=1e-5), embedding=dict(scale=1.0), token_side=dict(dim=side), layers=out)


LAYERED = {
    "gibutar_w2048": gibutar(2048, 16, 8192, 512, 768),
    "gibutar_w4096": gibutar(4096, 32, 14336, 512, 1536),
    "kevatar_w2048": kevatar(2048, 16, 4, 8192, 128, 1024),
    "kevatar_w4096": kevatar(4096, 32, 8, 14336, 256, 1024),
}


def listed():
    return [
        # the smallest call: one float32 step of the small Llama, a chain of launches
        dict(name="small_step_f32", kind="decode", model="small_llama", dtype="f32", batch=1, context=100, steps=1),
        # the reference's own route: the traced graph compiled, a 32-token prompt recomputed as its generation loop does
        dict(name="small_graph_f32", kind="graph", model="small_llama", batch=1, tokens=32),
        # one user at a time: a step streams the weights
        dict(name="llama3_8b_decode_b1", kind="decode", model="llama3_8b", dtype="bf16", batch=1, context=1031, steps=8),
        # a serving batch at a middling context
        dict(name="phi3_decode_b16", kind="decode", model="phi3_mini", dtype="bf16", batch=16, context=2052, steps=8),
        # the flagship step: full batch, full context, weights and cache each streamed once
        dict(name="llama3_8b_decode_b32", kind="decode", model="llama3_8b", dtype="bf16", batch=32, context=8184, steps=4),
        # requests of unequal length arriving together
        dict(name="llama3_8b_prompt_ragged", kind="prompt", model="llama3_8b", dtype="bf16", batch=5, tokens=777, ragged=True),
        # the long prompt batch: tensor-core work
        dict(name="phi3_prompt_16x2048", kind="prompt", model="phi3_mini", dtype="bf16", batch=16, tokens=2048, ragged=False),
        # FlashAttentionOp at the size the benchmark names, and in float32 on a ragged causal sequence
        dict(name="flash_bf16", kind="flash", dtype="bf16", batch=4, heads=32, seq=4096, dim=128, causal=False),
        dict(name="flash_f32_causal", kind="flash", dtype="f32", batch=2, heads=16, seq=1531, dim=64, causal=True),
        # a batch of thirty-second clips transcribed
        dict(name="whisper_base_b8", kind="whisper", batch=8, frames=3000, steps=32),
        # layered decoders: a prompt-heavy and a generation-heavy request
        dict(name="gibutar_prompt", kind="layered", model="gibutar_w2048", batch=4, tokens=2048, steps=2),
        dict(name="kevatar_turns", kind="layered", model="kevatar_w2048", batch=16, tokens=131, steps=24),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "layered", "layered", "whisper", "flash", "flash", "graph"])
    if kind == "decode":
        model = rng.choice(["small_llama", "mid_gqa", "phi3_mini", "llama3_8b"])
        dtype = "f32" if model == "small_llama" else "bf16"
        return dict(kind=kind, model=model, dtype=dtype, batch=1 if model == "small_llama" else _log_int(rng, 1, 32),
                    context=_log_int(rng, 16, 120 if model == "small_llama" else 8180), steps=rng.randint(1, 8))
    if kind == "prompt":
        model = rng.choice(["mid_gqa", "phi3_mini", "llama3_8b"])
        batch = _log_int(rng, 1, 16)
        return dict(kind=kind, model=model, dtype="bf16", batch=batch, tokens=_log_int(rng, 9, min(4096, 8192 // batch)), ragged=rng.random() < 0.5)
    if kind == "layered":
        batch = _log_int(rng, 1, 32)
        return dict(kind=kind, model=rng.choice(sorted(LAYERED)), batch=batch, tokens=_log_int(rng, 3, min(2048, 8192 // batch)), steps=_log_int(rng, 1, 32))
    if kind == "whisper":
        return dict(kind=kind, batch=rng.randint(1, 8), frames=rng.randint(150, 1500) * 2, steps=_log_int(rng, 4, 96))
    if kind == "flash":
        dtype = rng.choice(["bf16", "f32"])
        batch, heads = rng.randint(1, 4), rng.randint(1, 32)
        return dict(kind=kind, dtype=dtype, batch=batch, heads=heads, seq=_log_int(rng, 32, 4096), dim=rng.choice([64, 96, 128]), causal=rng.random() < 0.5)
    return dict(kind=kind, model=rng.choice(["small_llama", "mid_gqa"]), batch=rng.randint(1, 4), tokens=_log_int(rng, 2, 128))


# ---------------------------------------------------------------------------------------------------------------------
# inputs.  Large models fill their weights and caches on the device from the library's documented generator (twelve 16-bit
# lanes of three splitmix64 outputs, centred, times sigma / 131072); the same numbers are formed here where they are needed.
# ---------------------------------------------------------------------------------------------------------------------
_M = (1 << 64) - 1


def _signed(x):
    x &= _M
    return x - (1 << 64) if x >> 63 else x


def _mix_int(x):
    z = (x + 0x9E3779B97F4A7C15) & _M
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & _M
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & _M
    return z ^ (z >> 31)


def _shift(z, n):
    return (z >> n) & ((1 << (64 - n)) - 1)


def _lanes(index, key):
    total = torch.zeros_like(index)
    for r in range(3):
        z = ((index * 3 + r) ^ key) + _signed(0x9E3779B97F4A7C15)
        z = (z ^ _shift(z, 30)) * _signed(0xBF58476D1CE4E5B9)
        z = (z ^ _shift(z, 27)) * _signed(0x94D049BB133111EB)
        z = z ^ _shift(z, 31)
        for lane in range(4):
            total += (z >> (16 * lane)) & 0xFFFF
    return total


def generated(seed, tensor, shape, sigma=SIGMA, offset=0.0, index=None):
    """float32 values of the generator for a row-major tensor (or at the given linear indices)."""
    key = _signed(_mix_int((seed * 0xD1342543DE82EF95 + tensor) & _M))
    n = math.prod(shape)
    out = torch.empty(n, device="cuda")
    for at in range(0, n, 1 << 26):
        m = min(1 << 26, n - at)
        i = torch.arange(at, at + m, device="cuda") if index is None else index.reshape(-1)[at:at + m]
        v = (2 * _lanes(i, key) - 12 * 65535).float() * torch.tensor(sigma, dtype=torch.float32).div(131072.0).item()
        out[at:at + m] = v + offset if offset else v
    return out.view(shape)


def tokens_of(case, seed, count, vocab):
    g = np.random.default_rng([seed, 77])
    return g.integers(0, vocab, (case["batch"], count)).astype(np.int32)


def lengths_of(case, seed):
    g = np.random.default_rng([seed, 78])
    n = g.integers(max(1, case["tokens"] // 8), case["tokens"] + 1, case["batch"])
    n[g.integers(0, case["batch"])] = case["tokens"]
    return n


def _capacity(case):
    n = case["context"] + case["steps"]
    return -(-n // 16) * 16


SLOTS = dict(input_layernorm=0, q_proj=1, k_proj=2, v_proj=3, o_proj=4, post_attention_layernorm=5, gate_proj=6, up_proj=7, down_proj=8)


def llama_tensor(cfg, seed, name):
    """One of a Llama's tensors by its registry name."""
    h, f, kv, v = cfg["hidden"], cfg["intermediate"], cfg["hidden"] // cfg["n_heads"] * cfg["n_kv_heads"], cfg["vocab"]
    part = name.split(".")[-2]
    if name.startswith("model.layers."):
        shape = dict(q_proj=(h, h), k_proj=(kv, h), v_proj=(kv, h), o_proj=(h, h), gate_proj=(f, h), up_proj=(f, h), down_proj=(h, f)).get(part, (h,))
        a = generated(seed, 16 * int(name.split(".")[2]) + SLOTS[part], shape, offset=1.0 if len(shape) == 1 else 0.0)
        return a * dict(input_layernorm=ATTENTION_GAIN, post_attention_layernorm=FEED_FORWARD_GAIN).get(part, 1.0)
    tensor, shape = dict(embed_tokens=(0xFFFF0, (v, h)), norm=(0xFFFF1, (h,)), lm_head=(0xFFFF2, (v, h)))[part]
    return generated(seed, tensor, shape, offset=1.0 if len(shape) == 1 else 0.0)


def whisper_weights(seed):
    """Random weights with an embedding as large as a trained one is beside the layers' contributions, so that no greedy choice is a near tie."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = {}
    for name, shape in sorted(L.whisper.registry_shapes(**WHISPER_BASE).items()):
        a = torch.randn(shape, device="cuda", generator=g) * (1.0 if name.endswith("embed_tokens.weight") else SIGMA)
        w[name] = a + 1.0 if name.endswith("layer_norm.weight") else a
    return w


def whisper_mel(case, seed):
    return np.random.default_rng([seed, 79]).standard_normal((case["batch"], WHISPER_BASE["n_mels"], case["frames"]), dtype=np.float32)


def flash_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (case["batch"], case["heads"], case["seq"], case["dim"])
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    return [torch.randn(shape, device="cuda", generator=g).to(dtype) for _ in range(3)]


class State:
    """What a user's program holds between calls; handles are given back when it goes."""

    def __init__(self, case):
        self.case, self.closing = case, []

    def hold(self, thing):
        self.closing.append(thing)
        return thing

    def __del__(self):
        for thing in reversed(self.closing):
            thing.close()
        self.closing = []


def prepare(case, seed):
    dev = L.get_device()
    s = State(case)
    kind = case["kind"]
    if kind in ("decode", "prompt"):
        cfg = LLAMA[case["model"]]
        model = s.hold(L.Model(dev, dtype=case["dtype"], **cfg))
        model.init_random(seed, SIGMA)
        for n in range(cfg["n_layers"]):
            for part in ("input_layernorm", "post_attention_layernorm"):
                name = f"model.layers.{n}.{part}.weight"
                model.set_weight(name, llama_tensor(cfg, seed, name).cpu().numpy())
        s.session = s.hold(L.Session(model, case["batch"], _capacity(case) if kind == "decode" else case["tokens"] + 1))
        if kind == "decode":
            s.session.fill_kv_random(case["context"], seed)
            s.tokens = tokens_of(case, seed, case["steps"], cfg["vocab"])
        else:
            s.tokens = tokens_of(case, seed, case["tokens"], cfg["vocab"])
            if case["ragged"]:
                s.prompts = [t[:n].copy() for t, n in zip(s.tokens, lengths_of(case, seed))]
    elif kind == "layered":
        cfg = LAYERED[case["model"]]
        shapes = {f"l{i}.mix.{t}": (x["mixer"]["dim"], cfg["width"]) for i, x in enumerate(cfg["layers"]) if x["type"] == "channel_delta" for t in ("a1", "g1")}
        model = s.hold(L.models.build_model(dev, cfg, "bf16", shapes))
        model.init_random(seed, SIGMA)
        s.session = s.hold(L.Session(model, case["batch"], case["tokens"] + case["steps"]))
        every = tokens_of(case, seed, case["tokens"] + case["steps"], cfg["vocab"])
        s.prompt, s.forced = np.ascontiguousarray(every[:, :case["tokens"]]), np.ascontiguousarray(every[:, case["tokens"]:])
    elif kind == "whisper":
        cfg = WHISPER_BASE
        w = {k: v.cpu().numpy() for k, v in whisper_weights(seed).items()}
        s.encoder = s.hold(L.whisper.FusedEncoder(dev, d_model=cfg["d_model"], heads=cfg["heads"], enc_layers=cfg["enc_layers"],
                                                  dec_layers=cfg["dec_layers"], ffn=cfg["ffn"], n_mels=cfg["n_mels"]))
        s.encoder.set_weights(w)
        model = s.hold(L.WhisperDecoderModel(dev, d_model=cfg["d_model"], heads=cfg["heads"], layers=cfg["dec_layers"], ffn=cfg["ffn"], vocab=cfg["vocab"],
                                             max_positions=cfg["max_positions"], cross_len=(case["frames"] - 1) // 2 + 1, dtype="bf16"))
        for name, a in w.items():
            if name.startswith("model.decoder."):
                model.set_weight(name, a)
        s.session = s.hold(L.Session(model, case["batch"], cfg["max_positions"]))
        s.mel, s.first = whisper_mel(case, seed), tokens_of(case, seed, 1, cfg["vocab"])[:, 0].copy()
    elif kind == "flash":
        s.q, s.k, s.v = flash_inputs(case, seed)
        s.out = torch.empty_like(s.q)
        s.device = dev
    else:
        cfg = LLAMA[case["model"]]
        g, reg = L.Graph(), {}
        net = L.nn.Llama(g, reg, vocab_size=cfg["vocab"], hidden=cfg["hidden"], n_layers=cfg["n_layers"], n_heads=cfg["n_heads"],
                         n_kv_heads=cfg["n_kv_heads"], intermediate=cfg["intermediate"])
        ids = L.tensor(g, [case["batch"], case["tokens"]])
        s.out = net(ids, 0).id
        L.weights.load_weights(g, reg, {name: llama_tensor(cfg, seed, name).cpu().numpy() for name in reg})
        s.ids, s.call = ids.id, L.compile(g, dev)
        s.tokens = tokens_of(case, seed, case["tokens"], cfg["vocab"]).astype(np.float32)
    return s


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "decode":
        s.session.set_position(case["context"])
        for i in range(case["steps"] - 1):
            s.session.decode_step(s.tokens[:, i])
        chosen, logits = s.session.decode_step(s.tokens[:, -1], want_logits=True)
        return dict(logits=logits, chosen_logit=np.take_along_axis(logits, chosen[:, None].astype(np.int64), 1))
    if kind == "prompt":
        s.session.reset()
        return dict(logits=s.session.prefill_ragged(s.prompts) if case["ragged"] else s.session.prefill(s.tokens))
    if kind == "layered":
        s.session.reset()
        first = s.session.prefill(s.prompt)
        for i in range(case["steps"] - 1):
            s.session.decode_step(s.forced[:, i])
        chosen, logits = s.session.decode_step(s.forced[:, -1], want_logits=True)
        return dict(prompt_logits=first, logits=logits, chosen_logit=np.take_along_axis(logits, chosen[:, None].astype(np.int64), 1))
    if kind == "whisper":
        s.encoder.run(s.mel, want_output=False)
        s.encoder.cross_kv_into(s.session)
        s.session.reset()
        tokens = s.session.decode_n(s.first, case["steps"])
        return dict(tokens=tokens, logits=s.session.decode_step(tokens[-1], want_logits=True)[1])
    if kind == "flash":
        p = [ctypes.c_void_p(t.data_ptr()) for t in (s.out, s.q, s.k, s.v)]
        _lib.call("lmb200_flash_attention", s.device.handle, *p, _lib.BF16 if case["dtype"] == "bf16" else _lib.F32, case["batch"], case["heads"],
                  case["seq"], case["dim"], 1.0 / math.sqrt(case["dim"]), int(case["causal"]))
        return s.out
    return s.call({s.ids: s.tokens})[s.out].numpy()


# ---------------------------------------------------------------------------------------------------------------------
# the work no implementation can leave out, and how far two correct ones may differ
# ---------------------------------------------------------------------------------------------------------------------
def _llama_params(cfg):
    h, d = cfg["hidden"], cfg["hidden"] // cfg["n_heads"]
    layer = 2 * h * h + 2 * h * cfg["n_kv_heads"] * d + 3 * h * cfg["intermediate"]
    return cfg["n_layers"] * layer, cfg["vocab"] * h


def _layered_params(cfg):
    """(weights of the layers, head weights, bytes a sequence's recurrent states take, cache bytes a token adds)"""
    total, state, cache, W = 0, 0, 0, cfg["width"]
    for x in cfg["layers"]:
        mx = x["mixer"]
        H, d, v = mx["heads"], mx["dim"], mx["vdim"]
        own = mx.get("kv_from") is None
        total += (2 if cfg["architecture"] == "Gibutar" else 3) * W * x["mlp"]["ff"] + W * H * v
        if x["type"] == "latent_attention":
            total += W * (mx["q_rank"] + H) + mx["q_rank"] * H * (d + mx["rot_dim"]) + mx["kv_rank"] * H * (d + v) + own * W * (mx["kv_rank"] + mx["rot_dim"])
            cache += own * 2 * (mx["kv_rank"] + mx["rot_dim"])
        elif x["type"] == "attention":
            total += W * H * d + own * W * mx["kv_heads"] * (d + v)
            cache += own * 2 * mx["kv_heads"] * (d + v)
        elif x["type"] == "channel_delta":
            total += W * (2 * mx["kv_heads"] * d + H * v + 2 * d + H) + d * H * (d + v)
            state += 4 * H * d * v
        else:
            total += 2 * W * H * (d + v)
            state += 4 * H * d * v
        total += 2 * W * (cfg.get("token_side") or {"dim": 0})["dim"]
    return total, cfg["vocab"] * W, state, cache


def work(case):
    kind, B = case["kind"], case["batch"]
    if kind in ("decode", "prompt"):
        cfg = LLAMA[case["model"]]
        body, head = _llama_params(cfg)
        size, kv = (4 if case["dtype"] == "f32" else 2), 2 * cfg["n_layers"] * cfg["n_kv_heads"] * (cfg["hidden"] // cfg["n_heads"])
        if kind == "decode":
            n, T = case["steps"], case["context"] + (case["steps"] + 1) / 2
            return dict(bytes=n * ((body + head) * size + B * T * kv * size) + 4 * B * cfg["vocab"],
                        flops=n * B * (2 * (body + head) + 4 * cfg["n_layers"] * cfg["hidden"] * T))
        T = case["tokens"] * (9 / 16 if case["ragged"] else 1.0)           # unequal prompts spread from an eighth to the whole
        return dict(bytes=(body + head) * size + B * T * kv * size + 4 * B * cfg["vocab"],
                    flops=B * (2 * (body * T + head) + 2 * cfg["n_layers"] * cfg["hidden"] * T * T))
    if kind == "layered":
        cfg = LAYERED[case["model"]]
        body, head, state, cache = _layered_params(cfg)
        n, T = case["steps"], case["tokens"]
        attn = 0
        for x in cfg["layers"]:
            mx = x["mixer"]
            H, d, v = mx["heads"], mx["dim"], mx["vdim"]
            w = min(T, (mx.get("mask") or {"size": T})["size"])
            if x["type"] in ("latent_attention", "attention"):
                attn += 2 * H * (d + mx.get("rot_dim", 0) + v) * w * (1 - w / (2 * T)) * T
            else:
                attn += 4 * H * d * v * T
        return dict(bytes=2 * (body + head) * (n + 1) + B * (n * (2 * state + cache * (T + n / 2)) + cache * T + state) + 8 * B * cfg["vocab"],
                    flops=B * (2 * body * (T + n) + 2 * head * (n + 1) + attn))
    if kind == "whisper":
        c = WHISPER_BASE
        d, T, n = c["d_model"], (case["frames"] - 1) // 2 + 1, case["steps"] + 1
        enc, dec, head = c["enc_layers"] * (4 * d * d + 2 * d * c["ffn"]), c["dec_layers"] * (6 * d * d + 2 * d * c["ffn"]), c["vocab"] * d
        cross = c["dec_layers"] * 2 * B * T * d
        return dict(bytes=4 * B * c["n_mels"] * case["frames"] + 2 * (enc + 2 * cross) + n * 2 * (dec + head + cross) + 4 * B * c["vocab"],
                    flops=B * T * (2 * enc + 4 * c["enc_layers"] * T * d + 6 * d * (2 * c["n_mels"] + d)) + 2 * cross * d + n * (2 * B * (dec + head) + 2 * cross))
    if kind == "flash":
        n = B * case["heads"] * case["seq"] * case["dim"]
        pairs = case["seq"] * (case["seq"] + 1) / 2 if case["causal"] else case["seq"] ** 2
        return dict(bytes=4 * n * (2 if case["dtype"] == "bf16" else 4), flops=4 * B * case["heads"] * case["dim"] * pairs)
    cfg = LLAMA[case["model"]]
    body, head = _llama_params(cfg)
    T = case["tokens"]
    return dict(bytes=4 * (body + head + B * T * cfg["vocab"]), flops=B * (2 * (body + head) * T + 4 * cfg["n_layers"] * cfg["hidden"] * T * T))


def tolerance(case):
    # float32 paths are 2e-7 to 2e-6 from exact(), the float32 flash kernel 6e-6, the bf16 one 2.3e-3
    if case["kind"] == "graph" or (case["kind"] == "decode" and case["dtype"] == "f32"):
        return {"rel": 1e-5}
    if case["kind"] == "flash":
        return {"rel": 1e-2} if case["dtype"] == "bf16" else {"rel": 3e-5}
    return {"rel": 3e-2 if case["kind"] == "layered" else 1.2e-2}      # measured against exact(): 0.006 to 0.010, and 0.002 to 0.004


# ---------------------------------------------------------------------------------------------------------------------
# the same outputs in 64 bits.  Matrices are rounded as the model holds them; everything after that is plain torch.
# ---------------------------------------------------------------------------------------------------------------------
def _held(a, dtype):
    return (a.bfloat16() if dtype == "bf16" and a.dim() > 1 else a).double()


def _rms(x, eps, w=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _rotate(x, pos, freq, factor=1.0, interleaved=False):
    """Rotates the first 2 * len(freq) features of x [..., T, D]; pos [T]."""
    n = len(freq)
    a = pos.double()[:, None] * freq
    c, s = factor * a.cos(), factor * a.sin()
    y = x.clone()
    u, v = (x[..., 0:2 * n:2], x[..., 1:2 * n:2]) if interleaved else (x[..., :n], x[..., n:2 * n])
    if interleaved:
        y[..., 0:2 * n:2], y[..., 1:2 * n:2] = u * c - v * s, v * c + u * s
    else:
        y[..., :n], y[..., n:2 * n] = u * c - v * s, v * c + u * s
    return y


def _freq(dims, base):
    return float(base) ** (-torch.arange(0, dims, 2, device="cuda", dtype=torch.float64) / dims)


def _ids(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda", dtype=torch.int64)


def _llama64(cfg, seed, dtype, ids, past=0, capacity=0, last=None, rope_base=None):
    """Logits of ids [B, S] behind `past` cached positions: at each sequence's place last[b], or everywhere."""
    B, S = ids.shape
    H, KV, D = cfg["n_heads"], cfg["n_kv_heads"], cfg["hidden"] // cfg["n_heads"]
    get = lambda name: _held(llama_tensor(cfg, seed, name), dtype)  # noqa: E731
    freq, pos = _freq(D, rope_base or cfg["rope_base"]), torch.arange(past, past + S, device="cuda")
    x = get("model.embed_tokens.weight")[ids]
    later = torch.arange(past + S, device="cuda")[None, :] > pos[:, None]

    def cached(layer, which):
        """the cache of `past` keys or values as fill_kv_random leaves it, one sequence at a time"""
        for b in range(B):
            i = (torch.arange(KV, device="cuda")[:, None, None] + b * KV) * capacity + torch.arange(past, device="cuda")[None, :, None]
            i = i * D + torch.arange(D, device="cuda")
            yield _held(generated(seed, 0x100000 + 2 * layer + which, (KV, past, D), 1.0, index=i), dtype)

    for n in range(cfg["n_layers"]):
        p = f"model.layers.{n}."
        h = _rms(x, cfg["eps"], get(p + "input_layernorm.weight"))
        q, k, v = ((h @ get(p + f"self_attn.{t}_proj.weight").T).view(B, S, D, heads).permute(0, 3, 1, 2) for t, heads in (("q", H), ("k", KV), ("v", KV)))
        q, k = _rotate(q, pos, freq), _rotate(k, pos, freq)
        o = torch.empty_like(q)
        old = zip(cached(n, 0), cached(n, 1)) if past else ((k[b, :, :0], v[b, :, :0]) for b in range(B))
        for b, (ko, vo) in enumerate(old):
            keys, values = torch.cat([ko, k[b]], 1), torch.cat([vo, v[b]], 1)
            for g in range(KV):                                    # query head h reads key head h mod KV
                s = (q[b, g::KV] @ keys[g].T) / math.sqrt(D)
                o[b, g::KV] = s.masked_fill_(later, -math.inf).softmax(-1) @ values[g]
        x = x + o.permute(0, 2, 3, 1).reshape(B, S, D * H) @ get(p + "self_attn.o_proj.weight").T
        h = _rms(x, cfg["eps"], get(p + "post_attention_layernorm.weight"))
        gate, up, down = (get(p + f"mlp.{t}_proj.weight") for t in ("gate", "up", "down"))
        for b in range(B):
            x[b] += (torch.nn.functional.silu(h[b] @ gate.T) * (h[b] @ up.T)) @ down.T
    if last is not None:
        x = x[torch.arange(B, device="cuda"), torch.as_tensor(last, device="cuda")]
    return _rms(x, cfg["eps"], get("model.norm.weight")) @ get("lm_head.weight").T


def _layered_names(cfg):
    """Tensor names and shapes in the order the generator numbers them."""
    W, V, post = cfg["width"], cfg["vocab"], cfg["architecture"] == "Kevatar"
    side = (cfg.get("token_side") or {"dim": 0})["dim"]
    out = [("embed", (V, W)), ("final.norm", (W,))]
    out += [("side.embed", (V, side * len(cfg["layers"])))] if post else [("head", (V, W))]
    for i, x in enumerate(cfg["layers"]):
        mx, p = x["mixer"], f"l{i}."
        H, d, v = mx["heads"], mx["dim"], mx["vdim"]
        G, own = mx.get("kv_heads", H), mx.get("kv_from") is None
        out.append((p + "norm1", (W,)))
        if x["type"] == "latent_attention":
            mix = [("dq", (mx["q_rank"], W)), ("dq.norm", (mx["q_rank"],)), ("uq", (H * (d + mx["rot_dim"]), mx["q_rank"])), ("uk", (H * d, mx["kv_rank"])),
                   ("uv", (H * v, mx["kv_rank"])), ("g", (H, W)), ("o", (W, H * v))]
            mix += [("dkv", (mx["kv_rank"] + mx["rot_dim"], W)), ("dkv.norm", (mx["kv_rank"],))] if own else []
        elif x["type"] == "attention":
            mix = [("q", (H * d, W)), ("o", (W, H * v))] + ([("k", (G * d, W)), ("v", (G * v, W))] if own else [])
        elif x["type"] == "channel_delta":
            mix = []
            for t, c in (("q", G * d), ("k", G * d), ("v", H * v)):
                mix += [(t, (c, W)), (t + ".conv", (c, mx["conv"]))]
            mix += [("b", (H, W)), ("A_log", (H,)), ("dt_bias", (H * d,)), ("a1", (d, W)), ("a2", (H * d, d)), ("g1", (d, W)), ("g2", (H * v, d)), ("norm", (v,)),
                    ("o", (W, H * v))]
        else:
            mix = [("q", (H * d, W)), ("k", (H * d, W)), ("v", (H * v, W)), ("g", (H * v, W)), ("o", (W, H * v))]
            mix += [("norm", (H * v,))] if post else []
        out += [(p + "mix." + t, s) for t, s in mix]
        ff = x["mlp"]["ff"]
        out += [(p + "mlp.up", (ff, W)), (p + "mlp.down", (W, ff))]
        if post:
            out += [(p + "mlp.gate", (ff, W)), (p + "norm2", (W,)), (p + "side.gate", (side, W)), (p + "side.proj", (W, side)), (p + "side.norm", (W,))]
    return out


def _layered_weights(cfg, seed):
    at = {name: (n, shape) for n, (name, shape) in enumerate(_layered_names(cfg))}

    def get(name):
        n, shape = at[name]
        conv = name.endswith(".conv")
        offset = 0.0 if len(shape) > 1 or name.endswith("A_log") else -2.0 if name.endswith("dt_bias") else 1.0
        a = generated(seed, 0x200000 + n, shape, 0.5 if conv else SIGMA, offset)
        return a.double() if conv else _held(a, "bf16")
    return get


def _split(x, heads):
    return x.view(x.shape[0], x.shape[1], heads, -1).transpose(1, 2)


def _merge(x):
    return x.transpose(1, 2).flatten(2)


def _decayed(q, k, v, decay):
    """o_i = sum_{j <= i} decay^(i - j) (q_i . k_j) v_j per head"""
    i = torch.arange(q.shape[2], device="cuda")
    dist = (i[:, None] - i[None]).double()
    o = torch.empty_like(v)
    for h, g in enumerate(decay):
        o[:, h] = ((q[:, h] @ k[:, h].transpose(1, 2)) * torch.where(dist >= 0, float(g) ** dist.clamp(min=0), 0.0)) @ v[:, h]
    return o


def _softmax_heads(score, seen, values):
    """score(h) and values(h): one head's scores [B, T, T] and values [B, T, D]"""
    return torch.stack([score(h).masked_fill(~seen, -math.inf).softmax(-1) @ values(h) for h in range(score.heads)], 1)


def _yarn(rot):
    """(frequencies, factor on cosine and sine) with the context extended by rot['scaling']"""
    n, base, sc = rot["dims"], float(rot["base"]), rot["scaling"]
    f = _freq(n, base)
    turns = lambda t: n * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(base))  # noqa: E731
    lo, hi = max(math.floor(turns(sc["fast"])), 0.0), min(math.ceil(turns(sc["slow"])), n - 1.0)
    ramp = ((torch.arange(n // 2, device="cuda", dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1


def _mixer64(layer, h, get, p, eps, pos, caches, i):
    mx, kind = layer["mixer"], layer["type"]
    H, d = mx["heads"], mx["dim"]
    sigmoid, silu = torch.sigmoid, torch.nn.functional.silu
    seen = pos[:, None] >= pos[None]
    proj = lambda t: h @ get(p + t).T  # noqa: E731
    src = i if mx.get("kv_from") is None else mx["kv_from"]
    if kind == "latent_attention":
        freq = _freq(mx["rot"]["dims"], mx["rot"]["base"])
        if src == i:
            y = proj("dkv")
            caches[i] = _rms(y[..., :mx["kv_rank"]], eps, get(p + "dkv.norm")), _rotate(y[..., mx["kv_rank"]:], pos, freq, interleaved=True)
        c, kr = caches[src]
        q = _split(_rms(proj("dq"), eps, get(p + "dq.norm")) @ get(p + "uq").T, H)
        qn, qr = q[..., :d], _rotate(q[..., d:].contiguous(), pos, freq, interleaved=True)
        k, v = _split(c @ get(p + "uk").T, H), _split(c @ get(p + "uv").T, H)

        def score(a):
            return (qn[:, a] @ k[:, a].transpose(1, 2) + qr[:, a] @ kr.transpose(1, 2)) * mx["scale"]
        score.heads = H
        o = _softmax_heads(score, seen, lambda a: v[:, a]) * sigmoid(proj("g")).transpose(1, 2)[..., None]
        return _merge(o) @ get(p + "o").T
    if kind == "retention":
        freq = _freq(mx["rot"]["dims"], mx["rot"]["base"])
        q, k = (_rotate(_split(proj(t), H), pos, freq) for t in "qk")
        o = _decayed(q, k * d ** -0.5, _split(proj("v"), H), mx["decay"])
        return (_merge(_rms(o, eps)) * silu(proj("g"))) @ get(p + "o").T
    if kind == "lightning":
        q, k, v = (_split(silu(proj(t)), H) for t in "qkv")
        return (_rms(_merge(_decayed(q, k, v, mx["decay"])), eps, get(p + "norm")) * sigmoid(proj("g"))) @ get(p + "o").T
    G = mx["kv_heads"]
    if kind == "attention":
        freq, factor = _yarn(mx["rot"])
        if src == i:
            caches[i] = _rms(_rotate(_split(proj("k"), G), pos, freq, factor, True), eps), _split(proj("v"), G)
        k, v = caches[src]
        q = _rms(_rotate(_split(proj("q"), H), pos, freq, factor, True), eps)

        def score(a):
            return mx["softcap"] * torch.tanh(q[:, a] @ k[:, a // (H // G)].transpose(1, 2) * mx["scale"] / mx["softcap"])
        score.heads = H
        o = _softmax_heads(score, seen & (pos[:, None] - pos[None] < mx["mask"]["size"]), lambda a: v[:, a // (H // G)])
        return _merge(o) @ get(p + "o").T

    def conv(t):                                                   # causal, the last tap meets the current row
        y, taps = proj(t), get(p + t + ".conv")
        n = taps.shape[1]
        y = torch.nn.functional.pad(y, (0, 0, n - 1, 0))
        return silu(sum(y[:, j:j + h.shape[1]] * taps[:, j] for j in range(n)))
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q = (unit(_split(conv("q"), G)) * d ** -0.5).repeat_interleave(H // G, 1)
    k, v = unit(_split(conv("k"), G)).repeat_interleave(H // G, 1), _split(conv("v"), H)
    beta = sigmoid(proj("b")).transpose(1, 2)
    g = torch.exp(-torch.exp(get(p + "A_log"))[None, :, None, None] * _split(torch.nn.functional.softplus(proj("a1") @ get(p + "a2").T + get(p + "dt_bias")), H))
    S, o = torch.zeros(h.shape[0], H, d, v.shape[-1], device="cuda", dtype=torch.float64), torch.empty_like(v)
    for t in range(h.shape[1]):
        S.mul_(g[:, :, t, :, None])
        u = beta[:, :, t, None] * (v[:, :, t] - torch.einsum("bhdv,bhd->bhv", S, k[:, :, t]))
        S.add_(k[:, :, t, :, None] * u[:, :, None, :])
        o[:, :, t] = torch.einsum("bhdv,bhd->bhv", S, q[:, :, t])
    return (_merge(_rms(o, eps, get(p + "norm"))) * sigmoid(proj("g1") @ get(p + "g2").T)) @ get(p + "o").T


def _layered64(cfg, seed, ids, places):
    get, eps, post = _layered_weights(cfg, seed), cfg["norm"]["eps"], cfg["architecture"] == "Kevatar"
    x = get("embed")[ids]
    pos = torch.arange(ids.shape[1], device="cuda")
    caches = {}
    side = get("side.embed") if post else None
    for i, layer in enumerate(cfg["layers"]):
        p = f"l{i}."
        if not post:
            h = _rms(x, eps, get(p + "norm1"))
            y = _mixer64(layer, h, get, p + "mix.", eps, pos, caches, i)
            x = x + y + torch.relu(h @ get(p + "mlp.up").T) ** 2 @ get(p + "mlp.down").T
            continue
        x = x + _rms(_mixer64(layer, x, get, p + "mix.", eps, pos, caches, i), eps, get(p + "norm1"))
        f = (torch.nn.functional.silu(x @ get(p + "mlp.gate").T) * (x @ get(p + "mlp.up").T)) @ get(p + "mlp.down").T
        x = x + _rms(f, eps, get(p + "norm2"))
        n = cfg["token_side"]["dim"]
        e = torch.nn.functional.gelu(x @ get(p + "side.gate").T, approximate="tanh") * side[ids, i * n:(i + 1) * n]
        x = x + _rms(e @ get(p + "side.proj").T, eps, get(p + "side.norm"))
    logits = _rms(x[:, places], eps, get("final.norm")) @ get("embed" if post else "head").T
    cap = cfg.get("logit_softcap")
    return cap * torch.tanh(logits / cap) if cap else logits


def _whisper64(case, seed):
    c, w = WHISPER_BASE, {k: _held(v, "bf16") for k, v in whisper_weights(seed).items()}
    H, d = c["heads"], c["d_model"]
    scale = (d / H) ** -0.25
    F = torch.nn.functional

    def heads(x):                                                  # feature f = head + H * d
        return x.view(x.shape[0], x.shape[1], d // H, H).permute(0, 3, 1, 2)

    def linear(x, p):
        return x @ w[p + ".weight"].T + w.get(p + ".bias", 0.0)

    def norm(x, p):
        return F.layer_norm(x, (d,), w[p + ".weight"], w[p + ".bias"], 1e-5)

    def attend(x, k, v, p):
        o = (heads(linear(x, p + ".q_proj") * scale) @ k.transpose(2, 3)).softmax(-1) @ v
        return linear(o.permute(0, 2, 3, 1).reshape(x.shape), p + ".out_proj")

    def keys(x, p):
        return heads(linear(x, p + ".k_proj") * scale), heads(linear(x, p + ".v_proj"))

    def mlp(x, p):
        return linear(F.gelu(linear(x, p + ".fc1"), approximate="tanh"), p + ".fc2")

    x = torch.as_tensor(whisper_mel(case, seed), device="cuda").double()
    for t, stride in (("conv1", 1), ("conv2", 2)):                 # merged weight column = channel + channels * tap
        weight = w[f"model.encoder.{t}.weight"].view(d, 3, -1).transpose(1, 2)
        x = F.gelu(F.conv1d(x, weight, w[f"model.encoder.{t}.bias"], stride, 1), approximate="tanh")
    x = x.transpose(1, 2)
    rates = torch.exp(-math.log(10000.0) / (d / 2 - 1) * torch.arange(d // 2, device="cuda", dtype=torch.float64))
    a = torch.arange(x.shape[1], device="cuda", dtype=torch.float64)[:, None] * rates
    x = x + torch.cat([a.sin(), a.cos()], 1)
    for i in range(c["enc_layers"]):
        p = f"model.encoder.layers.{i}"
        h = norm(x, p + ".self_attn_layer_norm")
        x = x + torch.cat([attend(h[b:b + 1], *keys(h[b:b + 1], p + ".self_attn"), p + ".self_attn") for b in range(len(h))])
        x = x + mlp(norm(x, p + ".final_layer_norm"), p)
    x = norm(x, "model.encoder.layer_norm")
    cross = [keys(x, f"model.decoder.layers.{i}.encoder_attn") for i in range(c["dec_layers"])]
    tok = _ids(tokens_of(case, seed, 1, c["vocab"])[:, 0])
    past = [None] * c["dec_layers"]
    for step in range(case["steps"] + 1):
        y = (w["model.decoder.embed_tokens.weight"][tok] + w["model.decoder.embed_positions.weight"][step])[:, None]
        for i in range(c["dec_layers"]):
            p = f"model.decoder.layers.{i}"
            h = norm(y, p + ".self_attn_layer_norm")
            new = keys(h, p + ".self_attn")
            past[i] = new if past[i] is None else tuple(torch.cat(t, 2) for t in zip(past[i], new))
            y = y + attend(h, *past[i], p + ".self_attn")
            y = y + attend(norm(y, p + ".encoder_attn_layer_norm"), *cross[i], p + ".encoder_attn")
            y = y + mlp(norm(y, p + ".final_layer_norm"), p)
        logits = (norm(y, "model.decoder.layer_norm") @ w["model.decoder.embed_tokens.weight"].T)[:, 0]
        tok = logits.argmax(-1)
    return logits


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "decode":
        cfg = LLAMA[case["model"]]
        ids = _ids(tokens_of(case, seed, case["steps"], cfg["vocab"]))
        y = _llama64(cfg, seed, case["dtype"], ids, case["context"], _capacity(case), last=[case["steps"] - 1] * case["batch"])
        return dict(logits=y, chosen_logit=y.max(-1, keepdim=True).values)
    if kind == "prompt":
        cfg = LLAMA[case["model"]]
        last = lengths_of(case, seed) - 1 if case["ragged"] else [case["tokens"] - 1] * case["batch"]
        return dict(logits=_llama64(cfg, seed, case["dtype"], _ids(tokens_of(case, seed, case["tokens"], cfg["vocab"])), last=last))
    if kind == "layered":
        cfg, n = LAYERED[case["model"]], case["tokens"]
        ids = _ids(tokens_of(case, seed, n + case["steps"], cfg["vocab"]))
        y = _layered64(cfg, seed, ids, [n - 1, n + case["steps"] - 1])
        return dict(prompt_logits=y[:, 0], logits=y[:, 1], chosen_logit=y[:, 1].max(-1, keepdim=True).values)
    if kind == "whisper":
        return dict(tokens=None, logits=_whisper64(case, seed))
    if kind == "flash":
        q, k, v = (t.double() for t in flash_inputs(case, seed))
        out = torch.empty_like(q)
        i = torch.arange(case["seq"], device="cuda")
        for b in range(case["batch"]):
            for h in range(case["heads"]):
                s = (q[b, h] @ k[b, h].T) / math.sqrt(case["dim"])
                out[b, h] = (s.masked_fill(i[None] > i[:, None], -math.inf) if case["causal"] else s).softmax(-1) @ v[b, h]
        return out
    cfg = LLAMA[case["model"]]
    return _llama64(cfg, seed, "f32", _ids(tokens_of(case, seed, case["tokens"], cfg["vocab"])), rope_base=L.nn.Llama.ROPE_BASE)
