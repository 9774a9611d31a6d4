"""Replays of recorded graphs (runs of primitive steps as one kernel) against the same steps called one by one, bit for bit and in every buffer."""
import numpy as np
import pytest

import luminal_oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def wherever_it_can_be(monkeypatch):
    """The kernel also where the library expects nothing of it: these tests are about what it computes."""
    monkeypatch.setenv("LMB200_GRAPH_KERNEL", "1")


def every_buffer(cg):
    return {nid: a.numpy() for nid, a in cg.results.items()}


def same_bits(L, device, g, inputs, varied=(), **kw):
    recorded, plain = L.compile(g, device, **kw), L.compile(g, device, capture=False, **kw)
    for turn in range(3):                                          # the first call records and replays, the others replay on other values
        for nid in varied:
            inputs[nid] = np.roll(inputs[nid], turn)
        recorded(inputs), plain(inputs)
        a, b = every_buffer(recorded), every_buffer(plain)
        keep = kw.get("outputs") or a
        for nid in keep:
            assert np.array_equal(a[nid].view(np.int32), b[nid].view(np.int32)), (turn, nid, type(g.nodes[nid - 1].op).__name__, a[nid].shape)
    before = device.launch_count()
    recorded(inputs)
    launches = device.launch_count() - before
    recorded.close()
    return launches, recorded.kernel_count()


@pytest.mark.parametrize("cfg,batch,tokens", [(dict(hidden=64, n_heads=4, n_kv_heads=2, intermediate=96), 2, 16), (dict(hidden=48, n_heads=3, n_kv_heads=3, intermediate=40), 1, 2),
                                              (dict(hidden=256, n_heads=8, n_kv_heads=8, intermediate=688), 1, 33), (dict(hidden=512, n_heads=8, n_kv_heads=2, intermediate=1408), 3, 70)])
@pytest.mark.parametrize("shared", [False, True])
def test_llama_graphs(lib_built, device, cfg, batch, tokens, shared):
    L = lib_built
    g, reg = L.Graph(), {}
    net = L.nn.Llama(g, reg, vocab_size=300, n_layers=2, **cfg)
    tok = L.tensor(g, [batch, tokens])
    out = net(tok, 0)
    inputs = {t.id: O.synth_normal(3, t.id, t.shape, 0.3) for t in reg.values()}
    inputs[tok.id] = O.synth_tokens(5, 999, (batch, tokens), 300).astype(np.float32)
    launches, steps = same_bits(L, device, g, inputs, [tok.id], **(dict(outputs=[out.id]) if shared else {}))
    if not shared and cfg["hidden"] <= 256:
        assert launches == 1 and steps > 100                       # small graphs are one kernel; with shared blocks their order may not allow it


def random_graph(G, rng, steps):
    """Movements on movements, broadcasts, reductions, products and element-wise steps on whatever is there."""
    g = G.Graph()
    pool = [G.tensor(g, [int(n) for n in rng.integers(1, 7, int(rng.integers(1, 5)))]) for _ in range(3)]
    pool.append(G.tensor(g, [int(rng.integers(2, 40)), int(rng.integers(2, 40))]))
    leaves = list(pool)
    for _ in range(steps):
        a = pool[-1 - int(rng.integers(min(4, len(pool))))] if rng.random() < 0.7 else pool[int(rng.integers(len(pool)))]
        r, size = len(a.shape), int(np.prod(a.shape))
        kind = int(rng.integers(11))
        if kind == 0:
            t = G.permute(a, [int(i) + 1 for i in rng.permutation(r)])
        elif kind == 1:
            d = [x for x in range(1, size + 1) if size % x == 0]
            x = int(rng.choice(d))
            y = int(rng.choice([z for z in range(1, size // x + 1) if (size // x) % z == 0]))
            t = G.reshape(a, [x, y, size // x // y][:: int(rng.choice([1, -1]))])
        elif kind == 2 and r < 6 and size < 4000:
            t = G.expand(a, int(rng.integers(1, r + 2)), int(rng.integers(1, 5)))
        elif kind == 3:
            lo = [int(rng.integers(n)) for n in a.shape]
            t = G.slice_(a, [(s, int(rng.integers(s + 1, n + 1))) for s, n in zip(lo, a.shape)])
        elif kind == 4 and size < 4000:
            t = G.pad(a, [(int(rng.integers(3)), int(rng.integers(3))) for _ in a.shape])
        elif kind == 5 and r > 1:
            t = (G.sum_ if rng.random() < 0.5 else G.max_reduce)(a, int(rng.integers(1, r + 1)))
        elif kind == 6 and 2 <= r <= 4:
            m = G.permute(a, list(range(1, r - 1)) + [r, r - 1])
            t = G.matmul(a, m) * np.float32(0.05) if rng.random() < 0.5 else G.matmul(m, a) * np.float32(0.05)
        elif kind == 7:
            t = G.cumsum_last_dim(a) * np.float32(0.25)
        elif kind == 8:
            t = a * np.float32(0.5) + G.permute(G.permute(a, list(range(r, 0, -1))), list(range(r, 0, -1)))
        elif kind == 9:
            t = G.sin(a) if rng.random() < 0.5 else G.relu(a) + np.float32(0.125)
        else:
            t = G.std_norm(a, r) if size > 1 else G.exp2(a * np.float32(0.01))
        pool.append(t)
    return g, leaves


@pytest.mark.parametrize("seed", range(24))
@pytest.mark.parametrize("fuse", [True, False])
def test_random_graphs(lib_built, device, seed, fuse):
    rng = np.random.default_rng(seed)
    g, leaves = random_graph(lib_built.graph, rng, 40)
    inputs = {t.id: rng.standard_normal(t.shape).astype(np.float32) for t in leaves}
    same_bits(lib_built, device, g, inputs, [t.id for t in leaves], fuse=fuse)


def test_large_steps_stay_kernels(lib_built, device):
    """Element-wise steps and products beyond the rule's sizes between small ones, and values the products' order must carry: infinities and NaN."""
    G = lib_built.graph
    rng = np.random.default_rng(1)
    g = G.Graph()
    a, w = G.tensor(g, [700, 800]), G.tensor(g, [900, 800])
    small = G.sum_(G.exp2(G.permute(a, [2, 1]) * np.float32(0.1)), 2)
    big = G.matmul(G.relu(a) + np.float32(1.0), G.permute(w, [2, 1]))
    out = G.sum_(big * np.float32(0.01), 1) + G.sum_(G.permute(w, [2, 1]), 1)
    tail = G.permute(G.expand(out, 1, 3), [2, 1]) * np.float32(2.0)
    tail = G.max_reduce(tail + G.reshape(G.sum_(small, 1) * np.float32(0.0) + np.float32(1.0), [1]), 1)
    x = rng.standard_normal((700, 800)).astype(np.float32)
    x[3, 5], x[7, 9], x[11, 2] = np.inf, -np.inf, np.nan
    launches, steps = same_bits(lib_built, device, g, {a.id: x, w.id: rng.standard_normal((900, 800)).astype(np.float32)}, [w.id])
    assert launches < steps


def large_movement(G, tail):
    """A product that reads past a large movement (a kernel of its own) to the movement's source, alone in front of everything; then large and small steps."""
    g = G.Graph()
    w, a = G.tensor(g, [1024, 1024]), G.tensor(g, [32, 1024])
    m = G.permute(w, [2, 1])
    x = G.matmul(a, m)
    big = m * np.float32(0.5) + np.float32(1.0)
    y = G.sum_(big, 1)
    for i in range(tail):
        y = y * np.float32(0.5) + G.sum_(x, 1) * np.float32(0.01 * (i + 1))
    return g, (w, a), (x, y)


@pytest.mark.parametrize("tail", [4, 9])
@pytest.mark.parametrize("fuse,shared", [(True, False), (False, False), (True, True), (False, True)])
def test_short_stage_reads_past_a_large_movement(lib_built, device, tail, fuse, shared):
    g, (w, a), outputs = large_movement(lib_built.graph, tail)
    rng = np.random.default_rng(tail)
    inputs = {t.id: rng.standard_normal(t.shape).astype(np.float32) for t in (w, a)}
    same_bits(lib_built, device, g, inputs, [w.id, a.id], fuse=fuse, **(dict(outputs=[t.id for t in outputs]) if shared else {}))


def stages_graph(G, rng, steps):
    """Steps around the sizes (2^19 elements, or 16 us longer here) from which one keeps its own kernel: runs fall apart into stages of one step and more, and
    small steps read large movements."""
    g = G.Graph()
    n = 720                                                        # n x n is just below 2^19, n x 800 above
    leaves = [G.tensor(g, [n, n]), G.tensor(g, [n, 800]), G.tensor(g, [24, n]), G.tensor(g, [800, 16])]
    pool = list(leaves)
    pick = lambda ok: [t for t in pool if ok(t)]  # noqa: E731
    for _ in range(steps):
        a = pool[int(rng.integers(len(pool)))]
        r, size, kind = len(a.shape), int(np.prod(a.shape)), int(rng.integers(7))
        if kind <= 1:
            t = G.permute(a, list(range(r, 0, -1)))
        elif kind == 2:
            lo = [int(rng.integers(0, 1 + d // 32)) for d in a.shape]
            t = G.slice_(a, [(s, d) for s, d in zip(lo, a.shape)])
        elif kind == 3 and r == 2:
            mates = pick(lambda t: len(t.shape) == 2 and t.shape[0] == a.shape[1] and t.shape[1] * a.shape[0] < 1 << 20)
            if not mates:
                continue
            t = G.matmul(a, mates[int(rng.integers(len(mates)))]) * np.float32(0.01)
        elif kind == 4 and r > 1:
            t = G.sum_(a, int(rng.integers(1, r + 1))) * np.float32(0.03)
        elif kind == 5 and size < 2000 and r < 3:
            t = G.expand(a, int(rng.integers(1, r + 2)), int(rng.choice([3, 700])))
        else:
            mates = pick(lambda t: t.shape == a.shape)
            t = a * np.float32(0.5) + mates[int(rng.integers(len(mates)))]
        pool.append(t)
    return g, leaves, pool[-4:]


@pytest.mark.parametrize("seed", range(32))
@pytest.mark.parametrize("shared", [False, True])
def test_random_graphs_in_stages(lib_built, device, seed, shared):
    rng = np.random.default_rng(100 + seed)
    g, leaves, last = stages_graph(lib_built.graph, rng, 9 + 3 * (seed % 8))
    inputs = {t.id: rng.standard_normal(t.shape).astype(np.float32) for t in leaves}
    same_bits(lib_built, device, g, inputs, [t.id for t in leaves], fuse=False, **(dict(outputs=sorted({t.id for t in last})) if shared else {}))


def alternating(G, n, k):
    g = G.Graph()
    a = G.tensor(g, [n // 64, 64])
    t = a
    for i in range(k):
        t = t * t if i % 2 else t + a
    return g, {a.id: np.linspace(-1.0, 1.0, n, dtype=np.float32).reshape(a.shape)}


def test_only_where_it_is_expected_to_be_faster(lib_built, device, monkeypatch):
    """Chains without a movement or a small product stay their recorded kernels; a step of many rounds keeps its kernel among steps that do not."""
    monkeypatch.delenv("LMB200_GRAPH_KERNEL")
    L = lib_built
    for n in (4096, 400_000):
        g, inputs = alternating(L.graph, n, 12)
        launches, steps = same_bits(L, device, g, inputs, fuse=False)
        assert launches == steps == 12
    g, reg = L.Graph(), {}
    net = L.nn.Llama(g, reg, vocab_size=300, n_layers=2, hidden=256, n_heads=8, n_kv_heads=8, intermediate=688)
    tok = L.tensor(g, [1, 33])
    net(tok, 0)
    inputs = {t.id: O.synth_normal(3, t.id, t.shape, 0.3) for t in reg.values()}
    inputs[tok.id] = O.synth_tokens(5, 999, (1, 33), 300).astype(np.float32)
    assert same_bits(L, device, g, inputs, [tok.id])[0] == 1
    g = L.Graph()
    a, w = L.tensor(g, [1, 1024]), L.tensor(g, [1024, 1024])
    t = a
    for _ in range(4):
        t = L.graph.matmul(t, L.graph.permute(w, [2, 1])) * np.float32(0.03)
    big = L.graph.sum_(L.graph.expand(L.graph.reshape(t, [1024]), 1, 3_000), 2)      # rows of 1024 values: a step that keeps its kernel
    out = L.graph.permute(L.graph.expand(big, 1, 2), [2, 1]) * np.float32(0.5)
    launches, steps = same_bits(L, device, g, {a.id: np.ones((1, 1024), np.float32), w.id: O.synth_normal(3, 7, (1024, 1024), 0.3)}, fuse=False)
    assert 1 < launches < steps


@pytest.mark.parametrize("rows,records_first", [(8, True), (40_000, False)])
def test_first_call_records_first_where_the_kernels_are_short(lib_built, device, rows, records_first):
    """Products of a few rows record before they run, products that keep the device busy run while they are recorded; the first call is the later ones' result."""
    G = lib_built.graph
    g = G.Graph()
    a, w = G.tensor(g, [rows, 256]), G.tensor(g, [256, 256])
    t = a
    for _ in range(4):
        t = G.matmul(t, w)
    inputs = {a.id: O.synth_normal(3, 1, a.shape, 1.0), w.id: O.synth_normal(3, 2, w.shape, 0.06)}
    cg = lib_built.compile(g, device)
    assert cg.records_first is records_first
    first = cg(inputs)[t.id].numpy()
    assert "cuda_exec" in cg.cache and np.array_equal(cg(inputs)[t.id].numpy(), first)
    cg.close()
