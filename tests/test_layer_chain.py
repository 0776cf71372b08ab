"""Decode steps in one persistent kernel (csrc/layer_chain.cu) against the kernels one by one and against plain PyTorch in 64 bits."""
import dataclasses
import types
import weakref

import pytest
import torch

from bee2bee_b200.models.config import resolve_config

gpu = pytest.mark.gpu

# Both sides keep every sum in fp32 and round the same intermediates to bf16 (queries, attention output, stream, MLP hidden); a sum in another order
# flips some of those roundings by one unit.  Five roundings of at most 2^-9 each reach the result per layer, so two layers stay below 10 * 2^-9 in the
# worst case and, because they are independent, near sqrt(10) * 2^-9 = 0.006; measured up to 0.004.
REL = 2.0 ** -7


def _tensors(cfg, layers, g):
    H, F, Q, KV = cfg.hidden_size, cfg.ffn_size, cfg.q_dim, cfg.kv_dim
    t = {}

    def rnd(*shape, std):
        return (torch.randn(*shape, generator=g, device="cuda") * std).to(torch.bfloat16)

    for l in range(layers):
        for n, r, c in (("wq", Q, H), ("wk", KV, H), ("wv", KV, H), ("wo", H, Q), ("w_gate", F, H), ("w_up", F, H), ("w_down", H, F)):
            if cfg.glu or n != "w_gate":
                t[f"l{l}.{n}"] = rnd(r, c, std=c ** -0.5)
        for n in ("ln1_w", "ln2_w") + (("post_attn_w", "post_ffn_w") if cfg.post_norms else ()):
            t[f"l{l}.{n}"] = rnd(H, std=0.1) + (0.0 if cfg.gemma_norm else 1.0)
        if cfg.bias:
            for n, w in (("bq", Q), ("bk", KV), ("bv", KV), ("bo", H), ("b_up", F), ("b_down", H), ("ln1_b", H), ("ln2_b", H)):
                t[f"l{l}.{n}"] = rnd(w, std=0.1)
    return t


def _setup(cfg, layers, ctxs, seed=3, spare_pages=1, quant="bf16", news=None, pad=0):
    """a piece and a step of sequences behind ``ctxs`` cached tokens: one new token each, or ``news``, and ``pad`` rows that belong to none"""
    from bee2bee_b200 import ops
    from bee2bee_b200.models.native import BatchMeta, NativePiece

    g = torch.Generator(device="cuda").manual_seed(seed)
    news = news or [1] * len(ctxs)
    S, T = len(ctxs), sum(news) + pad
    need = [(n + c + 63) // 64 for n, c in zip(news, ctxs)]
    order = (torch.randperm(sum(need), generator=g, device="cuda") + spare_pages).cpu().tolist()
    table, at = [], 0
    for n in need:
        table.append(order[at:at + n] + [0] * (max(need) - n))
        at += n
    pos = [c + i for n, c in zip(news, ctxs) for i in range(n)]
    seq = [s for s, n in enumerate(news) for _ in range(n)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    ops.native().init_kernels(0)
    t = _tensors(cfg, layers, g)
    piece = NativePiece(cfg, range(layers), False, False, t, torch.device("cuda", 0), T, S, sum(need) + spare_pages, quant=quant)
    meta = BatchMeta(ids=None, positions=i32(pos + [0] * pad), slots=i32([table[s][p // 64] * 64 + p % 64 for s, p in zip(seq, pos)] + [-1] * pad),
                     q_start=i32([sum(news[:s]) for s in range(S)]), q_len=i32(news), kv_len=i32([n + c for n, c in zip(news, ctxs)]), block_table=i32(table),
                     n_tokens=T, n_seqs=S, max_q=max(news), bucket=pad > 0)
    caches = [torch.randn(c.shape, generator=g, device="cuda").to(torch.bfloat16) for c in list(piece.k_cache.values()) + list(piece.v_cache.values())]
    x = torch.randn(T, cfg.hidden_size, generator=g, device="cuda").to(torch.bfloat16)
    piece.given = t, seq, pos
    return piece, meta, caches, x


def _exact(piece, meta, caches, x):
    """the step in 64 bits from the same weights: result and caches"""
    cfg, (t, seq, pos) = piece.cfg, piece.given
    D, G, H = cfg.head_dim, cfg.n_kv_heads, cfg.n_heads
    caches = [c.double().view(-1, G, D).clone() for c in caches]
    x, n = x.double()[:len(seq)], len(piece.layers)
    slots, table, p64 = meta.slots[:len(seq)].long(), meta.block_table.long(), torch.tensor(pos, device="cuda").double()

    def norm(name, y):
        w = t[name + "_w"].double()
        if cfg.norm == "ln":
            return torch.nn.functional.layer_norm(y, y.shape[-1:], w, t[name + "_b"].double(), cfg.norm_eps)
        return y * (y.pow(2).mean(-1, keepdim=True) + cfg.norm_eps).rsqrt() * (w + 1.0 if cfg.gemma_norm else w)

    def mul(w, y, b):
        return y @ t[w].double().t() + (t[b].double() if b in t else 0.0)

    def turned(y):                                           # channels i and i + D / 2 turn together and lie side by side in the cache
        if cfg.rope_theta <= 0:
            return y
        ang = (p64[:, None] * cfg.rope_theta ** (-torch.arange(0, D, 2, device="cuda").double() / D))[:, None]
        a, b = y[..., :D // 2], y[..., D // 2:]
        return torch.stack([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1).flatten(-2)

    for l in range(n):
        h = norm(f"l{l}.ln1", x)
        q, k, v = (mul(f"l{l}.w{c}", h, f"l{l}.b{c}").view(len(x), -1, D) for c in "qkv")
        q, kc, vc = turned(q) * cfg.softmax_scale, caches[l], caches[n + l]
        kc[slots], vc[slots] = turned(k), v
        a = torch.empty(len(x), H, D, device="cuda", dtype=torch.float64)
        for i, (s, p) in enumerate(zip(seq, pos)):
            w = cfg.layer_window(l)
            keys = torch.arange(max(0, p + 1 - w) if w else 0, p + 1, device="cuda")
            rows = table[s][keys // 64] * 64 + keys % 64
            sc = torch.einsum("gjd,kgd->gjk", q[i].view(G, H // G, D), kc[rows])
            if cfg.attn_softcap:
                sc = cfg.attn_softcap * torch.tanh(sc / cfg.attn_softcap)
            a[i] = torch.einsum("gjk,kgd->gjd", sc.softmax(-1), vc[rows]).reshape(H, D)
        o = mul(f"l{l}.wo", a.flatten(1), f"l{l}.bo")
        x = x + (norm(f"l{l}.post_attn", o) if cfg.post_norms else o)
        h = norm(f"l{l}.ln2", x)
        up = mul(f"l{l}.w_up", h, f"l{l}.b_up")
        if cfg.glu:
            gate = mul(f"l{l}.w_gate", h, "")
            up = up * (torch.nn.functional.gelu(gate, approximate="tanh") if cfg.act == "gelu_tanh" else torch.nn.functional.silu(gate))
        else:
            up = torch.nn.functional.gelu(up, approximate="tanh")
        o = mul(f"l{l}.w_down", up, f"l{l}.b_down")
        x = x + (norm(f"l{l}.post_ffn", o) if cfg.post_norms else o)
    return x, [c.view(-1, 64, G, D) for c in caches]


def _run(piece, meta, caches, x, chain):
    """one step: result and caches"""
    cache = list(piece.k_cache.values()) + list(piece.v_cache.values())
    for c, v in zip(cache, caches):
        c.copy_(v)
    piece._chain_pays = lambda m: chain                      # (the kernel is held against the others also where it is the slower one)
    out = piece.forward(meta, x_in=x).clone()
    del piece._chain_pays
    torch.cuda.synchronize()
    return out, [c.clone() for c in cache]


def _gave_up(piece):
    """launches of the piece's plan that ended early"""
    return int(piece._chain.control[2])


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


def _rows(a, b):
    """the largest relative error of a row"""
    a, b = a.double(), b.double()
    return float(((a - b).norm(dim=-1) / b.norm(dim=-1).clamp_min(1e-30)).max())


# The bound of a whole result is one of the mean over its rows: a single row has fewer values (128 at least) and may lie above the mean.  Twice the bound is
# still far below what a wrong row gives (a key or value of another token: 1.4; one that is turned for the position beside its own: 0.2 and more).
def _same_step(meta, caches, out, got, ref, ref_caches, rel):
    """results and new cache rows, row by row; all other rows of the caches are as they were"""
    new = meta.slots[meta.slots >= 0].long()
    live = torch.nonzero(meta.slots >= 0).flatten()
    assert _rel(out[live], ref[live]) < rel and _rows(out[live], ref[live]) < 2 * rel
    for a, b, was in zip(got, ref_caches, caches):
        a, b, was = (c.flatten(2).flatten(0, 1) for c in (a, b, was))
        assert _rows(a[new], b[new]) < 2 * rel
        old = torch.ones(len(a), dtype=torch.bool, device="cuda")
        old[new] = False
        assert torch.equal(a[old], was[old])


def _compare(piece, meta, caches, x, rel=REL, launches=1):
    from bee2bee_b200 import ops

    ref, ref_caches = _run(piece, meta, caches, x, False)
    n0 = ops.LAUNCHES[0]
    out, got = _run(piece, meta, caches, x, True)
    assert ops.LAUNCHES[0] == n0 + launches                  # the persistent kernel ran
    _same_step(meta, caches, out, got, ref, ref_caches, rel)
    again, _ = _run(piece, meta, caches, x, True)
    live = meta.slots >= 0
    assert torch.equal(again[live], out[live])               # sums in a fixed order
    assert _gave_up(piece) == 0
    return out


class _Plan:
    """stands in for the native plan where there is no GPU"""
    step_tokens, ctas, refused = 64, 132, False

    def __init__(self, *args):
        self.args = args


def _cpu_piece(monkeypatch, cfg=None, layers=2):
    """a piece (of a small Llama) on the CPU, planned as on a GPU"""

    from bee2bee_b200 import ops
    from bee2bee_b200.models.native import NativePiece

    cfg = cfg or resolve_config("tiny-llama")
    H, F, Q, KV = cfg.hidden_size, cfg.ffn_size, cfg.q_dim, cfg.kv_dim
    t = {f"l{l}.{n}": torch.randn(r, c) for l in range(layers)
         for n, r, c in (("wq", Q, H), ("wk", KV, H), ("wv", KV, H), ("wo", H, Q), ("w_gate", F, H), ("w_up", F, H), ("w_down", H, F))}
    t.update({f"l{l}.{n}": torch.ones(H) for l in range(layers) for n in ("ln1_w", "ln2_w", "ln1_b", "ln2_b")})
    t.update({f"l{l}.{n}": torch.ones(w) for l in range(layers) for n, w in (("bq", Q), ("bk", KV), ("bv", KV), ("bo", H), ("b_up", F), ("b_down", H))})
    piece = NativePiece(cfg, range(layers), False, False, t, torch.device("cpu"), 4, 4, 8)
    def stamp(rows):                                         # (the native one where the extension is built)
        return [[(x.data_ptr(), x.shape, x.stride(), x.dtype) for x in row] for row in rows]

    try:
        stamp = ops.native().tensor_stamp
    except RuntimeError:
        pass
    monkeypatch.setattr(ops, "native", lambda: types.SimpleNamespace(LayerChain=_Plan, get_attn_tc_min_q=lambda: 2, tensor_stamp=stamp))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    piece._plan_chain()
    return piece


def _step(n=1):
    from bee2bee_b200.models.native import BatchMeta

    i32 = lambda v: torch.tensor(v, dtype=torch.int32)  # noqa: E731
    return BatchMeta(ids=None, positions=i32([3] * n), slots=i32([67] * n), q_start=i32(list(range(n))), q_len=i32([1] * n), kv_len=i32([4] * n),
                     block_table=i32([[1, 0]] * n), n_tokens=n, n_seqs=n, max_q=1)


# measured on B200, two layers, us: kernels one by one / the persistent kernel
@pytest.mark.parametrize("seqs,keys,takes", [(1, 500, True),          # 187 / 163
                                             (1, 8000, True),         # 201 / 188
                                             (8, 8000, True),         # 266 / 239
                                             (17, 500, True),         # 201 / 179
                                             (17, 4000, False),       # 276 / 292
                                             (20, 8000, False),       # 387 / 420
                                             (32, 8000, True),        # 502 / 462
                                             (34, 8000, False),       # 536 / 581
                                             (40, 8000, True),        # 652 / 593
                                             (50, 8000, False),       # 694 / 730
                                             (64, 8000, True)])       # 804 / 770
def test_route_follows_the_keys(monkeypatch, seqs, keys, takes):
    """attention of the persistent kernel leaves most CTAs waiting where the (sequence, head) pairs do not fill its last round: behind many keys that costs more
    than the kernel gains.  The block table says how many there may be"""
    from bee2bee_b200.models.native import Handoff

    piece = _cpu_piece(monkeypatch)
    piece.cfg = dataclasses.replace(piece.cfg, n_heads=32, n_kv_heads=8, head_dim=128)       # (Llama-3-8B's)
    meta = dataclasses.replace(_step(seqs), block_table=torch.zeros(seqs, (keys + 64) // 64, dtype=torch.int32))
    assert piece._chain_takes(meta, torch.zeros(seqs, 256, dtype=torch.bfloat16), Handoff()) == takes


# measured on B200, the layers of gpt2, us: kernels one by one / the persistent kernel
@pytest.mark.parametrize("tokens,keys,takes", [(1, 900, True),        # 450 / 441
                                               (8, 1024, True),       # 564 / 470
                                               (12, 256, True),       # 517 / 385
                                               (16, 900, False),      # 609 / 641
                                               (24, 124, True),       # 469 / 389
                                               (32, 300, False),      # 497 / 521
                                               (64, 64, True),        # 612 / 426
                                               (64, 184, False),      # 640 / 659
                                               (64, 964, False),      # 753 / 1533
                                               (65, 65, False)])
def test_route_of_layer_norm_models_follows_the_keys(monkeypatch, tokens, keys, takes):
    """the persistent kernel reads all keys of a (token, head) for that one alone; a call that knows how many there are says so"""
    from bee2bee_b200.models.native import BatchMeta, Handoff

    piece = _cpu_piece(monkeypatch, _gpt2(768, 12, 768), layers=1)
    x = torch.zeros(tokens, 768, dtype=torch.bfloat16)
    i32 = lambda *shape: torch.zeros(shape, dtype=torch.int32)  # noqa: E731
    meta = BatchMeta(ids=None, positions=i32(tokens), slots=i32(tokens), q_start=i32(1), q_len=i32(1), kv_len=i32(1), block_table=i32(1, (keys + 63) // 64),
                     n_tokens=tokens, n_seqs=1, max_q=tokens, max_keys=keys)
    assert piece._chain_takes(meta, x, Handoff()) == takes
    # without that the block table's width is taken, at most the model's positions
    assert piece._chain_takes(dataclasses.replace(meta, max_keys=0, block_table=i32(1, 64)), x, Handoff()) == (tokens * 12 <= 132)
    assert piece._chain_takes(dataclasses.replace(meta, max_keys=0, block_table=i32(1, 1)), x, Handoff()) == (tokens <= 64)


# The other families of layers, two layers, us: kernels one by one / the persistent kernel.  The gains are the smallest that were measured, so close calls go one by one.
@pytest.mark.parametrize("name,mx,seqs,keys,pays", [("gemma-2-2b", False, 1, 500, True),          # 120 / 97
                                                    ("gemma-2-2b", False, 2, 4000, True),         # 123 / 115
                                                    ("gemma-2-2b", False, 2, 8000, False),        # 135 / 132
                                                    ("gemma-2-2b", False, 8, 8000, True),         # 176 / 154
                                                    ("gemma-2-2b", False, 34, 4000, False),       # 303 / 352
                                                    ("gemma-2-2b", False, 40, 8000, True),        # 501 / 479
                                                    ("llama-3-8b", True, 17, 500, True),          # 151 / 135
                                                    ("llama-3-8b", True, 17, 2000, False),        # 189 / 187
                                                    ("llama-3-8b", True, 17, 4000, False),        # 228 / 250
                                                    ("llama-3-8b", True, 24, 4000, True),         # 266 / 257
                                                    ("llama-3-8b", True, 24, 8000, False),        # 375 / 389
                                                    ("llama-3-8b", True, 32, 8000, True),         # 453 / 423
                                                    ("llama-3-8b", False, 10, 16000, True),       # 385 / 378
                                                    ("llama-3-8b", False, 50, 2000, True),        # 346 / 322
                                                    ("llama-3-8b", False, 50, 4000, False)])      # 456 / 458
def test_what_attention_costs(name, mx, seqs, keys, pays):
    """attention's loss against what the persistent kernel gains besides (``NativePiece._chain_pays``)"""
    from bee2bee_b200.models.native import NativePiece

    piece = types.SimpleNamespace(cfg=resolve_config(name), layers=range(2), mx_fuse=mx, _chain_ln=False, _chain=types.SimpleNamespace(ctas=132))
    meta = types.SimpleNamespace(max_keys=keys + 1, n_tokens=seqs, n_seqs=seqs)
    assert NativePiece._chain_pays(piece, meta) == pays


def test_plans_of_graphs_are_kept(monkeypatch):
    from bee2bee_b200.models.native import Handoff

    piece = _cpu_piece(monkeypatch)
    x = torch.zeros(1, piece.cfg.hidden_size, dtype=torch.bfloat16)
    recording = [True]
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: recording[0])
    assert piece._chain_takes(_step(), x, Handoff())
    first = weakref.ref(piece._chain)
    recording[0] = False
    piece.w["l0.wo"] = piece.w["l0.wo"].clone()
    assert piece._chain_takes(_step(), x, Handoff()) and piece._chain is not first()
    assert first() is not None                               # a graph reads it
    second = weakref.ref(piece._chain)
    piece.w["l0.wo"] = piece.w["l0.wo"].clone()
    assert piece._chain_takes(_step(), x, Handoff())
    assert second() is None                                  # no graph does


def test_what_a_plan_refuses(monkeypatch):
    """weights and metadata that the persistent kernel does not take are no error: the kernels one by one have them"""
    from bee2bee_b200 import ops
    from bee2bee_b200.models.native import Handoff

    piece = _cpu_piece(monkeypatch)
    x = torch.zeros(2, piece.cfg.hidden_size, dtype=torch.bfloat16)
    meta = _step(2)
    # room for more sequences than take part
    assert not piece._chain_takes(dataclasses.replace(meta, q_len=torch.tensor([1, 1, 0], dtype=torch.int32)), x, Handoff())
    assert piece._chain_takes(meta, x, Handoff())
    with monkeypatch.context() as mp:                        # attention on CUDA cores
        mp.setattr(ops, "get_attn_tc_min_q", lambda: 0)
        assert not piece._chain_takes(meta, x, Handoff())

    def refuse(self, *args):
        raise RuntimeError("sizes")

    old = piece.w["l0.wo"]
    with monkeypatch.context() as mp:
        mp.setattr(_Plan, "__init__", refuse)
        piece.w["l0.wo"] = old[:, :-8]
        for _ in range(2):
            assert not piece._chain_takes(meta, x, Handoff())
    piece.w["l0.wo"] = old
    assert piece._chain_takes(meta, x, Handoff())


def test_plans_follow_shapes_and_types(monkeypatch):
    """what replaces a weight may lie where the old one lay"""
    from bee2bee_b200.models.native import Handoff

    piece = _cpu_piece(monkeypatch)
    x = torch.zeros(1, piece.cfg.hidden_size, dtype=torch.bfloat16)
    w = piece.w["l0.wo"]
    for new in (w.view(-1, 64), w.view(torch.float16), w.t()):
        old = piece._chain
        assert piece._chain_takes(_step(), x, Handoff()) and piece._chain is old
        piece.w["l0.wo"] = new
        assert piece._chain_takes(_step(), x, Handoff()) and piece._chain is not old


@gpu
@pytest.mark.parametrize("seqs", [1, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("model", ["tiny-llama", "tiny-mistral", "tiny-gemma2"])
def test_token_tiles(model, seqs):
    """edges of the token tiles; few and many CTAs per (sequence, key/value head); windows that cut keys off; capped scores and norms behind O and down"""
    _compare(*_setup(resolve_config(model), 2, [1 + (37 * i) % 290 for i in range(seqs)]))


@gpu
@pytest.mark.parametrize("hidden,heads,kv,dim,ffn", [(384, 4, 2, 128, 448), (2304, 8, 4, 256, 1216), (1024, 16, 2, 128, 8256), (4096, 32, 8, 128, 14336)])
def test_shares_of_the_products(hidden, heads, kv, dim, ffn):
    """odd numbers of blocks of K, CTAs without a share, tiles of fewer than 128 rows, gate/up shares that start inside a block of 64 features"""
    cfg = dataclasses.replace(resolve_config("tiny-llama"), hidden_size=hidden, n_heads=heads, n_kv_heads=kv, head_dim=dim, ffn_size=ffn)
    _compare(*_setup(cfg, 2, [5, 130, 64, 63, 127]))


@gpu
@pytest.mark.parametrize("model,ctxs", [("tiny-llama", [0]), ("tiny-llama", [127, 128, 129, 255, 256]), ("tiny-llama", [3000, 1, 700]), ("tiny-llama", [1500] * 20),
                                        ("zephyr-7b-beta", [1200 - 13 * i for i in range(64)])])
def test_key_tiles(model, ctxs):
    """one key, the edges of a tile, long beside short sequences, and more tiles per CTA than the ring has entries"""
    cfg = resolve_config(model)
    _compare(*_setup(cfg, 1, ctxs))


@gpu
def test_sequences_that_take_no_part():
    piece, meta, caches, x = _setup(resolve_config("tiny-llama"), 2, [50, 80, 0, 200])
    meta.q_len[1] = 0                                        # as GpuRunner marks a free slot
    meta.slots[1] = -1
    ref, ref_caches = _run(piece, meta, caches, x, False)
    piece.attn_buf.zero_()
    out, got = _run(piece, meta, caches, x, True)
    _same_step(meta, caches, out, got, ref, ref_caches, REL)


@gpu
@pytest.mark.parametrize("first", [120, 126, 127, 250])
@pytest.mark.parametrize("rows", [2, 5, 20])
def test_tokens_of_one_text_as_sequences(first, rows):
    """consecutive tokens of a text as sequences that share its pages: each sees the keys and values that the ones in front of it leave in the same step"""
    piece, meta, caches, x = _setup(resolve_config("tiny-llama"), 2, list(range(first, first + rows)))
    table = meta.block_table[-1].tolist()
    meta.block_table[:] = meta.block_table[-1]
    meta.slots.copy_(torch.tensor([table[p // 64] * 64 + p % 64 for p in range(first, first + rows)], dtype=torch.int32))
    for c in caches:                                         # what lies there before the step would be seen
        c.view(-1, c.shape[2] * c.shape[3])[meta.slots.long()] = 50.0
    _compare(piece, meta, caches, x)


@gpu
def test_graph_replay_sees_new_inputs_and_lengths():
    piece, meta, caches, x = _setup(resolve_config("tiny-llama"), 2, [60, 61, 62])
    _run(piece, meta, caches, x, True)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            out = piece.forward(meta, x_in=x)
    torch.cuda.current_stream().wait_stream(stream)
    for step in range(3):
        x.copy_(torch.randn(x.shape, device="cuda"))
        meta.kv_len.fill_(20 + step)
        meta.positions.fill_(19 + step)
        meta.slots.copy_(meta.block_table[:, 0] * 64 + 19 + step)
        ref, _ = _run(piece, meta, caches, x, False)
        for c, v in zip(list(piece.k_cache.values()) + list(piece.v_cache.values()), caches):
            c.copy_(v)
        graph.replay()
        assert _rel(out, ref) < REL


@gpu
def test_a_graph_outlives_its_plan():
    """a graph that was recorded before a weight was replaced goes on reading what it was recorded with"""
    piece, meta, caches, x = _setup(resolve_config("tiny-llama"), 2, [60, 61, 62])
    ref, _ = _run(piece, meta, caches, x, True)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            out = piece.forward(meta, x_in=x)
    torch.cuda.current_stream().wait_stream(stream)
    old = piece.w["l1.w_down"]                               # (the graph's own inputs stay the caller's to keep)
    piece.w["l1.w_down"] = old * 2
    assert _rel(_run(piece, meta, caches, x, True)[0], ref) > 0.1
    fill = [torch.full((n,), 255, device="cuda", dtype=torch.uint8) for n in [512 * k for k in range(1, 65)] for _ in range(8)]
    for c, v in zip(list(piece.k_cache.values()) + list(piece.v_cache.values()), caches):
        c.copy_(v)
    graph.replay()
    assert torch.equal(out, ref)
    del fill


@gpu
def test_replaced_weights_are_let_go():
    """a plan holds no weight or cache that its piece has replaced, also while no decode step follows"""
    piece, meta, caches, x = _setup(dataclasses.replace(resolve_config("tiny-llama"), hidden_size=2048, ffn_size=8192), 2, [60, 61])
    _run(piece, meta, caches, x, True)
    del piece.given
    new = [piece.w["l1.w_down"].clone(), piece.k_cache[0].clone()]
    held = torch.cuda.memory_allocated()
    gone = piece.w["l1.w_down"].nbytes + piece.k_cache[0].nbytes
    piece.w["l1.w_down"], piece.k_cache[0] = new
    del new
    assert torch.cuda.memory_allocated() <= held - gone
    _compare(piece, meta, caches, x)


def _gpt2(hidden=256, heads=4, ffn=1024):
    return dataclasses.replace(resolve_config("tiny-gpt2"), hidden_size=hidden, n_heads=heads, n_kv_heads=heads, head_dim=64, ffn_size=ffn)


# spans (new tokens, cached tokens) of the sequences: edges of the token tiles; one key, the edges of a run of 32 and of a page; more than 128 keys (a CTA
# per token and head) beside short ones; sequences without tokens and rows that belong to none (buckets)
@gpu
@pytest.mark.parametrize("spans,pad", [([(1, 0)], 0), ([(19, 0)], 0), ([(8, 0), (8, 57)], 0), ([(16, 31), (1, 64)], 0), ([(5, 0), (0, 0), (11, 3)], 5),
                                       ([(33, 96)], 0), ([(31, 0), (2, 700)], 4), ([(64, 65)], 0), ([(1, 40 * i) for i in range(20)], 0)])
@pytest.mark.parametrize("hidden,heads,ffn", [(256, 4, 1024), (768, 12, 3072), (384, 6, 512)])
def test_layer_norm_models(spans, pad, hidden, heads, ffn):
    """LayerNorm, biases, an MLP without a gate, 64-wide heads: prompts and decode steps; the norm in front of the first layer is a kernel of its own"""
    # (three layers: sqrt(15) roundings of 2^-9; the kernels one by one also round the weights of the attention)
    _compare(*_setup(_gpt2(hidden, heads, ffn), 3, [c for _, c in spans], seed=11, news=[n for n, _ in spans], pad=pad), rel=2 * REL, launches=2)


# From 64 bits: bf16 rounds five values on the way through a layer, 2^-9 each at most (as above; measured 0.004), LayerNorm models two more (the normed rows).  e4m3
# rounds weights and activations by up to 2^-4, 2^-5.5 in the mean, in each of four products per layer, which the stream they are added to halves.
@gpu
@pytest.mark.parametrize("cfg,news,ctxs,quant,rel", [
    ("tiny-llama", None, [0, 5, 63, 64, 127, 128, 300, 700, 12], "bf16", REL),
    (dict(hidden_size=1024, n_heads=16, n_kv_heads=2, head_dim=128, ffn_size=2752), None, [1 + 29 * i for i in range(40)], "bf16", REL),
    ("tiny-mistral", None, [3, 40, 150, 290, 500], "bf16", REL),
    ("tiny-gemma2", None, [0, 100, 129, 400], "bf16", REL),
    ("gpt2", [19], [0], "bf16", 2 * REL),
    ("gpt2", [5, 1, 20], [3, 127, 150], "bf16", 2 * REL),
    (dict(hidden_size=1024, n_heads=8, n_kv_heads=4, head_dim=128, ffn_size=2816), None, [1 + 37 * i for i in range(20)], "mxfp8", 2.0 ** -4)])
def test_against_64_bits(cfg, news, ctxs, quant, rel):
    cfg = _gpt2(768, 12, 3072) if cfg == "gpt2" else (resolve_config(cfg) if isinstance(cfg, str) else dataclasses.replace(resolve_config("tiny-llama"), **cfg))
    piece, meta, caches, x = _setup(cfg, 2, ctxs, seed=5, quant=quant, news=news)
    out, got = _run(piece, meta, caches, x, True)
    assert _gave_up(piece) == 0
    ref, ref_caches = _exact(piece, meta, caches, x)
    _same_step(meta, caches, out, got, ref, ref_caches, rel)


# Both sides round the same values to e4m3 with the same rule.  A bf16 rounding that falls the other way moves its e4m3 value by one unit (2^-3 of it at
# most), or, where it is the largest of its 32, their common power of two, which moves all of them by less than a unit: less than 2^-4 of the result
# even if half of all values moved.  Measured up to 0.027.
@gpu
@pytest.mark.parametrize("seqs", [1, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("hidden,heads,kv,dim,ffn", [(512, 4, 2, 128, 1024), (640, 8, 1, 128, 1152), (1024, 4, 2, 256, 4224), (4096, 32, 8, 128, 14336)])
def test_block_scaled_fp8(seqs, hidden, heads, kv, dim, ffn):
    """edges of the token tiles; shares that start inside a run of 128 rows; the quantiser of the piece's input is a kernel of its own"""
    cfg = dataclasses.replace(resolve_config("tiny-llama"), hidden_size=hidden, n_heads=heads, n_kv_heads=kv, head_dim=dim, ffn_size=ffn)
    _compare(*_setup(cfg, 2, [1 + (37 * i) % 290 for i in range(seqs)], quant="mxfp8"), rel=2.0 ** -4, launches=2)


@gpu
@pytest.mark.parametrize("seqs,quant", [(1, "bf16"), (8, "bf16"), (40, "bf16"), (5, "mxfp8"), (30, "mxfp8")])
def test_a_wait_that_runs_out(seqs, quant):
    """the launch ends, says so and leaves its counters ready for the next one, while weights, cache pages and activations were on their way"""
    from bee2bee_b200 import ops

    cfg = dataclasses.replace(resolve_config("tiny-llama"), hidden_size=2048, n_heads=16, n_kv_heads=4, head_dim=128, ffn_size=5632)
    piece, meta, caches, x = _setup(cfg, 3, [300] * seqs, quant=quant)
    C = ops.native()
    ref, _ = _run(piece, meta, caches, x, True)
    n0 = C.layer_chain_gave_up()
    word = C.peer_alloc(256)
    told = C.tensor_from_ptr(word, [64], "i32", 0)
    told.zero_()
    torch.cuda.synchronize()
    C.set_wait_policy(word, 1000.0)
    try:
        piece._chain.polls = 1                               # (a product takes several microseconds, a poll less than one)
        for i in range(3):
            _run(piece, meta, caches, x, True)
            assert C.layer_chain_gave_up() == n0 + i + 1 and _gave_up(piece) == i + 1 and int(told[0]) == 1
            words = piece._chain.control[:32 + 7 * 3].clone()
            words[2] = 0
            assert not bool(words.any())
    finally:
        C.set_wait_policy(0, 0.0)
        C.peer_free(word)
    piece._chain.polls = 0
    out, _ = _run(piece, meta, caches, x, True)
    assert torch.equal(out, ref) and _gave_up(piece) == 3


class _Refused:
    """a plan whose launches the device refuses"""
    refused, asked = False, 0

    def __init__(self, plan):
        self.plan = plan

    def __getattr__(self, name):
        return getattr(self.plan, name)

    def run(self, *args):
        self.asked += 1
        self.refused = True
        return False


@gpu
@pytest.mark.parametrize("quant", ["bf16", "mxfp8"])
def test_a_launch_that_is_refused(quant):
    """the kernels one by one take the step and the ones after it"""
    cfg = dataclasses.replace(resolve_config("tiny-llama"), hidden_size=512, n_heads=4, n_kv_heads=2, head_dim=128, ffn_size=1024)
    piece, meta, caches, x = _setup(cfg, 2, [30, 40, 200], quant=quant)
    ref, ref_caches = _run(piece, meta, caches, x, False)
    piece._chain = plan = _Refused(piece._chain)
    for _ in range(2):
        out, got = _run(piece, meta, caches, x, True)
        assert torch.equal(out, ref) and all(torch.equal(a, b) for a, b in zip(got, ref_caches))
    assert plan.asked == 1


@gpu
def test_routes():
    """what the persistent kernel does not take runs on the kernels one by one; replaced weights and caches are seen"""
    from bee2bee_b200 import ops
    from bee2bee_b200.models.native import Handoff

    piece, meta, caches, x = _setup(resolve_config("tiny-llama"), 2, [30] * 65)
    assert not piece._chain_takes(meta, x, Handoff())        # 65 tokens
    wide = dataclasses.replace(resolve_config("tiny-llama"), hidden_size=512, n_heads=4, n_kv_heads=2, head_dim=128, ffn_size=1024)
    for seqs in (32, 33):                                    # block-scaled fp8: up to 32
        piece, meta, caches, x = _setup(wide, 1, [30] * seqs, quant="mxfp8")
        assert piece._chain_takes(meta, x, Handoff()) == (seqs == 32)
    piece, meta, caches, x = _setup(resolve_config("tiny-llama"), 2, [30, 40])
    assert piece._chain_takes(meta, x, Handoff())
    assert not piece._chain_takes(dataclasses.replace(meta, max_q=2), x, Handoff())
    assert not piece._chain_takes(meta, x, Handoff(in_flag=1)) and not piece._chain_takes(meta, x, Handoff(out_x=1))
    wide = torch.zeros(2, 2 * x.shape[1], device="cuda", dtype=torch.bfloat16)
    wide[:, : x.shape[1]] = x
    assert not piece._chain_takes(meta, wide[:, : x.shape[1]], Handoff())
    to = torch.zeros_like(x)
    n0 = ops.LAUNCHES[0]
    piece.forward(meta, x_in=x, out_x=to)                    # a result that goes elsewhere
    assert ops.LAUNCHES[0] > n0 + 1
    old = _compare(piece, meta, caches, x)
    piece.w["l1.w_down"] = piece.w["l1.w_down"] * 2
    assert _rel(_compare(piece, meta, caches, x), old) > 0.1


def _host(seed=0):
    from bee2bee_b200.parallel.gpu_piece import GpuPieceHost

    return GpuPieceHost("tiny-llama", 0, 99, device="cuda:0", max_tokens=64, max_sessions=2, max_seq_len=256, seed=seed)


@gpu
def test_piece_host_reports_a_launch_that_gave_up():
    """a hop whose kernel gave up is an error and leaves its session as it was"""
    host, ref = _host(), _host()
    for h in (host, ref):
        h.forward("a", ids=list(range(3, 40)))
    want = [ref.forward("a", ids=[t])["logits"].clone() for t in (7, 9)]
    assert torch.equal(host.forward("a", ids=[7])["logits"], want[0])
    host.piece._chain.polls = 1
    for _ in range(2):
        with pytest.raises(RuntimeError, match="gave up"):
            host.forward("a", ids=[9])
    host.piece._chain.polls = 0
    assert host.sessions["a"]["len"] == ref.sessions["a"]["len"] - 1
    assert torch.equal(host.forward("a", ids=[9])["logits"], want[1])


@gpu
def test_launch_counts():
    """what is reported is what was launched: a decode step of whole layers is the persistent kernel, embedding and head"""
    from bee2bee_b200.engine.runner import GpuRunner

    host = _host()
    host.forward("a", ids=list(range(3, 40)))
    n0 = host.launches
    host.forward("a", ids=[7])
    assert host.launches - n0 == 3
    for graphs in (False, True):
        r = GpuRunner(resolve_config("tiny-llama"), "", 0, 1, torch.device("cuda:0"), max_batch=4, max_seq_len=256, use_graphs=graphs)
        assert r.launches_per_decode_step() == 5             # (and the positions' advance and the sampler)
        r.close()


@gpu
@pytest.mark.parametrize("model,quant,launches", [("llama", "bf16", 3), ("llama", "mxfp8", 5), ("gpt2", "bf16", 5)])
def test_pieces_named_by_thirds_of_a_layer(model, quant, launches):
    """as the engine names them: token ids in, logits out, one launch for all layers (beside embedding, quantisers or norms, and head)"""
    from bee2bee_b200 import ops
    from bee2bee_b200.models.native import BatchMeta, NativePiece
    from bee2bee_b200.models.weights import init_random

    cfg = _gpt2() if model == "gpt2" else dataclasses.replace(resolve_config("tiny-llama"), hidden_size=512, n_heads=4, n_kv_heads=2, head_dim=128, ffn_size=1024)
    dev, S, n = torch.device("cuda", 0), 3, cfg.n_layers
    ops.native().init_kernels(0)
    t = init_random(cfg, range(n), True, True, device="cuda", dtype=torch.bfloat16, seed=0)
    piece = NativePiece(cfg, range(n), True, True, t, dev, S, S, 4, quant=quant, units=(0, 3 * n))
    assert piece._chain is not None
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    meta = BatchMeta(ids=i32([5, 77, 200]), positions=i32([9, 0, 62]), slots=i32([73, 128, 254]), q_start=i32([0, 1, 2]), q_len=i32([1] * S), kv_len=i32([10, 1, 63]),
                     block_table=i32([[1], [2], [3]]), n_tokens=S, n_seqs=S, max_q=1)
    g = torch.Generator(device="cuda").manual_seed(1)
    caches = [torch.randn(c.shape, generator=g, device="cuda").to(torch.bfloat16) for c in list(piece.k_cache.values()) + list(piece.v_cache.values())]
    ref, ref_caches = _run(piece, meta, caches, None, False)
    n0 = ops.LAUNCHES[0]
    out, got = _run(piece, meta, caches, None, True)
    assert ops.LAUNCHES[0] - n0 == launches
    # (as test_block_scaled_fp8 and test_layer_norm_models, and the head)
    _same_step(meta, caches, out[:, :cfg.vocab_size], got, ref[:, :cfg.vocab_size], ref_caches, 2.0 ** -4 if quant == "mxfp8" else 2 * REL)
    if model == "llama":                                     # pieces that start or end inside a layer
        for units, first, last in (((0, 3 * n - 1), True, False), ((1, 3 * n), False, True), ((2, 3 * n), False, True), ((0, 3 * n - 2), True, False)):
            part = NativePiece(cfg, range(n), first, last, t, dev, S, S, 4, quant=quant, units=units)
            assert part._chain is None and part._chain_of is None


@gpu
def test_two_pieces_at_the_same_time():
    """steps of two pieces on streams of their own, each asked for before the other's have ended: every one gives what it gives alone"""
    import threading

    cfg = dataclasses.replace(resolve_config("tiny-llama"), hidden_size=2048, n_heads=16, n_kv_heads=4, head_dim=128, ffn_size=5632)
    both = [_setup(cfg, 3, [300 + 10 * i for i in range(n)], seed=n) for n in (3, 20)]
    refs = [_run(*b, True)[0] for b in both]
    outs, errors = [[], []], []
    ready = threading.Barrier(2)

    def steps(i):
        try:
            piece, meta, caches, x = both[i]
            with torch.cuda.device(0), torch.cuda.stream(torch.cuda.Stream()):
                ready.wait(30)
                for _ in range(60):
                    outs[i].append(piece.forward(meta, x_in=x).clone())
                torch.cuda.current_stream().synchronize()
        except BaseException as e:
            errors.append(e)

    threads = [threading.Thread(target=steps, args=(i,)) for i in range(2)]
    for th in threads:
        th.start()
    for th in threads:
        th.join(60)
    assert not errors
    assert all(_gave_up(b[0]) == 0 for b in both)
    assert all(torch.equal(o, refs[i]) for i in range(2) for o in outs[i])
