"""What the framework is timed on: the layers, blocks and whole calls that serving a model runs on one GPU.

Kinds of cases (sizes are those of the presets in ``bee2bee_b200/models/config.py`` and of ``bench.py``'s configurations):

* ``layer``   decoder layers of a dense model through ``NativePiece.forward``: prompts (``new`` > 1) or one decode step
              (``new`` = 1), on an empty cache or behind ``ctx`` cached tokens.  As in serving (``GpuRunner``), the call is
              recorded once into a CUDA graph and replayed per step.
* ``model``   a whole GPT-2 sized model, token ids in, logits out, through the same call.
* ``attention``  decode attention over a long paged cache (``ops.attention``).
* ``head``    final norm, head matrix and sampler of a decode step (``NativePiece.forward`` of the last piece, ``ops.sample``).
* ``scan``    gated linear recurrences of the hybrid families over prompts (``ops.lin_scan``).
* ``window``  softmax attention of the hybrid families over prompts: window with kept first keys, capped scores, a sink
              (``ops.softmax_attention``).
"""
import dataclasses
import math

import torch

from bee2bee_b200 import ops
from bee2bee_b200.models.config import resolve_config
from bee2bee_b200.models.native import BatchMeta, NativePiece

PAGE = 64                 # tokens per page of the key / value cache
SMS = 148


# ------------------------------------------------------------------------------------------------------------ cases
def listed():
    def layer(name, model, layers, seqs, new, ctx=0, quant="bf16"):
        return {"name": name, "kind": "layer", "model": model, "layers": layers, "seqs": seqs, "new": new, "ctx": ctx, "quant": quant}

    return [
        # one user, one token: the latency of a decode step (bench.py --config 2)
        layer("decode-1", "llama-3-8b", 2, 1, 1, 700),
        # the headline: a decode step of 32 sequences (bench.py)
        layer("decode-32", "llama-3-8b", 2, 32, 1, 500),
        # the same in block-scaled fp8 (bench.py --config 3)
        layer("decode-32-mxfp8", "llama-3-8b", 2, 32, 1, 500, "mxfp8"),
        # 32 short prompts admitted together (the prefill of the headline's end-to-end run)
        dict(layer("prompts-32x16", "llama-3-8b", 1, 32, 16), even=True),
        # a few chat turns of odd lengths behind a cached prefix (zephyr, bench.py --config 5)
        layer("chat-5x333", "zephyr-7b-beta", 1, 5, 333, 410),
        # one long prompt: a full chunk of prefill
        layer("prompt-4096", "llama-3-8b", 1, 1, 4096),
        # a long prompt on Gemma-2 (bench.py --config 4): 256-wide heads, capped scores, a windowed and a full layer
        layer("prompt-gemma-4096", "gemma-2-2b", 2, 1, 4096),
        # decode attention when contexts have grown long
        {"name": "context-32x8k", "kind": "attention", "seqs": 32, "ctx": 8100, "n_q": 32, "n_kv": 8, "dim": 128},
        # what turns hidden states into tokens in the headline's decode step
        {"name": "head-32", "kind": "head", "seqs": 32, "hidden": 4096, "vocab": 128256},
        # the smallest model of the reference: a short prompt through all of distilgpt2
        {"name": "distilgpt2-19", "kind": "model", "model": "distilgpt2", "seqs": 1, "new": 19},
        # a prompt chunk through a recurrent layer of the hybrid families at width 2048
        {"name": "scan-2048", "kind": "scan", "mode": "gla", "seqs": 1, "new": 2048, "heads": 16, "dim": 128},
        # a prompt chunk through their windowed attention
        {"name": "window-2048", "kind": "window", "seqs": 1, "new": 2048, "heads": 16, "kv_heads": 4, "dim": 128, "window": 1024},
    ]


def _between(rng, lo, hi):
    """an integer, spread evenly over the logarithm"""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "prefill", "attention", "head", "model", "scan", "scan", "window"])
    if kind == "decode":
        return {"kind": "layer", "model": rng.choice(["llama-3-8b", "zephyr-7b-beta", "gemma-2-2b"]), "layers": 2,
                "seqs": _between(rng, 1, 64), "new": 1, "ctx": _between(rng, 30, 2000), "quant": "bf16"}
    if kind == "prefill":
        model = rng.choice(["llama-3-8b", "zephyr-7b-beta", "gemma-2-2b"])
        seqs = _between(rng, 1, 32)
        quant = rng.choice(["bf16", "bf16", "mxfp8"]) if model != "gemma-2-2b" else "bf16"
        return {"kind": "layer", "model": model, "layers": 1, "seqs": seqs, "new": max(2, _between(rng, 70, 3500) // seqs),
                "ctx": rng.choice([0, 0, _between(rng, 20, 1200)]), "quant": quant}
    if kind == "attention":
        n_q, n_kv, dim = rng.choice([(32, 8, 128), (32, 8, 128), (8, 4, 256), (12, 12, 64)])
        return {"kind": "attention", "seqs": _between(rng, 2, 32), "ctx": _between(rng, 300, 8000), "n_q": n_q, "n_kv": n_kv, "dim": dim}
    if kind == "head":
        hidden, vocab = rng.choice([(4096, 128256), (4096, 32000), (2304, 256000)])
        return {"kind": "head", "seqs": _between(rng, 1, 32), "hidden": hidden, "vocab": vocab}
    if kind == "model":
        return {"kind": "model", "model": rng.choice(["distilgpt2", "gpt2"]), "seqs": _between(rng, 1, 4), "new": _between(rng, 5, 240)}
    if kind == "scan":
        seqs = _between(rng, 1, 8)
        return {"kind": "scan", "mode": rng.choice(["gla", "hgrn2"]), "seqs": seqs, "new": max(40, _between(rng, 150, 2048) // seqs),
                "heads": rng.choice([8, 16, 32]), "dim": rng.choice([64, 128])}
    heads = rng.choice([8, 16, 32])
    seqs = _between(rng, 1, 6)
    return {"kind": "window", "seqs": seqs, "new": max(40, _between(rng, 200, 2048) // seqs), "heads": heads, "kv_heads": heads // 4,
            "dim": rng.choice([64, 128]), "window": rng.choice([0, 256, 1024])}


# ------------------------------------------------------------------------------------------------- sizes of a case
def _lengths(case):
    """new tokens and cached tokens of every sequence: the longest is the case's, the others are shorter in odd steps"""
    n, c, s = case["new"], case.get("ctx", 0), case["seqs"]
    if case.get("even"):
        return [n] * s, [c] * s
    news = [max(1, n - (7 * i) % (n // 3 + 1)) for i in range(s)]
    ctxs = [max(0, c - (13 * i) % (c // 2 + 1)) for i in range(s)]
    return news, ctxs


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(g, *shape, std=1.0, dtype=torch.bfloat16):
    return torch.randn(*shape, generator=g, device="cuda", dtype=dtype).mul_(std)


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def _pages(g, lens):
    """block table of sequences whose pages lie scattered in the cache, and the number of pages (page 0 is unused)"""
    need = [(n + PAGE - 1) // PAGE for n in lens]
    order = (torch.randperm(sum(need), generator=g, device="cuda") + 1).cpu().tolist()
    table, at = [], 0
    for n in need:
        table.append(order[at:at + n] + [0] * (max(need) - n))
        at += n
    return table, sum(need) + 1


def _span_meta(table, news, ctxs, ids=None, last=None):
    pos = [c + i for n, c in zip(news, ctxs) for i in range(n)]
    slots = [table[s][(c + i) // PAGE] * PAGE + (c + i) % PAGE for s, (n, c) in enumerate(zip(news, ctxs)) for i in range(n)]
    starts, at = [], 0
    for n in news:
        starts.append(at)
        at += n
    return BatchMeta(ids=ids, positions=_i32(pos), slots=_i32(slots), q_start=_i32(starts), q_len=_i32(news),
                     kv_len=_i32([n + c for n, c in zip(news, ctxs)]), block_table=_i32(table), n_tokens=at, n_seqs=len(news),
                     max_q=max(news), last_idx=None if last is None else _i32([a + n - 1 for a, n in zip(starts, news)]))


# --------------------------------------------------------------------------------------------------- inputs by kind
def _weights(cfg, layers, g, whole=False):
    H, F, Q, KV = cfg.hidden_size, cfg.ffn_size, cfg.q_dim, cfg.kv_dim
    t = {}
    base = 0.0 if cfg.gemma_norm else 1.0

    def norm(n):
        return _randn(g, n, std=0.1) + base

    for l in range(layers):
        p = f"l{l}."
        for name, rows, cols in (("wq", Q, H), ("wk", KV, H), ("wv", KV, H), ("wo", H, Q), ("w_up", F, H), ("w_down", H, F)):
            t[p + name] = _randn(g, rows, cols, std=cols ** -0.5)
        if cfg.glu:
            t[p + "w_gate"] = _randn(g, F, H, std=H ** -0.5)
        for name in ("ln1_w", "ln2_w") + (("post_attn_w", "post_ffn_w") if cfg.post_norms else ()):
            t[p + name] = norm(H)
        if cfg.norm == "ln":
            t[p + "ln1_b"], t[p + "ln2_b"] = _randn(g, H, std=0.1), _randn(g, H, std=0.1)
        if cfg.bias:
            for name, n in (("bq", Q), ("bk", KV), ("bv", KV), ("bo", H), ("b_up", F), ("b_down", H)):
                t[p + name] = _randn(g, n, std=0.1)
    if whole:
        t["embed"] = _randn(g, cfg.vocab_size, H, std=0.05)
        t["pos_embed"] = _randn(g, cfg.max_position, H, std=0.05)
        t["final_norm_w"], t["final_norm_b"] = norm(H), _randn(g, H, std=0.1)
    return t


def _inputs_layer(case, seed):
    g = _generator(seed)
    cfg = resolve_config(case["model"])
    news, ctxs = _lengths(case)
    table, n_pages = _pages(g, [n + c for n, c in zip(news, ctxs)])
    t = _weights(cfg, case["layers"], g)
    caches = []
    for _ in range(case["layers"]):
        shape = (n_pages, PAGE, cfg.n_kv_heads, cfg.head_dim)
        full = any(ctxs)
        caches.append(tuple(_randn(g, *shape) if full else torch.zeros(shape, device="cuda", dtype=torch.bfloat16) for _ in "kv"))
    x = _randn(g, sum(news), cfg.hidden_size)
    return cfg, news, ctxs, table, n_pages, t, caches, x


def _record(call):
    """the call, warmed up, as a CUDA graph (what serving keeps per batch shape)"""
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        call()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            out = call()
    torch.cuda.current_stream().wait_stream(stream)
    return graph, out


def _prepare_layer(case, seed):
    cfg, news, ctxs, table, n_pages, t, caches, x = _inputs_layer(case, seed)
    ops.native().init_kernels(torch.cuda.current_device())
    piece = NativePiece(cfg, range(case["layers"]), False, False, t, torch.device("cuda", torch.cuda.current_device()), sum(news),
                        len(news), n_pages, quant=case["quant"])
    del t
    for l, (k, v) in enumerate(caches):
        piece.k_cache[l].copy_(k)
        piece.v_cache[l].copy_(v)
    meta = _span_meta(table, news, ctxs)
    if meta.max_q == 1 and max(ctxs) + 1 > 1024:       # few sequences with a long context: the keys are split (GpuRunner's rule)
        meta.splits = max(1, min(piece.max_splits, SMS // (len(news) * cfg.n_kv_heads)))
    graph, out = _record(lambda: piece.forward(meta, x_in=x))
    return {"kind": "layer", "graph": graph, "keep": (piece, meta, x),
            "out": {"x": out, "k": [piece.k_cache[l] for l in range(case["layers"])], "v": [piece.v_cache[l] for l in range(case["layers"])]}}


def _inputs_model(case, seed):
    g = _generator(seed)
    cfg = resolve_config(case["model"])
    news, ctxs = _lengths(case)
    table, n_pages = _pages(g, news)
    t = _weights(cfg, cfg.n_layers, g, whole=True)
    ids = torch.randint(0, cfg.vocab_size, (sum(news),), generator=g, device="cuda", dtype=torch.int32)
    return cfg, news, ctxs, table, n_pages, t, ids


def _prepare_model(case, seed):
    cfg, news, ctxs, table, n_pages, t, ids = _inputs_model(case, seed)
    ops.native().init_kernels(torch.cuda.current_device())
    piece = NativePiece(cfg, range(cfg.n_layers), True, True, t, torch.device("cuda", torch.cuda.current_device()), max(16, sum(news)),
                        len(news), n_pages)
    meta = _span_meta(table, news, ctxs, ids=ids, last=True)
    graph, out = _record(lambda: piece.forward(meta))
    return {"kind": "model", "graph": graph, "keep": (piece, meta), "out": out}


def _inputs_attention(case, seed):
    g = _generator(seed)
    _, ctxs = _lengths(dict(case, new=1))
    kv_lens = [c + 1 for c in ctxs]
    table, n_pages = _pages(g, kv_lens)
    shape = (n_pages, PAGE, case["n_kv"], case["dim"])
    k, v = _randn(g, *shape), _randn(g, *shape)
    q = _randn(g, case["seqs"], case["n_q"] * case["dim"], std=2.0 * case["dim"] ** -0.5)
    return kv_lens, table, k, v, q


def _prepare_attention(case, seed):
    kv_lens, table, k, v, q = _inputs_attention(case, seed)
    S = case["seqs"]
    splits = max(1, min(16, SMS // (S * case["n_kv"]))) if max(kv_lens) > 1024 else 1       # GpuRunner's rule
    rows = max(4, (case["n_q"] // case["n_kv"] + 3) // 4 * 4)
    ws = torch.zeros(S * case["n_kv"] * 16 * rows * (case["dim"] + 2), device="cuda")
    return {"kind": "attention", "args": (q, k, v, torch.zeros_like(q), _i32(table), _i32(list(range(S))), _i32([1] * S), _i32(kv_lens)),
            "opts": dict(max_q=1, n_q=case["n_q"], n_kv=case["n_kv"], head_dim=case["dim"], splits=splits, ws=ws)}


def _inputs_head(case, seed):
    g = _generator(seed)
    H, V = case["hidden"], case["vocab"]
    t = {"lm_head": _randn(g, V, H, std=2.0 * H ** -0.5), "final_norm_w": _randn(g, H, std=0.1) + 1.0}
    return t, _randn(g, case["seqs"], H)


def _prepare_head(case, seed):
    t, x = _inputs_head(case, seed)
    S, V = case["seqs"], case["vocab"]
    cfg = dataclasses.replace(resolve_config("llama-3-8b"), hidden_size=case["hidden"], vocab_size=V)
    ops.native().init_kernels(torch.cuda.current_device())
    piece = NativePiece(cfg, [], False, True, t, torch.device("cuda", torch.cuda.current_device()), max(16, S), S, 1)
    meta = BatchMeta(ids=None, positions=None, slots=None, q_start=None, q_len=None, kv_len=None, block_table=None, n_tokens=S, n_seqs=S,
                     max_q=1)
    full = lambda v: torch.full((S,), v, device="cuda")  # noqa: E731
    opts = dict(seen=torch.zeros((S, (V + 31) // 32), device="cuda", dtype=torch.int32), temperature=full(0.7), top_p=full(0.95),
                rep_penalty=full(1.15), seeds=_i32([1000 + i for i in range(S)]), step=_i32([seed % 1000]), vocab=V)
    return {"kind": "head", "piece": piece, "meta": meta, "x": x, "tokens": _i32([0] * S), "opts": opts}


def _inputs_scan(case, seed):
    g = _generator(seed)
    news, _ = _lengths(case)
    H, D, T = case["heads"], case["dim"], sum(news)
    f32 = torch.float32
    gla = case["mode"] == "gla"
    d = {"proj": _randn(g, T, 3 * H * D, dtype=f32), "z": _randn(g, T, H * D, dtype=f32), "news": news}
    d["zbias"] = _randn(g, H * D, std=0.5, dtype=f32) + (2.0 if gla else 1.0)
    d["lower"] = None if gla else torch.rand(H * D, generator=g, device="cuda") * 0.8
    return d


def _prepare_scan(case, seed):
    d = _inputs_scan(case, seed)
    H, D, news = case["heads"], case["dim"], d["news"]
    S, T = len(news), sum(news)
    starts = [sum(news[:i]) for i in range(S)]
    gla = case["mode"] == "gla"
    state = torch.zeros((S, H, D, D), device="cuda")
    out = torch.zeros((T, H * D), device="cuda")
    args = (ops.SCAN_GLA if gla else ops.SCAN_HGRN2, d["proj"], 0, H * D if gla else 0, d["proj"], 2 * H * D, state, out, _i32(starts),
            _i32(news), _i32(news), _i32(list(range(S))), S, max(news), H, H, D, D)
    opts = dict(z=d["z"], zbias=d["zbias"], hparam=d["lower"])
    if gla:
        opts.update(qscale=D ** -0.5, inv_tau=1.0 / 8.0)
    return {"kind": "scan", "args": args, "opts": opts, "out": {"o": out, "state": state}}


def _inputs_window(case, seed):
    g = _generator(seed)
    news, ctxs = _lengths(case)
    H, G, D = case["heads"], case["kv_heads"], case["dim"]
    table, n_pages = _pages(g, news)
    k, v = _randn(g, n_pages, PAGE, G, D), _randn(g, n_pages, PAGE, G, D)
    q = _randn(g, sum(news), H * D, std=1.5, dtype=torch.float32)
    return news, table, k, v, q, _randn(g, H, dtype=torch.float32)


def _prepare_window(case, seed):
    news, table, k, v, q, sink = _inputs_window(case, seed)
    H, G, D, S = case["heads"], case["kv_heads"], case["dim"], len(news)
    starts = [sum(news[:i]) for i in range(S)]
    out = torch.zeros((sum(news), H * D), device="cuda", dtype=torch.bfloat16)
    args = (q, k, v, out, _i32(table), _i32(starts), _i32(news), _i32(news), S, max(news), H, G, D, D, case["window"], D ** -0.5)
    return {"kind": "window", "args": args, "opts": dict(softcap=30.0, keep_first=64 if case["window"] else 0, sink=sink), "out": out}


def prepare(case, seed):
    return {"layer": _prepare_layer, "model": _prepare_model, "attention": _prepare_attention, "head": _prepare_head,
            "scan": _prepare_scan, "window": _prepare_window}[case["kind"]](case, seed)


def run(state):
    kind = state["kind"]
    if kind in ("layer", "model"):
        state["graph"].replay()
        return state["out"]
    if kind == "attention":
        return ops.attention(*state["args"], **state["opts"])
    if kind == "head":
        logits = state["piece"].forward(state["meta"], x_in=state["x"])
        ops.sample(logits, state["tokens"], **state["opts"])
        return {"logits": logits, "tokens": state["tokens"]}
    if kind == "scan":
        ops.lin_scan(*state["args"], **state["opts"])
        return state["out"]
    ops.softmax_attention(*state["args"], **state["opts"])
    return state["out"]


# ------------------------------------------------------------------------------------------------------- 64-bit values
def _norm64(cfg, t, name, x):
    w = t[name + "_w"].double()
    if cfg.norm == "ln":
        return torch.nn.functional.layer_norm(x, (x.shape[-1],), w, t[name + "_b"].double(), cfg.norm_eps)
    return x / (x.pow(2).mean(-1, keepdim=True) + cfg.norm_eps).sqrt() * (w + 1.0 if cfg.gemma_norm else w)


def _attend64(q, k, v, pos, window=0, softcap=0.0, keep_first=0, sink=None):
    """q [T, heads, D] (scaled), k / v [keys, kv heads, D], query positions [T] -> [T, heads, D]"""
    T, H, _ = q.shape
    per = H // k.shape[1]
    at = torch.arange(k.shape[0], device=q.device)[None, :]
    ok = at <= pos[:, None]
    if window:
        ok &= (at > pos[:, None] - window) | (at < keep_first)
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    for h in range(H):
        s = q[:, h] @ k[:, h // per].t()
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(~ok, float("-inf"))
        m = s.amax(-1, keepdim=True)
        e = (s - m).exp()
        den = e.sum(-1, keepdim=True)
        if sink is not None:
            den = den + (sink[h] - m).exp()
        out[:, h] = (e / den) @ v[:, h // per]
    return out


def _layers64(cfg, t, layers, x, news, ctxs, table, caches):
    """x [T, H] through the layers; ``caches`` [(k, v)] in 64 bits are filled in, keys in the cache's order of channels"""
    D, Hq, G = cfg.head_dim, cfg.n_heads, cfg.n_kv_heads
    rows = torch.tensor([s for s, n in enumerate(news) for _ in range(n)], device="cuda")
    pos = torch.tensor([c + i for n, c in zip(news, ctxs) for i in range(n)], device="cuda")
    tab = torch.tensor(table, device="cuda")
    slots = tab[rows, pos // PAGE] * PAGE + pos % PAGE
    turn = cfg.rope_theta > 0
    if turn:
        ang = pos.double()[:, None] * cfg.rope_theta ** (-torch.arange(0, D, 2, device="cuda", dtype=torch.float64) / D)
        cos, sin = ang.cos()[:, None], ang.sin()[:, None]

    def rotated(y):               # pairs (i, i + D / 2) of the model, side by side as the cache holds them
        a, b = y[..., :D // 2], y[..., D // 2:]
        return torch.stack([a * cos - b * sin, b * cos + a * sin], -1).flatten(-2)

    def mul(name, y, bias):
        r = y @ t[name].double().t()
        return r + t[bias].double() if bias in t else r

    for l in range(layers):
        p = f"l{l}."
        kc, vc = (c.view(-1, G, D) for c in caches[l])
        h = _norm64(cfg, t, p + "ln1", x)
        q, k, v = (mul(p + "w" + n, h, p + "b" + n).view(len(x), -1, D) for n in "qkv")
        if turn:
            q, k = rotated(q), rotated(k)
        kc[slots], vc[slots] = k, v
        a = torch.empty(len(x), Hq, D, dtype=torch.float64, device="cuda")
        at = 0
        for s, (n, c) in enumerate(zip(news, ctxs)):
            keys = torch.arange(n + c, device="cuda")
            keys = tab[s][keys // PAGE] * PAGE + keys % PAGE
            a[at:at + n] = _attend64(q[at:at + n] * cfg.softmax_scale, kc[keys], vc[keys], pos[at:at + n], cfg.layer_window(l),
                                     cfg.attn_softcap)
            at += n
        o = mul(p + "wo", a.flatten(1), p + "bo")
        x = x + (_norm64(cfg, t, p + "post_attn", o) if cfg.post_norms else o)
        h = _norm64(cfg, t, p + "ln2", x)
        if cfg.glu:
            gate = mul(p + "w_gate", h, "")
            gate = torch.nn.functional.gelu(gate, approximate="tanh") if cfg.act == "gelu_tanh" else torch.nn.functional.silu(gate)
            m = mul(p + "w_down", gate * mul(p + "w_up", h, ""), "")
        else:
            m = mul(p + "w_down", torch.nn.functional.gelu(mul(p + "w_up", h, p + "b_up"), approximate="tanh"), p + "b_down")
        x = x + (_norm64(cfg, t, p + "post_ffn", m) if cfg.post_norms else m)
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "layer":
        cfg, news, ctxs, table, _, t, caches, x = _inputs_layer(case, seed)
        caches = [tuple(c.double() for c in kv) for kv in caches]
        x = _layers64(cfg, t, case["layers"], x.double(), news, ctxs, table, caches)
        return {"x": x, "k": [k for k, _ in caches], "v": [v for _, v in caches]}
    if kind == "model":
        cfg, news, ctxs, table, n_pages, t, ids = _inputs_model(case, seed)
        shape = (n_pages, PAGE, cfg.n_kv_heads, cfg.head_dim)
        caches = [tuple(torch.zeros(shape, device="cuda", dtype=torch.float64) for _ in "kv") for _ in range(cfg.n_layers)]
        pos = torch.tensor([i for n in news for i in range(n)], device="cuda")
        x = t["embed"][ids.long()].double() + t["pos_embed"][pos].double()
        x = _layers64(cfg, t, cfg.n_layers, x, news, ctxs, table, caches)
        ends = torch.tensor(news, device="cuda").cumsum(0) - 1
        logits = _norm64(cfg, t, "final_norm", x[ends]) @ t["embed"].double().t()
        return torch.nn.functional.pad(logits, (0, -cfg.vocab_size % 128))       # the head's rows come in blocks of 128
    if kind == "attention":
        kv_lens, table, k, v, q = _inputs_attention(case, seed)
        k, v = (c.view(-1, case["n_kv"], case["dim"]).double() for c in (k, v))
        tab = torch.tensor(table, device="cuda")
        out = torch.empty(q.shape, device="cuda", dtype=torch.float64)
        for s, n in enumerate(kv_lens):
            keys = torch.arange(n, device="cuda")
            keys = tab[s][keys // PAGE] * PAGE + keys % PAGE
            out[s] = _attend64(q[s].double().view(1, case["n_q"], case["dim"]), k[keys], v[keys], torch.tensor([n - 1], device="cuda")).flatten()
        return out
    if kind == "head":
        t, x = _inputs_head(case, seed)
        cfg = resolve_config("llama-3-8b")
        return {"logits": _norm64(cfg, t, "final_norm", x.double()) @ t["lm_head"].double().t(), "tokens": None}
    if kind == "scan":
        d = _inputs_scan(case, seed)
        H, D, news = case["heads"], case["dim"], d["news"]
        q, k, v = (y.double().view(-1, H, D) for y in d["proj"].split(H * D, 1))
        gate = (d["z"].double() + d["zbias"].double()).sigmoid().view(-1, H, D)
        if case["mode"] == "gla":
            q, decay = q * D ** -0.5, gate ** 0.125
        else:
            low = d["lower"].double().view(H, D)
            q, decay = torch.nn.functional.silu(q), low + (1.0 - low) * gate
            k = 1.0 - decay
        starts = torch.tensor([sum(news[:i]) for i in range(len(news))], device="cuda")
        state = torch.zeros(len(news), H, D, D, device="cuda", dtype=torch.float64)
        out = torch.zeros(sum(news), H, D, device="cuda", dtype=torch.float64)
        by_length = sorted(range(len(news)), key=lambda s: -news[s])
        for i in range(max(news)):
            live = torch.tensor([s for s in by_length if news[s] > i], device="cuda")
            r = starts[live] + i
            st = state[live] * decay[r][..., None] + k[r][..., None] * v[r][:, :, None, :]
            state[live] = st
            out[r] = (st * q[r][..., None]).sum(2)
        return {"o": out.flatten(1), "state": state}
    news, table, k, v, q, sink = _inputs_window(case, seed)
    G, D = case["kv_heads"], case["dim"]
    k, v = (c.view(-1, G, D).double() for c in (k, v))
    tab = torch.tensor(table, device="cuda")
    q = q.double().view(-1, case["heads"], D) * D ** -0.5
    out, at = torch.empty_like(q), 0
    for s, n in enumerate(news):
        keys = torch.arange(n, device="cuda")
        pos = keys.clone()
        keys = tab[s][keys // PAGE] * PAGE + keys % PAGE
        out[at:at + n] = _attend64(q[at:at + n], k[keys], v[keys], pos, case["window"], 30.0, 64 if case["window"] else 0, sink.double())
        at += n
    return out.flatten(1)


# --------------------------------------------------------------------------------------------- cost and tolerance
def _pairs(news, ctxs, window, keep=0):
    """(query, key) pairs of causal attention"""
    n = 0
    for a, c in zip(news, ctxs):
        for i in range(a):
            seen = c + i + 1
            n += seen if not window or seen <= window else min(seen, window + keep)
    return n


def work(case):
    kind = case["kind"]
    if kind in ("layer", "model"):
        cfg = resolve_config(case["model"])
        news, ctxs = _lengths(case)
        T, layers = sum(news), case["layers"] if kind == "layer" else cfg.n_layers
        params = cfg.hidden_size * (2 * cfg.q_dim + 2 * cfg.kv_dim) + (3 if cfg.glu else 2) * cfg.hidden_size * cfg.ffn_size
        size = 1.03 if case.get("quant") == "mxfp8" else 2            # a byte and a scale per 32 of them
        nbytes = layers * (params * size + 2 * 2 * cfg.kv_dim * (sum(ctxs) + T)) + 2 * 2 * T * cfg.hidden_size
        flops = layers * 2.0 * params * T + sum(4.0 * cfg.q_dim * _pairs(news, ctxs, cfg.layer_window(l)) for l in range(layers))
        if kind == "model":
            nbytes += 2 * cfg.vocab_size * cfg.hidden_size + 4 * len(news) * cfg.vocab_size
            flops += 2.0 * len(news) * cfg.vocab_size * cfg.hidden_size
        return {"bytes": nbytes, "flops": flops}
    if kind == "attention":
        keys = sum(c + 1 for c in _lengths(dict(case, new=1))[1])
        return {"bytes": 4 * keys * case["n_kv"] * case["dim"] + 4 * case["seqs"] * case["n_q"] * case["dim"],
                "flops": 4.0 * keys * case["n_q"] * case["dim"]}
    if kind == "head":
        S, H, V = case["seqs"], case["hidden"], case["vocab"]
        return {"bytes": 2 * V * H + 2 * S * H + 4 * S * V, "flops": 2.0 * S * V * H}
    T = sum(_lengths(case)[0])
    H, D = case["heads"], case["dim"]
    if kind == "scan":       # query, key (hgrn2: none), value and gate rows in, output rows and final states out
        rows = 5 if case["mode"] == "gla" else 4
        return {"bytes": 4 * (rows * T * H * D + case["seqs"] * H * D * D), "flops": 5.0 * T * H * D * D}
    G, keep = case["kv_heads"], 64 if case["window"] else 0
    news, ctxs = _lengths(case)
    return {"bytes": 6 * T * H * D + 4 * T * G * D, "flops": 4.0 * H * D * _pairs(news, ctxs, case["window"], keep)}


def tolerance(case):
    kind = case["kind"]
    if kind == "layer":
        return {"rel": 0.05} if case["quant"] == "mxfp8" else {"rel": 0.01}
    if kind == "head":
        return {"rel": 0.01, "differ": 0.1}
    if kind == "scan":
        return {"rel": 1e-5}
    return {"rel": 0.02}
