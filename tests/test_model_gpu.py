"""Whole-piece numerics on the GPU: NativePiece (hand-written kernels, paged KV, fused
epilogues, CUDA graphs) against the plain-PyTorch fp32 oracle, for every model family."""
import dataclasses

import pytest
import torch

pytestmark = pytest.mark.gpu

from bee2bee_b200 import ops  # noqa: E402
from bee2bee_b200.engine.core import Engine, SamplingParams  # noqa: E402
from bee2bee_b200.engine.runner import GpuRunner, SeqInit  # noqa: E402
from bee2bee_b200.models.config import resolve_config  # noqa: E402
from bee2bee_b200.models.torch_ref import TorchPiece  # noqa: E402
from bee2bee_b200.models.weights import init_random  # noqa: E402


def _oracle(cfg):
    t = init_random(cfg, range(cfg.n_layers), True, True, device="cuda", dtype=torch.bfloat16, seed=0)
    return TorchPiece(cfg, range(cfg.n_layers), True, True, {k: v.float() for k, v in t.items()})


def _rel_err(a, b):
    return ((a.float() - b.float()).abs().max() / b.float().abs().max().clamp_min(1e-6)).item()


@pytest.mark.parametrize("name", ["tiny-llama", "tiny-mistral", "tiny-gemma2", "tiny-gpt2"])
@pytest.mark.parametrize("graphs", [False, True])
def test_piece_matches_oracle(name, graphs):
    cfg = resolve_config(name)
    torch.manual_seed(0)
    runner = GpuRunner(cfg, "", 0, 1, torch.device("cuda:0"), max_batch=4, groups=1, max_seq_len=512,
                       max_prefill_tokens=128, seed=0, use_graphs=graphs)
    oracle = _oracle(cfg)
    V = cfg.vocab_size
    prompts = [list(range(5, 5 + 150)), [7, 3, 9], list(range(200, 264))]      # chunked (150 > 128), short, page-exact
    seqs = [SeqInit(slot=i, prompt=[t % V for t in p], pages=list(range(1 + 8 * i, 9 + 8 * i)), temperature=0.0,
                    top_p=1.0, repetition_penalty=1.0, seed=i) for i, p in enumerate(prompts)]
    runner.prefill(seqs)
    caches = [oracle.new_cache() for _ in seqs]
    with torch.no_grad():
        ref_last = []
        for s, c in zip(seqs, caches):
            ids = torch.tensor([s.prompt], device="cuda")
            pos = torch.arange(len(s.prompt), device="cuda")[None]
            ref_last.append(oracle.forward(ids, pos, c, logits_last_only=True)[0, -1])
    # the last prefill chunk holds sequences in work-list order; compare through the sampled tokens instead:
    first = runner.tokens[:3].tolist()
    for b, r in enumerate(ref_last):
        top2 = r.topk(2).values
        if (top2[0] - top2[1]).item() > 0.05 * r.abs().max().item():     # only when the arg-max is not a near-tie
            assert first[b] == int(r.argmax()), f"first token mismatch for seq {b}"
    # decode: feed the GPU-sampled token to the oracle, compare full logits every step
    for step in range(5):
        fed = runner.tokens[:3].tolist()
        pos_next = [len(s.prompt) + step for s in seqs]
        runner.decode(1)
        runner.sync()
        got = runner.piece.logits[:3, :V]
        with torch.no_grad():
            for b in range(3):
                ref = oracle.forward(torch.tensor([[fed[b]]], device="cuda"),
                                     torch.tensor([[pos_next[b]]], device="cuda"), caches[b])[0, -1]
                if cfg.final_softcap > 0:
                    g = torch.tanh(got[b] / cfg.final_softcap) * cfg.final_softcap
                else:
                    g = got[b]
                err = _rel_err(g, ref)
                assert err < 6e-2, f"{name} step {step} seq {b}: rel err {err}"
    hist, hpos = runner.read_history()
    assert hpos[:3].tolist() == [6, 6, 6]
    runner.close()


def test_engine_gpu_continuous_batching():
    eng = Engine("tiny-llama", device="cuda", max_batch=4, max_seq_len=256, decode_burst=4)
    sp = SamplingParams(max_new_tokens=12, temperature=0.8, ignore_eos=True, seed=3)
    prompts = [[1, 2, 3, 4, 5], [9, 8, 7], list(range(20, 90)), [4], [5, 6], [7, 8, 9, 10]]   # 6 requests > 4 slots
    outs = eng.generate(prompts, sp)
    assert [len(o) for o in outs] == [12] * 6
    assert all(0 <= t < eng.cfg.vocab_size for o in outs for t in o)
    # determinism: same seeds -> same tokens, independent of the decode burst length.  (The prompt set is kept
    # identical: a 70-token prompt in the prefill chunk selects the tcgen05 attention kernel for the whole chunk,
    # whose bf16 rounding differs from the CUDA-core kernel used for short chunks.)
    eng2 = Engine("tiny-llama", device="cuda", max_batch=4, max_seq_len=256, decode_burst=3)
    outs2 = eng2.generate(prompts, sp)
    assert outs2 == outs
    eng.close()
    eng2.close()


@pytest.mark.parametrize("quant", ["fp8", "mxfp8"])
@pytest.mark.parametrize("name", ["tiny-llama", "tiny-mistral"])
def test_piece_fp8_close_to_oracle(name, quant):
    """W8A8 e4m3 GEMMs (per-row/per-token scales, or MX block scaling): logits stay within fp8 noise of the oracle."""
    cfg = resolve_config(name)
    runner = GpuRunner(cfg, "", 0, 1, torch.device("cuda:0"), max_batch=4, groups=1, max_seq_len=256,
                       max_prefill_tokens=128, seed=0, quant=quant)
    assert runner.piece.fp8 and runner.piece.w["l0.wqkv"].dtype == torch.float8_e4m3fn
    assert runner.piece.mx == (quant == "mxfp8")
    oracle = _oracle(cfg)
    V = cfg.vocab_size
    prompts = [list(range(5, 45)), [7, 3, 9]]
    seqs = [SeqInit(slot=i, prompt=[t % V for t in p], pages=[1 + 4 * i, 2 + 4 * i], temperature=0.0, top_p=1.0,
                    repetition_penalty=1.0, seed=i) for i, p in enumerate(prompts)]
    runner.prefill(seqs)
    caches = [oracle.new_cache() for _ in seqs]
    with torch.no_grad():
        for s, c in zip(seqs, caches):
            oracle.forward(torch.tensor([s.prompt], device="cuda"), torch.arange(len(s.prompt), device="cuda")[None], c)
    for step in range(3):
        fed = runner.tokens[:2].tolist()
        runner.decode(1)
        runner.sync()
        got = runner.piece.logits[:2, :V]
        with torch.no_grad():
            for b in range(2):
                ref = oracle.forward(torch.tensor([[fed[b]]], device="cuda"),
                                     torch.tensor([[len(seqs[b].prompt) + step]], device="cuda"), caches[b])[0, -1]
                err = _rel_err(got[b], ref)
                assert err < 0.2, f"{name} step {step} seq {b}: rel err {err}"
                cos = torch.nn.functional.cosine_similarity(got[b].float(), ref.float(), dim=0).item()
                assert cos > 0.98, cos
    runner.close()


@pytest.mark.parametrize("name", ["tiny-llama", "tiny-mistral"])
def test_block_scaled_prompt_close_to_oracle(name, monkeypatch):
    """block-scaled prompts of more than 64 tokens run on the CTA-pair products: the steps that read their keys and values stay within fp8 noise of the oracle"""
    cfg = resolve_config(name)
    wide, use = [], ops.use_wide
    monkeypatch.setattr(ops, "use_wide", lambda n, t, mx=False: wide.append((t, mx)) or use(n, t, mx))
    runner = GpuRunner(cfg, "", 0, 1, torch.device("cuda:0"), max_batch=4, groups=1, max_seq_len=512, max_prefill_tokens=512, seed=0, quant="mxfp8")
    oracle = _oracle(cfg)
    V = cfg.vocab_size
    prompts = [[(7 * i + 5) % V for i in range(150)], [(11 * i + 3) % V for i in range(61)]]
    seqs = [SeqInit(slot=i, prompt=p, pages=list(range(1 + 8 * i, 9 + 8 * i)), temperature=0.0, top_p=1.0, repetition_penalty=1.0, seed=i)
            for i, p in enumerate(prompts)]
    runner.prefill(seqs)
    assert any(mx and t > 128 for t, mx in wide)
    caches = [oracle.new_cache() for _ in seqs]
    with torch.no_grad():
        for s, c in zip(seqs, caches):
            oracle.forward(torch.tensor([s.prompt], device="cuda"), torch.arange(len(s.prompt), device="cuda")[None], c)
    for step in range(3):
        fed = runner.tokens[:2].tolist()
        runner.decode(1)
        runner.sync()
        got = runner.piece.logits[:2, :V]
        with torch.no_grad():
            for b in range(2):
                ref = oracle.forward(torch.tensor([[fed[b]]], device="cuda"), torch.tensor([[len(seqs[b].prompt) + step]], device="cuda"), caches[b])[0, -1]
                err = _rel_err(got[b], ref)
                assert err < 0.2, f"{name} step {step} seq {b}: rel err {err}"
                assert torch.nn.functional.cosine_similarity(got[b].float(), ref.float(), dim=0).item() > 0.98
    assert ops.native().gemm_wide_gave_up() == 0
    runner.close()


def test_prefill_buckets_know_whether_keys_are_few():
    """GPT-2: chunks of up to 64 tokens have a graph for few keys (the persistent kernel) and one for many; both give what the kernels one by one give."""
    cfg = dataclasses.replace(resolve_config("tiny-gpt2"), hidden_size=256, n_heads=4, n_kv_heads=4, head_dim=64, ffn_size=1024)
    outs = []
    for chain in (True, False):
        r = GpuRunner(cfg, "", 0, 1, torch.device("cuda:0"), max_batch=4, groups=1, max_seq_len=512, max_prefill_tokens=64, seed=0)
        if not chain:
            r.piece._chain = None
            r._pf.clear()
        logits = []
        for slot, L in enumerate((40, 64, 300)):                   # 300 tokens: five chunks, the later ones behind up to 256 keys
            s = SeqInit(slot=slot, prompt=[(3 * i + slot) % cfg.vocab_size for i in range(L)], pages=list(range(1 + 8 * slot, 9 + 8 * slot)),
                        temperature=0.0, top_p=1.0, repetition_penalty=1.0, seed=slot)
            r.prefill([s])
            r.sync()
            logits.append(r.piece.logits[0, :cfg.vocab_size].clone())
        outs.append(torch.stack(logits))
        few = r.piece.span_keys(64)
        assert few == (256 if chain else 0)
        if chain:                                                  # (44 tokens of the last chunk, behind 256 keys: many)
            assert set(r._pf) == {((64, 1, 64, 0), 256), (64, 1, 64, 0)}
            assert r._pf[(64, 1, 64, 0)]["launches"] > r._pf[((64, 1, 64, 0), 256)]["launches"]
        r.close()
    # (roundings of bf16 through two layers and the head; the kernels one by one also round the attention's weights)
    assert _rel_err(outs[0], outs[1]) < 0.02


def test_graph_prefill_matches_eager_prefill():
    """Prefill chunks run as bucketed CUDA graphs (one pinned staging copy + one replay per chunk); results equal
    the eager execution of the same chunk body.  A multi-sequence, multi-chunk batch goes through both as well."""
    cfg = resolve_config("tiny-llama")
    outs = []
    for graphs in (True, False):
        r = GpuRunner(cfg, "", 0, 1, torch.device("cuda:0"), max_batch=4, groups=1, max_seq_len=256,
                      max_prefill_tokens=128, seed=0, use_graphs=graphs)
        toks = []
        for slot, L in enumerate((5, 16, 17, 40)):
            s = SeqInit(slot=slot, prompt=[(3 * i + slot) % cfg.vocab_size for i in range(L)], pages=[1 + 2 * slot, 2 + 2 * slot],
                        temperature=0.0, top_p=1.0, repetition_penalty=1.0, seed=slot)
            r.prefill([s])
            r.sync()                        # prefill only enqueues; the read-back kernel is the synchronisation point
            toks.append(int(r.tokens[slot]))
        assert set(r._pf) == {(16, 1, 16, 0), (32, 1, 32, 0), (64, 1, 64, 0)}
        assert all((st["graph"] is not None) == graphs for st in r._pf.values())
        r.decode(4)
        r.sync()
        hist, hp = r.read_history()
        outs.append((toks, hist[:4, :5].tolist(), hp[:4].tolist()))
        r.close()
    assert outs[0] == outs[1]
    # several sequences per chunk, several chunks, one prompt spanning two chunks
    outs = []
    for graphs in (True, False):
        r = GpuRunner(cfg, "", 0, 1, torch.device("cuda:0"), max_batch=8, groups=1, max_seq_len=256,
                      max_prefill_tokens=64, seed=0, use_graphs=graphs)
        seqs = [SeqInit(slot=b, prompt=[(5 * i + b) % cfg.vocab_size for i in range(L)], pages=[1 + 4 * b + j for j in range(4)],
                        temperature=0.0, top_p=1.0, repetition_penalty=1.0, seed=b)
                for b, L in enumerate((9, 30, 3, 100, 17, 64, 1, 2))]
        r.prefill(seqs)
        r.decode(3)
        outs.append(r.fetch_window([0] * 8, 4).tolist())
        assert r.pf_chunks >= 5
        r.close()
    assert outs[0] == outs[1]


def test_legacy_worker_hf_part_on_the_gpu_data_plane():
    """hf_part_load / hf_part_forward run the layer range on NativePiece and the hop payload stays in
    device memory (hidden_ref: cudaMemcpyPeerAsync of a cudaMalloc buffer, exportable as a CUDA IPC handle) instead of
    the reference's JSON list of fp32 (bee2bee/node.py:270-277).  Result == whole-model oracle."""
    import asyncio
    import json

    from bee2bee_b200 import protocol as P
    from bee2bee_b200.engine.tokenizer import load_tokenizer
    from bee2bee_b200.node import TaskExecutor

    cfg = resolve_config("tiny-llama")
    ex = TaskExecutor(device="cuda")
    a = ex.execute({"kind": P.HF_PART_LOAD, "model_name": "tiny-llama", "start": 0, "end": 2})
    b = ex.execute({"kind": P.HF_PART_LOAD, "model_name": "tiny-llama", "start": 2, "end": 4})
    assert a["backend"] == b["backend"] == "b200-native"
    text = "the mesh hops on the device"
    r1 = ex.execute({"kind": P.HF_PART_FORWARD, "model_id": a["model_id"], "text": text, "keep_on_device": True})
    ref = r1["hidden_ref"]
    assert set(ref) == {"ref", "device", "shape", "ipc"} and len(json.dumps(r1)) < 400       # the frame is ~200 bytes
    r2 = ex.execute({"kind": P.HF_PART_FORWARD, "model_id": b["model_id"], "hidden_ref": ref})
    logits = torch.tensor(r2["hidden"])[0, -1]
    # legacy framing through the same GPU pieces gives the same answer
    l1 = ex.execute({"kind": P.HF_PART_FORWARD, "model_id": a["model_id"], "text": text, "session": "s2", "binary": True})
    l2 = ex.execute({"kind": P.HF_PART_FORWARD, "model_id": b["model_id"], "hidden_b64": l1["hidden_b64"], "session": "s2"})
    assert torch.allclose(torch.tensor(l2["hidden"])[0, -1], logits, atol=1e-3, rtol=1e-3)
    # oracle: all four layers in fp32 on the same random-init weights
    tok = load_tokenizer("tiny-llama", cfg.vocab_size, cfg.eos_token_id, cfg.bos_token_id)
    ids = tok.encode(text)
    t = init_random(cfg, range(cfg.n_layers), True, True, device="cuda", dtype=torch.float32)
    oracle = TorchPiece(cfg, range(cfg.n_layers), True, True, t)
    with torch.no_grad():
        want = oracle.forward(torch.tensor([ids], device="cuda"), torch.arange(len(ids), device="cuda")[None])[0, -1]
    assert _rel_err(logits.cuda(), want) < 0.2
    cos = torch.nn.functional.cosine_similarity(logits.cuda().float(), want.float(), dim=0).item()
    assert cos > 0.98, cos
    # decode continues in the session's paged KV cache (no pos0: the piece tracks the session length)
    r3 = ex.execute({"kind": P.HF_PART_FORWARD, "model_id": a["model_id"], "ids": [int(want.argmax())], "keep_on_device": True})
    r4 = ex.execute({"kind": P.HF_PART_FORWARD, "model_id": b["model_id"], "hidden_ref": r3["hidden_ref"]})
    assert len(r4["hidden"][0][0]) == cfg.vocab_size


def test_prefix_cache_shares_kv_pages_and_skips_prefill():
    """Content-addressed prompt pages.  A second request with the same 150-token prefix re-uses the resident KV
    pages (same physical pages in its block table) and prefills only its suffix; greedy output equals the engine without
    the cache.  The reference re-sends and re-computes the whole transcript every turn."""
    V = resolve_config("tiny-llama").vocab_size
    sys_prompt = [(11 * i + 3) % (V - 8) + 4 for i in range(150)]
    prompts = [sys_prompt + [5, 6, 7], sys_prompt + [9, 10, 11, 12], sys_prompt[:70] + [1, 2]]
    sp = SamplingParams(max_new_tokens=6, temperature=0.0, ignore_eos=True)
    outs, stats = [], []
    for cache in (True, False):
        eng = Engine("tiny-llama", device="cuda:0", max_batch=4, max_seq_len=512, max_prefill_tokens=128, decode_burst=3,
                     prefix_cache=cache)
        res = [eng.generate([p], sp)[0] for p in prompts]            # one after the other: later ones can hit the cache
        res.append(eng.generate(prompts, sp))                         # and all at once (requests of one round do not share)
        outs.append(res)
        stats.append(eng.metrics())
        eng.close()
    assert outs[0] == outs[1]
    on, off = stats
    assert off["prefix_cache_hit_tokens"] == 0
    # second prompt: 2 full pages (128 tokens) of the shared prefix; third: 1 page; the batch round: 2 + 2 + 1 pages
    assert on["prefix_cache_hit_tokens"] == 128 + 64 + (128 + 128 + 64)
    assert on["prefill_tokens"] == off["prefill_tokens"] - on["prefix_cache_hit_tokens"]
    assert on["prefix_cache"]["cached_pages"] >= 2
