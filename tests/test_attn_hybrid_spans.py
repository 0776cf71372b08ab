"""Spans of the hybrid graphs' softmax attention on the tcgen05 kernel (csrc/attention_tc.cu) against 64-bit sums: every head group size, spans around
a query block and a page, cached tokens in front, window edges, kept first keys that reach into and past the window, cap, sink, output rows with
a gap."""
import pytest
import torch

from bee2bee_b200 import ops

pytestmark = pytest.mark.gpu

# The rounding of the queries to bf16 (2^-9 of each channel) moves a score s by up to 2^-9 |s| when the channels' errors agree in sign, and
# |s| reaches 1.5 x 3 sigma here, so a weight is off by up to 4.5 x 2^-9; the weight's own rounding and the result's add 2^-9 each.
BOUND = 6.5 * 2.0 ** -9


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


@pytest.mark.parametrize("H,G,D", [(8, 2, 128), (4, 4, 64), (16, 1, 64), (8, 4, 128), (8, 1, 128)])
@pytest.mark.parametrize("news,ctxs", [([33], [0]), ([300, 1, 0, 65], [0, 100, 0, 63]), ([129, 64], [500, 0])])
@pytest.mark.parametrize("window,keep,cap,sink", [(0, 0, 0.0, False), (100, 10, 30.0, True), (64, 130, 0.0, True), (37, 0, 5.0, False)])
def test_spans(H, G, D, news, ctxs, window, keep, cap, sink):
    g = torch.Generator(device="cuda").manual_seed(H + D + len(news))
    lens = [a + b for a, b in zip(news, ctxs)]
    need = [(n + 63) // 64 for n in lens]
    order = (torch.randperm(sum(need), generator=torch.Generator().manual_seed(2)) + 1).tolist()
    table, at = [], 0
    for n in need:
        table.append(order[at:at + n] + [0] * (max(need) - n))
        at += n
    k, v = (torch.randn(sum(need) + 1, 64, G, D, generator=g, device="cuda").bfloat16() for _ in "kv")
    T = sum(news)
    q = torch.randn(T, H * D, generator=g, device="cuda") * 1.5
    sk = torch.randn(H, generator=g, device="cuda") if sink else None
    wide = torch.zeros(T, H * D + 8, device="cuda", dtype=torch.bfloat16)
    out = wide[:, :H * D]
    ops.softmax_attention(q, k, v, out, i32(table), i32([sum(news[:i]) for i in range(len(news))]), i32(news), i32(lens), len(news), max(news), H,
                          G, D, D, window, D ** -0.5, softcap=cap, keep_first=keep, sink=sk)
    at = 0
    for s, (n, L) in enumerate(zip(news, lens)):
        pos = torch.arange(L, device="cuda")
        rows = i32(table)[s].long()[pos // 64] * 64 + pos % 64
        kk, vv = (c.view(-1, G, D)[rows].double().repeat_interleave(H // G, 1) for c in (k, v))
        sc = torch.einsum("qhd,khd->hqk", q[at:at + n].double().view(n, H, D) * D ** -0.5, kk)
        if cap:
            sc = cap * torch.tanh(sc / cap)
        qp = torch.arange(L - n, L, device="cuda")[:, None]
        ok = pos[None] <= qp
        if window:
            ok &= (pos[None] > qp - window) | (pos[None] < keep)
        sc = sc.masked_fill(~ok, float("-inf"))
        if sink:
            sc = torch.cat([sc, sk.double()[:, None, None].expand(H, n, 1)], 2)
        ref = torch.einsum("hqk,khd->qhd", sc.softmax(-1)[:, :, :L], vv).reshape(n, H * D)
        if n:
            assert float((out[at:at + n].double() - ref).norm() / ref.norm()) < BOUND
        at += n
    assert float(wide[:, H * D:].abs().max()) == 0.0


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("cap", [3.0, 9.0, 30.0, 1000.0])
def test_cap_of_small_and_large_scores(D, cap):
    """scores below half the cap (a polynomial) and rows far above it (exponentials), in warps of their own and beside one another; an infinite score; what
    lies behind the last key is not a number and stays out"""
    g = torch.Generator(device="cuda").manual_seed(5)
    n, H = 150, 2
    k, v = (torch.randn(4, 64, 1, D, generator=g, device="cuda").bfloat16() for _ in "kv")
    k[3, n - 128:] = float("nan")
    v[3, n - 128:] = 0.0
    q = torch.randn(n, H * D, generator=g, device="cuda")
    q[40:43] *= 30.0                                         # (beside small rows)
    q[64:96] *= 30.0                                         # (a warp's rows)
    q[20, :D] = 0.0
    q[20, 0] = 1e38                                          # (infinite as a product with a key: plus or minus the cap)
    out = torch.zeros(n, H * D, device="cuda", dtype=torch.bfloat16)
    scale = D ** -0.5
    ops.softmax_attention(q, k, v, out, i32([[1, 2, 3]]), i32([0]), i32([n]), i32([n]), 1, n, H, 1, D, D, 0, scale, softcap=cap)
    kk, vv = (c.view(-1, D)[64:64 + n].double() for c in (k, v))
    sc = cap * torch.tanh(torch.einsum("qhd,kd->hqk", (q * scale).bfloat16().double().view(n, H, D), kk) / cap)
    ref = torch.einsum("hqk,kd->qhd", sc.masked_fill(~torch.ones(n, n, device="cuda", dtype=torch.bool).tril(), float("-inf")).softmax(-1), vv).reshape(n, H * D)
    # (the queries are rounded on both sides.  A score in fp32 is off by sqrt(D) 2^-24 of its largest products, up to 150 here, less than 2^-12 of a weight;
    # the weights' roundings to bf16 and the result's are 2^-9 each)
    assert float((out.double() - ref).norm() / ref.norm()) < 2.5 * 2.0 ** -9
    assert bool(torch.isfinite(out).all())
