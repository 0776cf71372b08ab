"""Recurrences over spans with a whole head per block and segments side by side (csrc/lin_span.cu) against a plain 64-bit loop: lengths around
a staged tile (16 tokens) and a segment, sequences without tokens, states that continue, both head widths, every mode it takes, launches
sized for more and longer spans than there are."""
import pytest
import torch

from bee2bee_b200 import ops

# every token rounds a state element twice (2^-24 each) and the decays forget: under 1e-6 for spans of this length
BOUND = 1e-6


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def reference(mode, D, H, G, news, pos0, src, z, zb, hp, beta, aux, qscale, tau, state, slots):
    out, st, t = torch.zeros(sum(news), H, D, dtype=torch.float64, device="cuda"), state.double().clone(), 0
    for s, n in enumerate(news):
        S = st[slots[s]].clone() if pos0[s] > 0 else torch.zeros(H, D, D, dtype=torch.float64, device="cuda")
        for _ in range(n):
            row = src[t].double()
            hq = G if mode == ops.SCAN_SSD else H
            q, k, v = row[:hq * D].view(hq, D), row[hq * D:2 * hq * D].view(hq, D), row[2 * H * D:].view(H, D)
            if mode == ops.SCAN_GLA:
                d, q = torch.sigmoid(z[t].double() + zb.double()).pow(tau).view(H, D), q * qscale
            elif mode == ops.SCAN_MLSTM:
                a = aux[t].double()
                d, k, q = a[:, :1].expand(H, D), k * a[:, 1:2], q * qscale
            elif mode == ops.SCAN_HGRN2:
                low = hp.double().view(H, D)
                d, q = low + (1 - low) * torch.sigmoid(z[t].double() + zb.double()).view(H, D), torch.nn.functional.silu(q)
                k = 1 - d
            else:
                q, k = q.repeat_interleave(H // G, 0), k.repeat_interleave(H // G, 0)
                dt = torch.nn.functional.softplus(beta[t].double() + zb.double())
                d, k, q = torch.exp(-torch.exp(hp.double()) * dt)[:, None].expand(H, D), k * dt[:, None], q * qscale
            S = S * d[:, :, None] + k[:, :, None] * v[:, None, :]
            out[t] = (S * q[:, :, None]).sum(1)
            t += 1
        if n:
            st[slots[s]] = S
    return out.flatten(1), st


def scan_ns(H, D, lens):
    """the measured time of lin_scan, as the rule has it"""
    return max(max(lens) * (285 if D == 128 else 200), sum(lens) * H * (9.0 if D == 128 else 2.3))


def plan_ns(H, D, lens, plan):
    def rounds(blocks):
        r = -(-blocks // 148)
        return r if D == 128 else (0.85 * r if r > 1 else 1)

    token, longest = (420 if D == 128 else 180), max(lens)
    if plan < 0:
        return scan_ns(H, D, lens)
    if plan == 0:
        return rounds(-(-sum(lens) * H // longest)) * longest * token + 2000
    return rounds(H * sum(-(-n // plan) for n in lens)) * plan * token * 1.6 + 10000 + 300 * -(-longest // plan)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("H", [4, 8, 16, 32])
@pytest.mark.parametrize("lens", [[300] * 2, [300] * 3, [1000] * 2, [1000] * 3, [2000] * 2, [2000] * 3, [2000] + [20] * 7, [40] * 2, [100] * 8, [130]])
def test_plan_of_a_bucket(D, H, lens):
    """The launch knows 8 sequences and a power of two of tokens; the plan is that of the true lengths, and no slower than lin_scan."""
    native = pytest.importorskip("bee2bee_b200._C")
    bucket = 1
    while bucket < max(lens):
        bucket *= 2
    n_seqs = 1 if len(lens) == 1 else 8
    plan = native.span_plan(lens, n_seqs, bucket, H, D)
    if max(lens) > 128 and len(lens) > 1:
        assert plan == native.span_plan(lens, len(lens), max(lens), H, D)
    edge = 5000 if (H, D, lens) == (32, 128, [130]) else 1000           # (just above 128 tokens, where lin_scan is not asked)
    assert plan_ns(H, D, lens, plan) <= 1.04 * scan_ns(H, D, lens) + edge
    if (H, D, lens) == (16, 128, [1000, 1000]):
        assert plan_ns(H, D, lens, plan) < 200000


@pytest.mark.gpu
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("mode", [ops.SCAN_GLA, ops.SCAN_MLSTM, ops.SCAN_HGRN2, ops.SCAN_SSD])
@pytest.mark.parametrize("H,news,pos0", [(4, [300], [0]), (4, [257], [7]), (8, [33, 1, 200, 0, 47], [0, 5, 3, 0, 0]), (40, [40] * 9, [0] * 9),
                                         (16, [17, 515], [2, 0])])
@pytest.mark.parametrize("ragged", [False, True])
def test_spans(D, mode, H, news, pos0, ragged):
    run_spans(D, mode, H, news, pos0, len(news), max(news), ragged)


# buckets: sequences without tokens behind the live ones, lengths rounded up; one long span beside short ones.  Up to 128 tokens two kernels
# are launched and one of them leaves (2 x 40: lin_scan stays, 8 x 40 at 16 heads: whole spans); (none live: both leave)
@pytest.mark.gpu
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("H,news,n_seqs,max_q", [(16, [40, 33], 8, 64), (16, [40] * 8, 8, 64), (16, [300, 290], 8, 512), (4, [700, 20, 20, 5], 8, 1024),
                                                 (16, [129], 1, 256), (40, [150] * 5, 32, 256), (16, [0, 0], 8, 64), (8, [0, 0], 8, 512)])
def test_buckets(D, H, news, n_seqs, max_q):
    run_spans(D, ops.SCAN_GLA, H, news, [3 * (i % 2) if n else 0 for i, n in enumerate(news)], n_seqs, max_q, True)


def run_spans(D, mode, H, news, pos0, n_seqs, max_q, ragged):
    g = torch.Generator(device="cuda").manual_seed(D + mode + H)

    def rnd(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    T, n, G = sum(news), len(news), H // 2 if mode == ops.SCAN_SSD else H
    ssd = mode == ops.SCAN_SSD
    idle = [0] * (n_seqs - n)
    src, z, aux = rnd(max(T, 1), 3 * H * D), rnd(max(T, 1), H * D), torch.rand(max(T, 1), H, 4, generator=g, device="cuda")
    zb = rnd(H) - 2 if ssd else rnd(H * D) + 1
    hp = rnd(H) * 0.5 if ssd else torch.rand(H * D, generator=g, device="cuda") * 0.9
    beta = rnd(max(T, 1), H)
    slots = torch.randperm(n + 2, generator=torch.Generator().manual_seed(H))[:n].tolist()
    state = rnd(n + 2, H, D, D)
    start = state.clone()
    out = torch.zeros(T, H * D, device="cuda")
    kw = {ops.SCAN_GLA: dict(z=z, zbias=zb, qscale=D ** -0.5, inv_tau=0.125), ops.SCAN_MLSTM: dict(aux=aux, qscale=D ** -0.5),
          ops.SCAN_HGRN2: dict(z=z, zbias=zb, hparam=hp), ops.SCAN_SSD: dict(zbias=zb, hparam=hp, beta=beta, qscale=D ** -0.5)}[mode]
    ops.lin_scan(mode, src, 0, G * D if ssd else H * D, src, 2 * H * D, state, out, i32([sum(news[:i]) for i in range(n)] + idle), i32(news + idle),
                 i32([a + b for a, b in zip(news, pos0)] + idle), i32(slots + idle), n_seqs, max_q, H, G, D, D, ragged=ragged, **kw)
    want, end = reference(mode, D, H, G, news, pos0, src, z, zb, hp, beta, aux, D ** -0.5, 0.125, start, slots)
    for got, ref in ((out, want), (state, end)):
        assert torch.isfinite(got).all()
        assert float((got.double() - ref).norm()) <= BOUND * float(ref.norm())
    untouched = [i for i in range(n + 2) if i not in [s for s, m in zip(slots, news) if m]]
    assert torch.equal(state[untouched], start[untouched])
