"""Recurrences over spans with a whole head per block and segments side by side (csrc/lin_span.cu) against a plain 64-bit loop: lengths around
a staged tile (16 tokens) and a segment, sequences without tokens, states that continue, both head widths, every mode it takes."""
import pytest
import torch

from bee2bee_b200 import ops

pytestmark = pytest.mark.gpu

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


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("mode", [ops.SCAN_GLA, ops.SCAN_MLSTM, ops.SCAN_HGRN2, ops.SCAN_SSD])
@pytest.mark.parametrize("H,news,pos0", [(4, [300], [0]), (4, [257], [7]), (8, [33, 1, 200, 0, 47], [0, 5, 3, 0, 0]), (40, [40] * 9, [0] * 9),
                                         (16, [17, 515], [2, 0])])
def test_spans(D, mode, H, news, pos0):
    g = torch.Generator(device="cuda").manual_seed(D + mode + H)

    def rnd(*shape):
        return torch.randn(*shape, generator=g, device="cuda")

    T, n, G = sum(news), len(news), H // 2 if mode == ops.SCAN_SSD else H
    ssd = mode == ops.SCAN_SSD
    src, z, aux = rnd(T, 3 * H * D), rnd(T, H * D), torch.rand(T, H, 4, generator=g, device="cuda")
    zb = rnd(H) - 2 if ssd else rnd(H * D) + 1
    hp = rnd(H) * 0.5 if ssd else torch.rand(H * D, generator=g, device="cuda") * 0.9
    beta = rnd(T, H)
    slots = torch.randperm(n + 2, generator=torch.Generator().manual_seed(H))[:n].tolist()
    state = rnd(n + 2, H, D, D)
    start = state.clone()
    out = torch.zeros(T, H * D, device="cuda")
    kw = {ops.SCAN_GLA: dict(z=z, zbias=zb, qscale=D ** -0.5, inv_tau=0.125), ops.SCAN_MLSTM: dict(aux=aux, qscale=D ** -0.5),
          ops.SCAN_HGRN2: dict(z=z, zbias=zb, hparam=hp), ops.SCAN_SSD: dict(zbias=zb, hparam=hp, beta=beta, qscale=D ** -0.5)}[mode]
    ops.lin_scan(mode, src, 0, G * D if ssd else H * D, src, 2 * H * D, state, out, i32([sum(news[:i]) for i in range(n)]), i32(news),
                 i32([a + b for a, b in zip(news, pos0)]), i32(slots), n, max(news), H, G, D, D, **kw)
    want, end = reference(mode, D, H, G, news, pos0, src, z, zb, hp, beta, aux, D ** -0.5, 0.125, start, slots)
    for got, ref in ((out, want), (state, end)):
        assert torch.isfinite(got).all()
        assert float((got.double() - ref).norm() / ref.norm()) < BOUND
    untouched = [i for i in range(n + 2) if i not in [s for s, m in zip(slots, news) if m]]
    assert torch.equal(state[untouched], start[untouched])
