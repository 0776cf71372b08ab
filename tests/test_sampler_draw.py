"""The sampler's draw (csrc/sampler.cu) against sums in 64 bits: the kept set of top-p and the id whose share of its cumulated mass holds the random number, for
every cluster size, flat and peaked rows, and rows whose mass lies in the slice of one CTA."""
import pytest
import torch

from bee2bee_b200 import ops

pytestmark = pytest.mark.gpu


def _hash(x):
    x ^= x >> 16
    x = x * 0x7FEB352D & 0xFFFFFFFF
    x ^= x >> 15
    x = x * 0x846CA68B & 0xFFFFFFFF
    return x ^ x >> 16


# The kernel's exponentials are off by 2^-21 and less, their sums over 2^17 ids (tree of rows, warps and CTAs) by 2^-20, and the boundary of the kept set is exact to
# 2^-17 of a value: 2^-16 of the mass in all, and as much again for ids of the same weight beside the boundary of flat rows.
EDGE = 2.0 ** -15


@pytest.mark.parametrize("B,V", [(1, 1000), (3, 32003), (20, 50257), (40, 128256), (150, 1023), (8, 256000)])
@pytest.mark.parametrize("top_p", [0.3, 0.95, 0.9999, 1.0])
@pytest.mark.parametrize("shape", ["flat", "peaked", "one slice", "one id"])
def test_draw(B, V, top_p, shape):
    g = torch.Generator(device="cuda").manual_seed(V + B)
    ld = (V + 127) // 128 * 128
    logits = torch.randn(B, ld, generator=g, device="cuda") * 2.0
    if shape == "peaked":
        logits[:, ::max(1, V // 40)] += 14.0
    elif shape == "one slice":                               # the others are below 2^-32 of the largest
        logits[:, V - 70:] += 40.0
    elif shape == "one id":
        logits[:, V // 3] = 60.0
    logits[:, V:] = 1e9
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    full = lambda v: torch.full((B,), v, device="cuda")  # noqa: E731
    out = i32([0] * B)
    e = torch.exp(logits[:, :V].double() - logits[:, :V].double().amax(1, keepdim=True))
    order = e.sort(1, descending=True)
    before = order.values.cumsum(1) - order.values
    # in front of the boundary all weights together stay below top_p
    least = torch.where(before < top_p * e.sum(1, keepdim=True), order.values, 2.0).amin(1, keepdim=True)
    kept = torch.where(e >= least * (1 - 2.0 ** -17) * (0.0 if top_p == 1.0 else 1.0), e, 0.0)
    cdf = kept.cumsum(1)
    total = cdf[:, -1:]
    for step in range(4):
        ops.sample(logits, out, temperature=full(1.0), top_p=full(top_p), seeds=i32([11 + 5 * b for b in range(B)]), step=i32([step]), vocab=V)
        tok = out.long()[:, None]
        u = torch.tensor([[((_hash((11 + 5 * b) ^ _hash((step * 0x9E3779B9 + b) & 0xFFFFFFFF)) >> 8) + 0.5) / 2 ** 24] for b in range(B)], device="cuda", dtype=torch.float64)
        assert bool((kept.gather(1, tok) > 0).all())
        hi = cdf.gather(1, tok) / total
        lo = hi - kept.gather(1, tok) / total
        assert bool((u >= lo - EDGE).all()) and bool((u <= hi + EDGE).all())
