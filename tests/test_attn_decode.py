"""Decode attention with the keys as MMA rows (csrc/attn_decode.cu) against 64-bit sums: lengths around a tile (128 keys) and a page (64), one key,
clusters that share the keys (few sequences, wide block tables), every head group size, windows, capped scores, idle rows, the e4m3 copy."""
import pytest
import torch

from bee2bee_b200 import ops

pytestmark = pytest.mark.gpu

# probabilities are rounded to bf16 (2^-9 each, independent) as operands of the second product and the result once more: 2^-8 covers both
BOUND = 2.0 ** -8


def i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def setup(lens, nq, nkv, D, spare=0):
    g = torch.Generator(device="cuda").manual_seed(nq * D + len(lens))
    need = [(n + 63) // 64 for n in lens]
    order = (torch.randperm(sum(need), generator=torch.Generator().manual_seed(1)) + 1).tolist()
    table, at = [], 0
    for n in need:
        table.append(order[at:at + n] + [0] * (max(need) + spare - n))
        at += n
    k = torch.randn(sum(need) + 1, 64, nkv, D, generator=g, device="cuda").bfloat16()
    v = torch.randn(sum(need) + 1, 64, nkv, D, generator=g, device="cuda").bfloat16()
    q = (torch.randn(len(lens), nq * D, generator=g, device="cuda") * 2 * D ** -0.5).bfloat16()
    return q, k, v, i32(table)


def reference(q, k, v, table, lens, nq, nkv, D, window, cap):
    out = torch.zeros(q.shape, device="cuda", dtype=torch.float64)
    for s, n in enumerate(lens):
        at = torch.arange(n, device="cuda")
        at = (table[s].long()[at // 64] * 64 + at % 64)[max(0, n - window) if window else 0:]
        kk, vv = (c.view(-1, nkv, D)[at].double().repeat_interleave(nq // nkv, 1) for c in (k, v))
        sc = torch.einsum("hd,khd->hk", q[s].double().view(nq, D), kk)
        if cap:
            sc = cap * torch.tanh(sc / cap)
        out[s] = torch.einsum("hk,khd->hd", sc.softmax(-1), vv).flatten()
    return out


@pytest.mark.parametrize("nq,nkv,D", [(32, 8, 128), (6, 1, 128), (16, 1, 128), (4, 2, 256), (12, 1, 256), (3, 3, 128)])
@pytest.mark.parametrize("lens,spare", [([1], 0), ([700], 5), ([128, 129, 127, 64, 63, 65], 0), ([1, 3000, 250, 17], 40), ([90 * i + 1 for i in range(40)], 0)])
@pytest.mark.parametrize("window,cap", [(0, 0.0), (100, 50.0), (0, 50.0), (128, 0.0)])
def test_decode(nq, nkv, D, lens, spare, window, cap):
    q, k, v, table = setup(lens, nq, nkv, D, spare)
    S = len(lens)
    idle = S // 2 if S > 2 else -1
    on = [0 if s == idle else 1 for s in range(S)]
    out = torch.full_like(q, 7.0)
    ops.attention(q, k, v, out, table, i32(list(range(S))), i32(on), i32(lens), max_q=1, n_q=nq, n_kv=nkv, head_dim=D, window=window, softcap=cap)
    keep = [s for s in range(S) if on[s]]
    ref = reference(q, k, v, table, lens, nq, nkv, D, window, cap)[keep]
    err = (out[keep].double() - ref).norm(dim=1) / ref.norm(dim=1)
    assert float(err.max()) < BOUND
    if idle >= 0:
        assert bool((out[idle] == 7.0).all())
    assert ops.native().attn_decode_gave_up() == 0


def test_large_scores_move_the_reference():
    """every later tile outgrows the reference maximum of the tiles before it"""
    lens, nq, nkv, D = [1000], 8, 2, 128
    q, k, v, table = setup(lens, nq, nkv, D)
    at = torch.arange(1000, device="cuda")
    rows = table[0].long()[at // 64] * 64 + at % 64
    k.view(-1, nkv, D)[rows] = (k.view(-1, nkv, D)[rows].float() * (1 + at.float()[:, None, None] / 60)).bfloat16()
    out = torch.zeros_like(q)
    ops.attention(q, k, v, out, table, i32([0]), i32([1]), i32(lens), max_q=1, n_q=nq, n_kv=nkv, head_dim=D)
    ref = reference(q, k, v, table, lens, nq, nkv, D, 0, 0.0)
    assert float((out.double() - ref).norm() / ref.norm()) < BOUND


@pytest.mark.parametrize("S", [3, 40])
def test_quantised_copy(S):
    nq, nkv, D = 8, 2, 128
    lens = [100 + 37 * i for i in range(S)]
    q, k, v, table = setup(lens, nq, nkv, D)
    args = (table, i32(list(range(S))), i32([1] * S), i32(lens))
    kw = dict(max_q=1, n_q=nq, n_kv=nkv, head_dim=D)
    plain = ops.attention(q, k, v, torch.zeros_like(q), *args, **kw)
    bn = ops.pick_bn_mx(S)
    want_q, want_sf = ops.quant_mxfp8_rows(plain, bn)
    fq, sf = torch.zeros(S, nq * D, device="cuda", dtype=torch.float8_e4m3fn), torch.full_like(want_sf, 127)
    ops.attention(q, k, v, torch.zeros_like(q), *args, **kw, fq_out=fq, fq_sf=sf, fq_bn=bn)
    assert torch.equal(fq.view(torch.uint8), want_q.view(torch.uint8))
    assert torch.equal(ops.mx_unchunk(sf, S, nq * D, bn), ops.mx_unchunk(want_sf, S, nq * D, bn))


@pytest.mark.parametrize("cap", [0.0, 50.0])
@pytest.mark.parametrize("lens", [[300], [60, 200, 500]])
def test_nan_stays(lens, cap):
    """NaN in a query or a key reaches the heads that see it, capped or not, and no other"""
    nq, nkv, D = 8, 2, 128
    q, k, v, table = setup(lens, nq, nkv, D)
    q[-1, 3 * D + 5] = float("nan")                              # head 3 of the last sequence
    page = int(table[0, 0])
    k[page, 7, 1, 9] = float("nan")                              # a key of key/value head 1 of the first: its heads 4 to 7
    out = torch.zeros_like(q)
    ops.attention(q, k, v, out, table, i32(list(range(len(lens)))), i32([1] * len(lens)), i32(lens), max_q=1, n_q=nq, n_kv=nkv, head_dim=D, softcap=cap)
    got = out.view(len(lens), nq, D).isnan()
    want = torch.zeros_like(got)
    want[-1, 3], want[0, 4:] = True, True
    assert torch.equal(got, want)


def test_capped_scores_far_beyond_the_cap():
    lens, nq, nkv, D = [200], 4, 1, 128
    q, k, v, table = setup(lens, nq, nkv, D)
    q *= 3000.0                                                  # |score / cap| up to some hundreds
    out = torch.zeros_like(q)
    ops.attention(q, k, v, out, table, i32([0]), i32([1]), i32(lens), max_q=1, n_q=nq, n_kv=nkv, head_dim=D, softcap=50.0)
    ref = reference(q, k, v, table, lens, nq, nkv, D, 0, 50.0)
    assert float((out.double() - ref).norm() / ref.norm()) < BOUND


def test_dominant_weight():
    """One key of a later tile outweighs all others while the reference of the first tile is kept, so its weight is 2^c with any mantissa.  The sum
    is over rounded weights, so this rounding cancels and the result's own is left: 2^-8 / sqrt(3) / mantissa, 0.00166 in the mean square over
    mantissas (0.0023 with an unrounded sum)."""
    S, nq, nkv, D = 64, 4, 1, 128
    q, k, v, table = setup([300] * S, nq, nkv, D)
    q = q[:, :D].repeat(1, nq)                                   # (the heads of a sequence are alike)
    unit = (q[:, :D].float() / q[:, :D].float().pow(2).sum(1, keepdim=True))
    for s in range(S):
        score = torch.full((300, 1), -6.0, device="cuda")
        score[0], score[200] = 0.0, 3.0 + 2.0 * s / S            # natural units: c from 4.3 to 7.2
        at = torch.arange(300, device="cuda")
        k.view(-1, nkv, D)[table[s].long()[at // 64] * 64 + at % 64, 0] = (score * unit[s]).bfloat16()
    out = torch.zeros_like(q)
    ops.attention(q, k, v, out, table, i32(list(range(S))), i32([1] * S), i32([300] * S), max_q=1, n_q=nq, n_kv=nkv, head_dim=D)
    ref = reference(q, k, v, table, [300] * S, nq, nkv, D, 0, 0.0)
    assert float((out.double() - ref).norm() / ref.norm()) < 0.0019


# Two neighbouring key/value heads of 64 channels are one of 128: one query head each and several (in columns 4 or 8 apart), one pair and many, few sequences
# in clusters of 8, 4 and 2 and more of them than fit at once in the larger size (6 and 12 sequences of 6 pairs)
@pytest.mark.parametrize("nq,nkv", [(12, 12), (2, 2), (8, 4), (20, 4), (16, 2)])
@pytest.mark.parametrize("lens,spare", [([1], 0), ([128, 129, 127, 64, 63, 65], 0), ([1, 3000, 250, 17], 40), ([1100 + 31 * i for i in range(12)], 0),
                                        ([90 * i + 1 for i in range(40)], 0)])
@pytest.mark.parametrize("window,cap", [(0, 0.0), (100, 50.0)])
def test_pairs_of_64(nq, nkv, lens, spare, window, cap):
    test_decode(nq, nkv, 64, lens, spare, window, cap)


def test_a_pair_stays_apart():
    """keys and values of one head that are not finite reach its own query heads alone"""
    lens, nq, nkv = [70, 300], 8, 4
    q, k, v, table = setup(lens, nq, nkv, 64)
    ref = reference(q, k, v, table, lens, nq, nkv, 64, 0, 0.0).view(2, nq, 64)
    page = int(table[1][1])
    k[page, 5, 1, 3] = float("inf")
    v[page, 9, 2, 60] = float("nan")
    out = torch.empty_like(q)
    ops.attention(q, k, v, out, table, i32([0, 1]), i32([1, 1]), i32(lens), max_q=1, n_q=nq, n_kv=nkv, head_dim=64)
    out = out.view(2, nq, 64)
    assert torch.isnan(out[1, 4:6, 60]).all()
    for s, h in ((0, slice(0, 8)), (1, slice(0, 2)), (1, slice(6, 8))):
        assert float((out[s, h].double() - ref[s, h]).norm() / ref[s, h].norm()) < BOUND
    other = torch.arange(64, device="cuda") != 60
    assert float((out[1, 4:6, other].double() - ref[1, 4:6, other]).norm() / ref[1, 4:6, other].norm()) < BOUND


def test_pairs_quantised_copy():
    """the e4m3 copy of 64-wide heads is what quantising the output gives; with split keys it is refused"""
    lens, nq, nkv = [70, 300, 129], 8, 4
    q, k, v, table = setup(lens, nq, nkv, 64)
    args = (q, k, v, torch.empty_like(q), table, i32([0, 1, 2]), i32([1, 1, 1]), i32(lens))
    opts = dict(max_q=1, n_q=nq, n_kv=nkv, head_dim=64)
    out = ops.attention(*args, **opts)
    q8 = torch.zeros(3, nq * 64, device="cuda", dtype=torch.float8_e4m3fn)
    sf = torch.full((nq * 64 // 128 * 512,), 127, device="cuda", dtype=torch.uint8)
    ops.attention(*args, **opts, fq_out=q8, fq_sf=sf, fq_bn=32)
    want, want_sf = ops.quant_mxfp8_rows(out, 32)
    assert torch.equal(q8.view(torch.uint8), want.view(torch.uint8))
    assert torch.equal(ops.mx_unchunk(sf, 3, nq * 64, 32), ops.mx_unchunk(want_sf, 3, nq * 64, 32))
    with pytest.raises(RuntimeError):
        ops.attention(*args, **opts, splits=2, ws=torch.zeros(1 << 20, device="cuda"), fq_out=q8, fq_sf=sf, fq_bn=32)


@pytest.mark.parametrize("nq,nkv", [(6, 2), (20, 4), (12, 2), (14, 2)])
def test_other_groups_of_64_keep_fp32_weights(nq, nkv):
    """64-wide heads in groups that the tensor-core kernels with bf16 weights did not take in pairs: the CUDA-core kernel's result, bit for bit, whole and with
    split keys, and no e4m3 copy"""
    lens = [70, 3000, 129, 1]
    q, k, v, table = setup(lens, nq, nkv, 64)
    args = (table, i32([0, 1, 2, 3]), i32([1] * 4), i32(lens))
    opts = dict(max_q=1, n_q=nq, n_kv=nkv, head_dim=64)
    for split in (dict(), dict(splits=4, ws=torch.zeros(1 << 20, device="cuda"))):
        out, cuda_core = (ops.attention(q, k, v, torch.zeros_like(q), *args, **opts, **split, use_tc=tc) for tc in (-1, 0))
        assert torch.equal(out, cuda_core)
        ref = reference(q, k, v, table, lens, nq, nkv, 64, 0, 0.0)
        assert float((out.double() - ref).norm() / ref.norm()) < 0.0019     # (the rounding of the result; bf16 weights add as much again)
    with pytest.raises(RuntimeError):
        ops.attention(q, k, v, torch.zeros_like(q), *args, **opts, fq_out=torch.zeros(4, nq * 64, device="cuda", dtype=torch.float8_e4m3fn),
                      fq_sf=torch.zeros(1 << 14, device="cuda", dtype=torch.uint8), fq_bn=32)
