"""The CTA-pair GEMM of many tokens (csrc/gemm_wide.cu) against 64-bit products, at the sizes where its tiles can go wrong: one row more or
less than a 256-token tile, feature counts that leave part of a tile, every tile width and the split last round; neighbours that are late."""
import time

import pytest
import torch

from bee2bee_b200 import ops

pytestmark = pytest.mark.gpu

ROUND = 2.0 ** -8        # a bf16 result is within half a unit of 2^-8 of the exact one; fp32 sums of these lengths add less than 2^-14


def bf(*shape, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + sum(shape))
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


def near(a, b, bound=ROUND):
    assert torch.isfinite(a.float()).all()
    err = (a.double() - b.double()).norm() / b.double().norm()
    assert err <= bound, float(err)


# As the rule picks them.  129 / 255 / 256 / 257: around a token tile; 65: half a tile.  Features: 128 (one 128-wide tile), 384 and 1024
# (128-wide), 18944 (74 tiles of 256), 13056 and 4224 and 6144 (192-wide, no rest).  k 128: the shortest ring; 576: no multiple of the ring depth.
@pytest.mark.parametrize("m,n,k", [(65, 128, 128), (129, 384, 576), (255, 1024, 512), (256, 18944, 128), (257, 13056, 192), (700, 4224, 1024),
                                   (300, 6144, 4096)])
def test_epilogues(m, n, k):
    w, x, res = bf(n, k, scale=k ** -0.5), bf(m, k), bf(m, n)
    bias = torch.randn(n, device="cuda")
    rstd = torch.rand(m, device="cuda") + 0.5
    ref = x.double() @ w.double().t()
    near(ops.gemm(w, x, rstd=rstd, bias=bias), ref * rstd.double()[:, None] + bias.double())
    near(ops.gemm(w, x, bias=bias, out_fp32=True), ref + bias.double(), 1e-5)
    near(ops.gemm(w, x, epi=ops.EPI_RESIDUAL, residual=res), ref + res.double())
    wide = torch.zeros(m, n + 64, device="cuda", dtype=torch.bfloat16)               # rows longer than the result
    ops.gemm(w, x, out=wide[:, :n], epi=ops.EPI_GELU, act_gelu=ops.ACT_RELU_SQ)
    near(wide[:, :n], ref.clamp_min(0).pow(2), 2 * ROUND)
    assert float(wide[:, n:].abs().max()) == 0.0
    near(ops.gemm(w, x, epi=ops.EPI_GELU, bias=bias), torch.nn.functional.gelu(ref + bias.double(), approximate="tanh"))


@pytest.mark.parametrize("f,m", [(64, 129), (12672, 256), (1024, 1000)])             # 12672: 99 tiles, the last round is split
@pytest.mark.parametrize("gelu", [0, 1])
def test_gate_up(f, m, gelu):
    k = 512
    wg, wu, x = bf(f, k, scale=k ** -0.5, seed=1), bf(f, k, scale=k ** -0.5, seed=2), bf(m, k)
    rstd = torch.rand(m, device="cuda") + 0.5
    out = ops.gemm(ops.glu_interleave_rows(wg, wu), x, epi=ops.EPI_GLU, act_gelu=gelu, rstd=rstd)
    g, u = (x.double() @ w.double().t() * rstd.double()[:, None] for w in (wg, wu))
    g = torch.nn.functional.gelu(g, approximate="tanh") if gelu else torch.nn.functional.silu(g)
    near(out, g * u)


# Every tile, whole and cut along K, over feature counts that leave part of the last one: 640 = 3 x 192 + 64 = 2 x 256 + 128 (cut: the second
# pair of the cluster has no columns there), 896 = 4 x 192 + 128 = 3 x 256 + 128, 768: no rest.  k 512: the shortest that is cut; 576: halves of 4 and 5 blocks.
TILES = [(128, 0), (128, 1), (192, 0), (256, 0), (256, 1)]


@pytest.mark.parametrize("tile,split", TILES)
@pytest.mark.parametrize("m,n,k", [(300, 640, 512), (129, 896, 576), (513, 768, 1024)])
def test_every_tile(tile, split, m, n, k):
    kw = dict(wide_tile=tile, wide_split=split)
    w, x, res = bf(n, k, scale=k ** -0.5), bf(m, k), bf(m, n)
    bias = torch.randn(n, device="cuda")
    rstd = torch.rand(m, device="cuda") + 0.5
    ref = x.double() @ w.double().t()
    wide = torch.zeros(m, n + 64, device="cuda", dtype=torch.bfloat16)
    ops.gemm(w, x, out=wide[:, :n], rstd=rstd, bias=bias, **kw)
    near(wide[:, :n], ref * rstd.double()[:, None] + bias.double())
    assert float(wide[:, n:].abs().max()) == 0.0
    near(ops.gemm(w, x, bias=bias, out_fp32=True, **kw), ref + bias.double(), 1e-5)
    near(ops.gemm(w, x, epi=ops.EPI_RESIDUAL, residual=res, **kw), ref + res.double())
    near(ops.gemm(w, x, epi=ops.EPI_GELU, bias=bias, **kw), torch.nn.functional.gelu(ref + bias.double(), approximate="tanh"))
    if tile == 256 or (tile == 128 and not split):               # (a gate / up pair is 128 columns wide)
        g, u = (ref[:, i:i + n // 2] for i in (0, n // 2))
        out = ops.gemm(ops.glu_interleave_rows(w[:n // 2], w[n // 2:]), x, epi=ops.EPI_GLU, **kw)
        near(out, torch.nn.functional.silu(g) * u)
    assert ops.native().gemm_wide_gave_up() == 0


@pytest.mark.parametrize("tile,split", TILES)
@pytest.mark.parametrize("hd,nq,nkv,m", [(128, 3, 1, 300), (64, 6, 2, 129), (256, 3, 2, 257), (32, 20, 4, 140)])
def test_qkv_every_tile(tile, split, hd, nq, nkv, m):
    check_qkv(hd, nq, nkv, m, 512, wide_tile=tile, wide_split=split)


@pytest.mark.parametrize("hd,nq,nkv,m", [(128, 8, 2, 200), (64, 8, 4, 257), (256, 4, 2, 131)])
def test_qkv(hd, nq, nkv, m):
    check_qkv(hd, nq, nkv, m, 256)


def check_qkv(hd, nq, nkv, m, k, **tile):
    theta = 10000.0
    n = (nq + 2 * nkv) * hd
    w, x = bf(n, k, scale=k ** -0.5), bf(m, k)
    pages = m // ops.PAGE + 2
    pos = torch.randperm(600, device="cuda")[:m].int()
    slots = torch.randperm(pages * ops.PAGE, device="cuda")[:m].int()
    slots[::5] = -1
    kc = torch.zeros(pages, ops.PAGE, nkv, hd, device="cuda", dtype=torch.bfloat16)
    vc, q = torch.zeros_like(kc), torch.zeros(m, nq * hd, device="cuda", dtype=torch.bfloat16)
    ops.gemm(w, x, epi=ops.EPI_QKV_ROPE, q_out=q, k_cache=kc, v_cache=vc, positions=pos, slots=slots, n_q_heads=nq, n_kv_heads=nkv,
             head_dim=hd, rope_theta=theta, q_scale=0.25, **tile)
    y = (x.double() @ w.double().t()).view(m, -1, hd)
    ang = pos.double()[:, None] * theta ** (-torch.arange(0, hd, 2, device="cuda", dtype=torch.float64) / hd)
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]
    a, b = y[..., 0::2], y[..., 1::2]
    turned = torch.stack([a * cos - b * sin, b * cos + a * sin], -1).flatten(-2)
    near(q.view(m, nq, hd), turned[:, :nq] * 0.25)
    keep = slots >= 0
    want_k, want_v = torch.zeros(kc.view(-1, nkv, hd).shape, device="cuda", dtype=torch.float64), None
    want_v = want_k.clone()
    want_k[slots[keep].long()], want_v[slots[keep].long()] = turned[keep][:, nq:nq + nkv], y[keep][:, nq + nkv:]
    near(kc.view(-1, nkv, hd), want_k)
    near(vc.view(-1, nkv, hd), want_v)
    assert torch.equal(kc.view(-1, nkv, hd)[want_k.flatten(1).norm(dim=1) == 0], torch.zeros_like(kc.view(-1, nkv, hd)[want_k.flatten(1).norm(dim=1) == 0]))


def test_handoff_words():
    """upstream flag already published, consumer slot free: the flag words advance by one payload and both destinations hold the result"""
    m, n, k = 200, 512, 256
    w, x, res = bf(n, k, scale=k ** -0.5), bf(m, k), bf(m, n)
    word = torch.zeros(8, device="cuda", dtype=torch.int32)      # in flag, in epoch, out flag, out epoch, done, ack, (free), unused
    word[0] = 1
    at = [word.data_ptr() + 4 * i for i in range(8)]
    out, out2 = torch.zeros(m, n, device="cuda", dtype=torch.bfloat16), torch.zeros(m, n, device="cuda", dtype=torch.bfloat16)
    ops.gemm(w, x, out=out, epi=ops.EPI_RESIDUAL, residual=res, wait_flag=at[0], wait_epoch=at[1], signal_flag=at[2], signal_epoch=at[3],
             done_counter=at[4], bump_epoch=at[1], ack_flag=at[5], free_flag=at[6], out2_ptr=out2.data_ptr())
    near(out, x.double() @ w.double().t() + res.double())
    assert torch.equal(out, out2)
    assert word.tolist() == [1, 1, 1, 1, 0, 1, 0, 0]
    assert ops.native().gemm_wide_gave_up() == 0


@pytest.fixture
def abort_word():
    """bounded flag waits as in the engine: they raise this word at the limit"""
    word = torch.zeros(64, device="cuda", dtype=torch.int32)
    C = ops.native()

    def limit(ms):
        C.set_wait_policy(word.data_ptr(), float(ms))
        return word
    yield limit
    torch.cuda.synchronize()
    C.set_wait_policy(0, 0.0)


def _handoff(m, n, k, flags):
    """a product that waits for both neighbours, behind the kernels in front of it at the head of a piece"""
    w, x, res = bf(n, k, scale=k ** -0.5), bf(m, k), bf(m, n)
    word = torch.zeros(8, device="cuda", dtype=torch.int32)      # in epoch, out flag, out epoch, done, ack
    at = [word.data_ptr() + 4 * i for i in range(8)]
    out = torch.zeros(m, n, device="cuda", dtype=torch.bfloat16)
    word[2] = 1                                                  # one payload is out already: the next one waits for its release
    torch.cuda.synchronize()
    ops.native().flag_wait(flags.data_ptr(), at[0], 1)
    r = ops.rstd(x, 1e-5)
    ops.gemm(w, x, out=out, epi=ops.EPI_RESIDUAL, residual=res, rstd=r, wait_flag=flags.data_ptr(), wait_epoch=at[0], signal_flag=at[1],
             signal_epoch=at[2], done_counter=at[3], bump_epoch=at[0], ack_flag=at[4], free_flag=flags.data_ptr() + 64, free_lag=0)
    rs = (x.double().pow(2).mean(1, keepdim=True) + 1e-5).rsqrt()
    return out, (x.double() @ w.double().t()) * rs + res.double(), word


@pytest.mark.parametrize("m,n", [(200, 512), (1000, 18944)])     # one tile per pair and four (both accumulators in use)
def test_late_neighbours(m, n, abort_word):
    """the host publishes the upstream flag some seconds after the launch and releases the output slot a second later: no wait counts before"""
    abort = abort_word(30000)
    before = ops.native().gemm_wide_gave_up()
    flags = torch.ones(32, dtype=torch.int32).pin_memory()
    _handoff(m, n, 256, flags)                                   # (kernels are loaded on first use, which a waiting kernel would hold up)
    torch.cuda.synchronize()
    flags.zero_()
    out, ref, word = _handoff(m, n, 256, flags)
    time.sleep(4.5)                                              # (2^24 polls last 1 to 4 s)
    flags[0] = 1
    time.sleep(1.0)
    flags[16] = 1
    torch.cuda.synchronize()
    near(out, ref)
    assert word.tolist() == [1, 2, 2, 0, 1, 0, 0, 0]
    assert ops.native().gemm_wide_gave_up() == before and int(abort[0]) == 0


def test_neighbour_that_never_comes(abort_word):
    """the wait for the upstream flag runs out: the abort word is up, and neither the payload nor the input slot is released"""
    abort = abort_word(300)
    flags = torch.zeros(32, dtype=torch.int32).pin_memory()
    flags[16] = 1
    _, _, word = _handoff(200, 512, 256, flags)
    torch.cuda.synchronize()
    assert int(abort[0]) == 1
    assert word.tolist() == [0, 0, 1, 0, 0, 0, 0, 0]
    abort.zero_()


# Block-scaled fp8: the runs of scale factors of tokens come in tiles of 128 (m <= 512: 129 and 300 leave half a pair without one) or 256 (513), those of
# weights per 128 features: 640 and 896 leave the second run of the last 256-wide tile out.  k 256: two stages; 1152: 9, no multiple of a ring, halves of 4 and 5 blocks;
# 18944 features (74 and 148 tiles of 256): accumulators that overlap, as the rule picks them.
def spread(rows, k, seed):
    """rows whose blocks of 32 lie powers of two apart: a scale factor from another place is a large error"""
    g = torch.Generator(device="cuda").manual_seed(seed + rows + k)
    e = torch.randint(-3, 4, (rows, k // 32), generator=g, device="cuda").double().repeat_interleave(32, 1)
    return (torch.randn(rows, k, generator=g, device="cuda").double() * torch.exp2(e)).to(torch.bfloat16)


MX_TILES = [(0, -1), (128, 0), (128, 1), (256, 0), (256, 1)]


@pytest.mark.parametrize("tile,split", MX_TILES)
@pytest.mark.parametrize("m,n,k", [(65, 128, 1152), (129, 896, 256), (300, 640, 1152), (513, 1280, 1024), (700, 18944, 256)])
def test_block_scaled(tile, split, m, n, k):
    if split == 1 and k < 1024:
        pytest.skip("fewer than 8 stages are not cut")
    kw = dict(wide_tile=tile, wide_split=split) if tile else {}
    wq, sfa = ops.quantize_weight_mxfp8(spread(n, k, 1))
    bn = ops.pick_bn_mx(m)
    ss = torch.zeros(m, device="cuda")
    xq, sfb = ops.quant_mxfp8_rows(spread(m, k, 2), bn, sumsq_out=ss)
    w = ops.mx_dequant(wq, ops.mx_unchunk(sfa, n, k)).double()
    ref = ops.mx_dequant(xq, ops.mx_unchunk(sfb, m, k, bn)).double() @ w.t()
    sf = dict(sfa=sfa, sfb=sfb, **kw)
    near(ops.gemm(wq, xq, out_fp32=True, **sf), ref, 1e-5)

    def quantised(call, width):
        """a call that leaves a quantised copy of its bf16 result: the one that quantising the result gives, its sums of squares, and words cleared"""
        q8 = torch.zeros(m, width, device="cuda", dtype=torch.float8_e4m3fn)
        q_sf = torch.full(((m + bn - 1) // bn * (width // 128) * (bn // 128) * 512,), 127, device="cuda", dtype=torch.uint8)
        sums, clear = torch.zeros(m, device="cuda"), torch.ones(m, device="cuda")
        out = call(fq_out=q8, fq_sf=q_sf, fq_bn=bn, sumsq_out=sums, zero_buf=clear)
        want, want_sf = ops.quant_mxfp8_rows(out, bn)
        assert torch.equal(q8.view(torch.uint8), want.view(torch.uint8))
        assert torch.equal(ops.mx_unchunk(q_sf, m, width, bn), ops.mx_unchunk(want_sf, m, width, bn))
        near(sums, out.double().pow(2).sum(1), 1e-5)
        assert not clear.any()
        return out

    res = bf(m, n)
    rs = (ss.double() / k + 1e-5).rsqrt()[:, None]
    near(quantised(lambda **q: ops.gemm(wq, xq, epi=ops.EPI_RESIDUAL, residual=res, sumsq=ss, eps=1e-5, **q, **sf), n), ref * rs + res.double())
    if n % 256 == 0 and (tile != 128 or split <= 0):                       # (a gate / up pair is 128 columns wide)
        gu = (ref * rs).view(m, n // 128, 2, 64)
        near(quantised(lambda **q: ops.gemm(wq, xq, epi=ops.EPI_GLU, sumsq=ss, eps=1e-5, out=torch.empty(m, n // 2, device="cuda", dtype=torch.bfloat16),
                                            **q, **sf), n // 2), (torch.nn.functional.silu(gu[:, :, 0]) * gu[:, :, 1]).flatten(1))
    assert ops.native().gemm_wide_gave_up() == 0


@pytest.mark.parametrize("bn", [192, 512, 65536 + 128])
def test_unknown_token_tiles_are_refused(bn):
    """scale factors of tokens are read in runs of 128, alone or two side by side; a call that names any other tile is refused by the host, with the kernel's
    tile named or not, and so are copies that would be written in larger tiles"""
    m, n, k = 300, 256, 1024
    wq, sfa = ops.quantize_weight_mxfp8(bf(n, k))
    xq = torch.zeros(m, k, device="cuda", dtype=torch.float8_e4m3fn)
    sf = torch.full((((m + 127) // 128 + 1) * (k // 128) * 1024,), 127, device="cuda", dtype=torch.uint8)
    for tile in (dict(wide_tile=256), dict(wide_tile=1), dict()):
        with pytest.raises(RuntimeError):
            ops.gemm(wq, xq, sfa=sfa, sfb=sf, bn=bn, **tile)
    if bn > 256:
        with pytest.raises(RuntimeError):
            ops.quant_mxfp8_rows(bf(m, k), bn)
        with pytest.raises(RuntimeError):
            ops.gemm(wq, xq, sfa=sfa, sfb=sf, bn=128, epi=ops.EPI_RESIDUAL, residual=bf(m, n), fq_out=torch.zeros(m, n, device="cuda", dtype=torch.float8_e4m3fn),
                     fq_sf=sf, fq_bn=bn)


def mx_operands(m, n, k):
    """block-scaled weights and tokens with the tokens' sums of squares, and their exact product behind the norm"""
    wq, sfa = ops.quantize_weight_mxfp8(spread(n, k, 1))
    bn = ops.pick_bn_mx(m)
    ss = torch.zeros(m, device="cuda")
    xq, sfb = ops.quant_mxfp8_rows(spread(m, k, 2), bn, sumsq_out=ss)
    ref = ops.mx_dequant(xq, ops.mx_unchunk(sfb, m, k, bn)).double() @ ops.mx_dequant(wq, ops.mx_unchunk(sfa, n, k)).double().t()
    return wq, xq, dict(sfa=sfa, sfb=sfb, sumsq=ss, eps=1e-5), ref * (ss.double() / k + 1e-5).rsqrt()[:, None], bn


def mx_copy(m, width, bn):
    """room for an e4m3 copy and its scale factors"""
    return (torch.zeros(m, width, device="cuda", dtype=torch.float8_e4m3fn),
            torch.full(((m + bn - 1) // bn * (width // 128) * (bn // 128) * 512,), 127, device="cuda", dtype=torch.uint8))


def is_copy(q8, q_sf, out, bn):
    want, want_sf = ops.quant_mxfp8_rows(out, bn)
    assert torch.equal(q8.view(torch.uint8), want.view(torch.uint8))
    assert torch.equal(ops.mx_unchunk(q_sf, *out.shape, bn), ops.mx_unchunk(want_sf, *out.shape, bn))


# rotary pairs, cache rows and the norm of block-scaled tokens: every prompt of more than 64 tokens goes through them.  k 1152: 9 stages, halves of 4 and 5;
# 520 tokens: runs of scale factors in tiles of 256
@pytest.mark.parametrize("tile,split", MX_TILES)
@pytest.mark.parametrize("hd,nq,nkv,m", [(128, 3, 1, 300), (64, 6, 2, 129), (256, 3, 2, 520), (32, 20, 4, 65)])
def test_block_scaled_qkv(tile, split, hd, nq, nkv, m):
    theta, k, n = 10000.0, 1152, (nq + 2 * nkv) * hd
    wq, xq, mx, ref, _ = mx_operands(m, n, k)
    pages = m // ops.PAGE + 2
    pos = torch.randperm(600, device="cuda")[:m].int()
    slots = torch.randperm(pages * ops.PAGE, device="cuda")[:m].int()
    slots[::5] = -1
    kc = torch.zeros(pages, ops.PAGE, nkv, hd, device="cuda", dtype=torch.bfloat16)
    vc, q = torch.zeros_like(kc), torch.zeros(m, nq * hd, device="cuda", dtype=torch.bfloat16)
    ops.gemm(wq, xq, epi=ops.EPI_QKV_ROPE, q_out=q, k_cache=kc, v_cache=vc, positions=pos, slots=slots, n_q_heads=nq, n_kv_heads=nkv, head_dim=hd,
             rope_theta=theta, q_scale=0.25, **mx, **(dict(wide_tile=tile, wide_split=split) if tile else {}))
    y = ref.view(m, -1, hd)
    ang = pos.double()[:, None] * theta ** (-torch.arange(0, hd, 2, device="cuda", dtype=torch.float64) / hd)
    cos, sin = ang.cos()[:, None], ang.sin()[:, None]
    a, b = y[..., 0::2], y[..., 1::2]
    turned = torch.stack([a * cos - b * sin, b * cos + a * sin], -1).flatten(-2)
    near(q.view(m, nq, hd), turned[:, :nq] * 0.25)
    keep = slots >= 0
    for cache, rows in ((kc, turned[:, nq:nq + nkv]), (vc, y[:, nq + nkv:])):
        want = torch.zeros(pages * ops.PAGE, nkv, hd, device="cuda", dtype=torch.float64)
        want[slots[keep].long()] = rows[keep]
        got = cache.view(-1, nkv, hd)
        near(got, want)
        assert not got[want.flatten(1).norm(dim=1) == 0].any()
    assert ops.native().gemm_wide_gave_up() == 0


@pytest.mark.parametrize("gelu", [0, 1])
@pytest.mark.parametrize("m,n,k,tile", [(70, 512, 256, 0), (300, 768, 1024, 256), (1000, 18944, 256, 256)])
def test_block_scaled_gate_up_without_rows(m, n, k, tile, gelu):
    """a product whose only reader takes the e4m3 copy writes no bf16 rows: the copy is that of the call which does"""
    wq, xq, mx, ref, bn = mx_operands(m, n, k)
    kw = dict(epi=ops.EPI_GLU, act_gelu=gelu, **mx, **(dict(wide_tile=tile, wide_split=0) if tile else {}))
    out = ops.gemm(wq, xq, **kw)
    g, u = (ref.view(m, n // 128, 2, 64)[:, :, i] for i in (0, 1))
    act = torch.nn.functional.gelu(g, approximate="tanh") if gelu else torch.nn.functional.silu(g)
    near(out, (act * u).flatten(1))
    q8, q_sf = mx_copy(m, n // 2, bn)
    ops.gemm(wq, xq, fq_out=q8, fq_sf=q_sf, fq_bn=bn, no_out=True, **kw)
    is_copy(q8, q_sf, out, bn)
    assert ops.native().gemm_wide_gave_up() == 0


def test_block_scaled_copy_of_nan():
    """a token that is not a number leaves the copy that the quantiser would, its own rows alone"""
    m, n, k = 200, 512, 256
    wq, xq, mx, ref, bn = mx_operands(m, n, k)
    res = bf(m, n)
    res[7], res[9, 40] = float("nan"), float("inf")
    q8, q_sf = mx_copy(m, n, bn)
    out = ops.gemm(wq, xq, epi=ops.EPI_RESIDUAL, residual=res, fq_out=q8, fq_sf=q_sf, fq_bn=bn, **mx)
    assert out[7].isnan().all() and out.isfinite().sum() == m * n - n - 1
    is_copy(q8, q_sf, out, bn)


def _quantised_hop(m, n, k, flags):
    """a product between two neighbours that hand over block-scaled rows: it waits for the upstream one's, and leaves its rows, their e4m3 copy and their sums
    of squares in the downstream one's memory"""
    wq, xq, mx, ref, bn = mx_operands(m, n, k)
    res = bf(m, n)
    word = torch.zeros(8, device="cuda", dtype=torch.int32)      # in epoch, out flag, out epoch, done, ack
    at = [word.data_ptr() + 4 * i for i in range(8)]
    out, (q8, q_sf) = torch.zeros(m, n, device="cuda", dtype=torch.bfloat16), mx_copy(m, n, bn)
    sums, clear = torch.zeros(m, device="cuda"), torch.ones(m, device="cuda")
    word[2] = 1                                                  # one payload is out already: the next one waits for its release
    torch.cuda.synchronize()
    ops.gemm(wq, xq, out=out, epi=ops.EPI_RESIDUAL, residual=res, wait_flag=flags.data_ptr(), wait_epoch=at[0], signal_flag=at[1], signal_epoch=at[2],
             done_counter=at[3], bump_epoch=at[0], ack_flag=at[4], free_flag=flags.data_ptr() + 64, free_lag=0, fq_out=q8, fq_sf=q_sf, fq_bn=bn,
             sumsq_out=sums, zero_buf=clear, wide_tile=256, wide_split=0, **mx)

    def arrived():
        near(out, ref + res.double())
        is_copy(q8, q_sf, out, bn)
        near(sums, out.double().pow(2).sum(1), 1e-5)
        assert not clear.any()
    return arrived, word


@pytest.mark.parametrize("m,n", [(200, 512), (1000, 18944)])     # one tile per pair and four, whose accumulators overlap
def test_quantised_hop(m, n, abort_word):
    """both neighbours are there, and then both are late, each by more than a bounded wait of a kernel lasts"""
    abort = abort_word(30000)
    before = ops.native().gemm_wide_gave_up()
    flags = torch.ones(32, dtype=torch.int32).pin_memory()
    arrived, word = _quantised_hop(m, n, 256, flags)
    torch.cuda.synchronize()
    arrived()
    assert word.tolist() == [1, 2, 2, 0, 1, 0, 0, 0]
    flags.zero_()
    arrived, word = _quantised_hop(m, n, 256, flags)
    time.sleep(4.5)                                              # (2^24 polls last 1 to 4 s)
    flags[0] = 1
    time.sleep(4.5)
    flags[16] = 1
    torch.cuda.synchronize()
    arrived()
    assert word.tolist() == [1, 2, 2, 0, 1, 0, 0, 0]
    assert ops.native().gemm_wide_gave_up() == before and int(abort[0]) == 0
