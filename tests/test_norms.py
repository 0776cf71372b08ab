"""RMS norm kernels around their size rules: 1/rms by warps from 592 rows on, outputs by blocks up to 4096 channels, 1/rms of the rows written."""
import pytest
import torch

from bee2bee_b200 import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [8, 264, 1024, 1032, 2304, 4096, 4104, 8192])
@pytest.mark.parametrize("T", [1, 591, 593, 1000])
def test_rms(h, T):
    g = torch.Generator(device="cuda").manual_seed(h + T)
    x, r, w = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((T, h), (T, h), (h,)))
    d = x.double()
    inv = (d.pow(2).mean(-1) + 1e-6).rsqrt()
    assert float((ops.rstd(x, 1e-6).double() / inv - 1).abs().max()) < 1e-5           # sums of h fp32 squares
    mine, own = torch.empty(T, device="cuda"), torch.empty(T, device="cuda")
    before = ops.LAUNCHES[0]
    out = ops.rmsnorm(x, w, residual=r, eps=1e-6, plus_one=True, rstd_out=mine, out_rstd=own)
    assert ops.LAUNCHES[0] - before == (1 if h <= 4096 else 2)
    ref = d * inv[:, None] * (1 + w.double()) + r.double()
    assert float(((out.double() - ref).abs() / ref.abs().clamp_min(1e-3)).max()) < 2.0 ** -8 + 1e-2 * 2.0 ** -4     # one bf16 rounding, cancelling sums
    assert float((mine.double() / inv - 1).abs().max()) < 1e-5
    assert float((own.double() * (out.double().pow(2).mean(-1) + 1e-6).sqrt() - 1).abs().max()) < 1e-5
    plain = ops.rmsnorm(x, w, eps=1e-6)
    ref = d * inv[:, None] * w.double()
    assert float((plain.double() - ref).norm() / ref.norm()) < 2.0 ** -8
