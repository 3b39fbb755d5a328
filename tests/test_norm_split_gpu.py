"""Norms on either side of the rule that gives a row a CTA or a warp, at the row lengths where the number of warps or of vectors per
thread changes: the sums keep one order, so every row has the bits of the same row by itself (a CTA each), and those are close
to float64."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
BF = torch.bfloat16


@pytest.mark.parametrize("d", [8, 256, 264, 512, 520, 768, 776, 1024, 2040, 2048, 2056, 4096, 4104, 8192, 8200, 16384])
@pytest.mark.parametrize("with_residual", [False, True])
@pytest.mark.parametrize("layernorm", [False, True])
def test_rows_have_the_bits_of_single_rows(cuda, d, with_residual, layernorm):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(d)
    rows = (4 if d <= 256 else 8 if d <= 512 else 15 if d <= 2048 else 1) * ops.sm_count() + 3
    x = (3 * torch.randn(rows, d, device=cuda, generator=g) + 1).to(BF)
    r = torch.randn(rows, d, device=cuda, generator=g).to(BF) if with_residual else None
    w, b = torch.randn(d, device=cuda, generator=g).to(BF), torch.randn(d, device=cuda, generator=g).to(BF)

    def norm(lo, hi):
        h, part = torch.empty_like(x[lo:hi]), None if r is None else r[lo:hi]
        if layernorm:
            return ops.add_layernorm(x[lo:hi], w, b, 1e-5, residual=part, resid_out=h), h
        return ops.add_rmsnorm(x[lo:hi], w, 1e-5, residual=part, resid_out=h), h

    y, h = norm(0, rows)
    few_y, few_h = norm(3, rows)  # the last row count that gives each row a CTA
    assert torch.equal(y[3:], few_y) and torch.equal(h[3:], few_h)
    for i in (0, 1, 7, 8, rows - 1):
        one_y, one_h = norm(i, i + 1)
        assert torch.equal(y[i:i + 1], one_y) and torch.equal(h[i:i + 1], one_h)
    hf = (x if r is None else r + x).double()
    assert torch.equal(h, hf.to(BF))
    if layernorm:
        # fp32 sums of d terms, then the last rounding: half a unit of bf16 and what the sums' error moves
        c = hf - hf.mean(-1, keepdim=True)
        n = c * torch.rsqrt(c.pow(2).mean(-1, keepdim=True) + 1e-5)
        ref, slack = n * w.double() + b.double(), 1e-5 * (n.abs() + 1) * w.double().abs()
        assert ((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1.01 * slack).all()
    else:
        # two roundings (h * rstd, then * weight) of at most half a unit of bf16 each
        ref = hf * torch.rsqrt(hf.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()
        assert ((y.double() - ref).abs() <= (2 * 2.0 ** -8 * 1.01 + 1e-5) * ref.abs() + 1e-30).all()
