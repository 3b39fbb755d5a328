"""Norms of many short rows: the warp-per-row kernel gives the bits of the CTA-per-row kernel (which fewer than 64 rows
take), for every row length it accepts."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
BF = torch.bfloat16


@pytest.mark.parametrize("d", [8, 64, 248, 256, 264, 768, 1000, 1600, 2040, 2048])
@pytest.mark.parametrize("with_residual", [False, True])
def test_same_bits_as_one_row_at_a_time(cuda, d, with_residual):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(d)
    rows = 131
    x = (3 * torch.randn(rows, d, device=cuda, generator=g) + 1).to(BF)
    r = torch.randn(rows, d, device=cuda, generator=g).to(BF) if with_residual else None
    w, b = torch.randn(d, device=cuda, generator=g).to(BF), torch.randn(d, device=cuda, generator=g).to(BF)
    for norm in (lambda *a, **k: ops.add_layernorm(*a, **k), lambda x_, w_, b_, e_, **k: ops.add_rmsnorm(x_, w_, e_, **k)):
        h = torch.empty_like(x)
        y = norm(x, w, b, 1e-5, residual=r, resid_out=h)
        for lo, hi in ((0, 1), (1, 40), (40, 103), (103, 131)):
            part = None if r is None else r[lo:hi]
            h1 = torch.empty_like(x[lo:hi])
            assert torch.equal(y[lo:hi], norm(x[lo:hi], w, b, 1e-5, residual=part, resid_out=h1))
            assert torch.equal(h[lo:hi], h1)


@pytest.mark.parametrize("d", [8, 256, 264, 768, 1024, 1032, 2040, 2048])
@pytest.mark.parametrize("with_residual", [False, True])
def test_same_bits_in_many_rows(cuda, d, with_residual):
    """Row counts on the warp-per-row side of the rule (which counts SMs): the bits of calls of few rows."""
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(d + 1)
    rows = 6 * ops.sm_count() + 5
    x = (3 * torch.randn(rows, d, device=cuda, generator=g) + 1).to(BF)
    r = torch.randn(rows, d, device=cuda, generator=g).to(BF) if with_residual else None
    w, b = torch.randn(d, device=cuda, generator=g).to(BF), torch.randn(d, device=cuda, generator=g).to(BF)
    for norm in (lambda *a, **k: ops.add_layernorm(*a, **k), lambda x_, w_, b_, e_, **k: ops.add_rmsnorm(x_, w_, e_, **k)):
        h = torch.empty_like(x)
        y = norm(x, w, b, 1e-5, residual=r, resid_out=h)
        for lo in range(0, rows, 60):
            part = None if r is None else r[lo:lo + 60]
            h1 = torch.empty_like(x[lo:lo + 60])
            assert torch.equal(y[lo:lo + 60], norm(x[lo:lo + 60], w, b, 1e-5, residual=part, resid_out=h1))
            assert torch.equal(h[lo:lo + 60], h1)
