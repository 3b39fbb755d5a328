"""postnorm_add_norm at every number of elements that a thread may hold, against float64.  Bound: fp32 sums of d squares
(d 2^-24 relative, halved by the root) and a few roundings beside them."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows", [5, 70])
@pytest.mark.parametrize("d", [8, 256, 257, 512, 1000, 1025, 2048, 2049, 4096, 4100, 8192, 8200])
def test_against_float64(cuda, d, rows, dt):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(d + rows)
    y, x = torch.randn(rows, d, device=cuda, generator=g).to(dt), 3 * torch.randn(rows, d, device=cuda, generator=g)
    unit = lambda v: v / (v.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt()  # noqa: E731
    want = x.double() + unit(y.double()) * 0.7
    hw = unit(want) * 1.3
    for with_norm in (True, False):
        xa, hn = x.clone(), torch.full_like(x, float("nan"))
        ops.postnorm_add_norm(y, xa, 0.7, 1e-5, hn if with_norm else None, 1.3 if with_norm else 1.0)
        tol = (d + 16) * 2.0 ** -24
        assert ((xa.double() - want).abs() <= tol * ((want - x.double()).abs() + want.abs() * 2.0 ** -3) + 2.0 ** -22).all()
        if with_norm:
            assert ((hn.double() - hw).abs() <= 2 * tol * hw.abs() + 2.0 ** -20).all()
