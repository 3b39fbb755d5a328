"""Decode rows through post-norm + add + norm + convolution with four channels a thread, at widths around whole warps and the largest
it takes, against the general form (which a tail that starts off 16 bytes takes).  Bound: fp32 sums of d squares in another order."""
import pytest
from test_conv_single_gpu import _state

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("d", [4, 124, 128, 132, 2044, 2052, 4092, 4096, 4100])
@pytest.mark.parametrize("post", [True, False])
def test_as_the_general_form(cuda, d, post, dt):
    from dli_b200 import ops

    y, x, tail, w, ent = _state(5, d, 4, dt, d)
    flat = torch.empty(tail.numel() + 1, device=cuda)
    off = flat[1:].view_as(tail).copy_(tail)
    got, want = torch.empty_like(y), torch.empty_like(y)
    xa, xb = x.clone(), x.clone()
    torch.cuda.synchronize()
    for xx, tt, out in ((xa, tail, got), (xb, off, want)):
        ops.postnorm_add_norm_conv_single(y if post else None, xx, tt, w, ent, out, 0.7, 1.3, 1e-5)
    unit = (d + 16) * 2.0 ** -24
    assert ((xa - xb).abs() <= 2 * unit * (xb.abs() + 4) + 2.0 ** -22).all()
    assert ((tail - off).abs() <= 4 * unit * (off.abs() + 2) + 2.0 ** -22).all()
    mag = (1 + w.abs().sum(1)) * 8
    ulp = 2.0 ** -7 if dt == torch.bfloat16 else 2.0 ** -22
    assert ((got.float() - want.float()).abs() <= 8 * unit * mag + 2.0 ** -20 + ulp * want.float().abs()).all()
