"""The GEMV's rows per task (csrc/gemv.cu): the choice depends on the matrix, the result does not.  A matrix is compared bit
for bit with the same rows in calls of other sizes (other choices), and with float64 within the fp32 sum's error (K 2^-24
sum |x w|, doubled) and the rounding to bf16 (2^-8 covers half an ulp of either rounding point)."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
BF = torch.bfloat16


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("N,K", [(1, 8), (7, 2048), (443, 768), (1777, 264), (2220, 2048), (2221, 2048), (2665, 1024),
                                 (3108, 4096), (3555, 2056), (8192, 2048), (32003, 512)])
def test_projection(cuda, M, N, K):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(N + K)
    x = torch.randn(M, K, device=cuda, generator=g).to(BF)
    w = (torch.randn(N, K, device=cuda, generator=g) * K ** -0.5).to(BF)
    res = torch.randn(M, N, device=cuda, generator=g).to(BF)
    ln = torch.randn(K, device=cuda, generator=g).to(BF)
    y = ops.gemv(x, w, residual=res)
    acc = x.double() @ w.double().T
    ref = acc + res.double()
    slack = 2 * K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    assert ((y.double() - ref).abs() <= slack + 2.0 ** -8 * (acc.abs() + slack + ref.abs())).all()
    normed = ops.rmsnorm_linear(x, ln, 1e-5, w)
    for step in (61, 997):
        if N // step > 64:
            continue
        parts = [ops.gemv(x, w[i:i + step].contiguous(), residual=res[:, i:i + step].contiguous()) for i in range(0, N, step)]
        assert torch.equal(y, torch.cat(parts, dim=1))
        parts = [ops.rmsnorm_linear(x, ln, 1e-5, w[i:i + step].contiguous()) for i in range(0, N, step)]
        assert torch.equal(normed, torch.cat(parts, dim=1))


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("F,K", [(128, 2048), (1280, 2048), (1408, 768), (5632, 2048), (1536, 4096)])
def test_gated(cuda, M, F, K):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(F)
    x = torch.randn(M, K, device=cuda, generator=g).to(BF)
    wg, wu = ((torch.randn(F, K, device=cuda, generator=g) * K ** -0.5).to(BF) for _ in range(2))
    y = ops.gemv_gated_silu(x, ops.pack_gate_up(wg, wu))
    parts = [ops.gemv_gated_silu(x, ops.pack_gate_up(wg[i:i + 128], wu[i:i + 128])) for i in range(0, F, 128)]
    assert torch.equal(y, torch.cat(parts, dim=1))
    a, b = ops.gemv(x, wg).float(), ops.gemv(x, wu).float()  # the same sums
    ref = torch.nn.functional.silu(a).to(BF).float() * b
    torch.testing.assert_close(y.float(), ref, rtol=2.0 ** -7, atol=1e-6)  # one ulp: expf against torch's


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("N,K", [(3000, 10752), (18432, 12288), (2221, 14336), (1500, 16384)])
def test_norm_of_long_rows(cuda, M, N, K):
    """Rows of x that take so much shared memory that it bounds the rows per task: the same bits as in pieces."""
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(N + K)
    x, ln = torch.randn(M, K, device=cuda, generator=g).to(BF), torch.randn(K, device=cuda, generator=g).to(BF)
    w = (torch.randn(N, K, device=cuda, generator=g) * K ** -0.5).to(BF)
    y = ops.rmsnorm_linear(x, ln, 1e-5, w)
    parts = [ops.rmsnorm_linear(x, ln, 1e-5, w[i:i + 997].contiguous()) for i in range(0, N, 997)]
    assert torch.equal(y, torch.cat(parts, dim=1))
