"""K-split cluster projections (csrc/gemm_rows.cu) at the edges of their tiles, splits and dispatch, against float64.

Bound per element: the accumulator is fp32 (K terms: |error| <= K 2^-24 sum |x w|, doubled for the order of the sums) and
every rounding point to bf16 adds half an ulp, 2^-9 of the value rounded there (the projection, the activation, the sum with
the residual); gelu's slope is below 1.13, silu(g) u's error is that of its factors."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
BF = torch.bfloat16
HALF_ULP = 2.0 ** -8  # of a value just above a power of two


def _inputs(M, N, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(M, K, device="cuda", generator=g).to(BF)
    w = (torch.randn(N, K, device="cuda", generator=g) * K ** -0.5).to(BF)
    acc = x.double() @ w.double().T
    slack = 2 * K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    return g, x, w, acc, slack


def _within(y, ref, bound):
    excess = ((y.double() - ref).abs() - bound).max().item()
    assert excess <= 0, excess


@pytest.mark.parametrize("M", [3, 16, 17, 128, 129, 161, 301, 1000])
@pytest.mark.parametrize("N,K", [(48, 64), (128, 512), (208, 1088), (768, 768), (2304, 4096), (2048, 5632)])
def test_projection(cuda, M, N, K):
    from dli_b200 import ops

    g, x, w, acc, slack = _inputs(M, N, K, M * 31 + N)
    bias = torch.randn(N, device=cuda, generator=g).to(BF)
    res = torch.randn(M, N, device=cuda, generator=g).to(BF)
    y = ops.gemm(x, w)
    _within(y, acc, slack + HALF_ULP * acc.abs())
    assert torch.equal(y, ops.gemm(x, w))  # the order of the sums is fixed
    z = acc + bias.double()
    ref = z + res.double()
    inplace = res.clone()
    ops.gemm(x, w, bias=bias, residual=inplace, out=inplace)
    _within(inplace, ref, slack + HALF_ULP * (z.abs() + slack + ref.abs() + 2.0 ** -7))
    ref = torch.nn.functional.gelu(z, approximate="tanh")
    _within(ops.gemm(x, w, bias=bias, epilogue=ops.EPI_GELU_NEW), ref,
            1.2 * (slack + HALF_ULP * z.abs()) + HALF_ULP * 1.1 * ref.abs() + 2e-6)


@pytest.mark.parametrize("M", [3, 31, 128, 150, 200, 301])
@pytest.mark.parametrize("F,K", [(128, 64), (384, 1024), (5632, 2048)])
def test_gated_projection(cuda, M, F, K):
    from dli_b200 import ops

    g, x, wg, gate, s1 = _inputs(M, F, K, M + F)
    wu = (torch.randn(F, K, device=cuda, generator=g) * K ** -0.5).to(BF)
    up, s2 = x.double() @ wu.double().T, 2 * K * 2.0 ** -24 * (x.double().abs() @ wu.double().abs().T)
    y = ops.gemm_gated_silu(x, ops.pack_gate_up(wg, wu))
    act = torch.nn.functional.silu(gate)
    e_gate, e_up = s1 + HALF_ULP * gate.abs(), s2 + HALF_ULP * up.abs()
    e_act = 1.1 * e_gate + HALF_ULP * (act.abs() + 1.1 * e_gate)  # silu's slope is below 1.1
    _within(y, act * up, e_act * (up.abs() + e_up) + act.abs() * e_up + HALF_ULP * 1.1 * (act * up).abs() + 1e-6)


@pytest.mark.parametrize("rows,H,KV,K", [(129, 4, 2, 512), (200, 32, 8, 1024), (333, 8, 2, 4096), (700, 4, 4, 2048)])
def test_qkv_projection_with_rope_equals_the_separate_steps(cuda, rows, H, KV, K):
    """The same bits as the projection followed by the rotation and append kernel, whatever the K split."""
    from dli_b200 import ops

    hd, page, g = 128, 16, torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, K, device=cuda, generator=g).to(BF)
    w = (torch.randn((H + 2 * KV) * hd, K, device=cuda, generator=g) * 0.05).to(BF)
    ang = torch.rand(rows + 9, hd // 2, device=cuda, generator=g) * 6.28
    cos, sin = ang.cos().to(BF), ang.sin().to(BF)
    positions = torch.arange(rows, device=cuda).int() + 9
    seq_ids = torch.zeros(rows, device=cuda).int()
    n_pages = (rows + 9 + page - 1) // page
    table = torch.randperm(n_pages, device=cuda, generator=g).int().reshape(1, n_pages)
    out = []
    for fused in (False, True):
        k = torch.zeros(n_pages, KV, page, hd, device=cuda, dtype=BF)
        v = torch.zeros_like(k)
        if fused:
            qkv = torch.empty(rows, (H + 2 * KV) * hd, device=cuda, dtype=BF)
            ops.linear_qkv_rope_append(x, w, qkv, cos, sin, positions, seq_ids, table, k, v, H, KV, hd)
        else:
            qkv = ops.gemm(x, w)
            ops.rope_kv_append(qkv, cos, sin, positions, seq_ids, table, k, v, H, KV, hd)
        out.append((qkv, k, v))
    assert all(torch.equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("M", [300, 1024, 1777])
@pytest.mark.parametrize("N,K", [(72, 512), (240, 768), (488, 1024), (2048, 2048), (4096, 512)])
def test_residual_read_by_the_line(cuda, M, N, K):
    """The residual added, also where it is the output, whatever kernel the sizes take (clusters, GEMV, persistent tiles)."""
    from dli_b200 import ops
    g, x, w, acc, slack = _inputs(M, N, K, M + N)
    r = torch.randn(M, N, device="cuda", generator=g).to(BF)
    y = ops.linear(x, w, residual=r)
    _within(y, acc + r.double(), slack + HALF_ULP * (acc.abs() + slack) + HALF_ULP * (acc + r.double()).abs() * 1.01)
    z = r.clone()
    ops.linear(x, w, residual=z, out=z)
    assert torch.equal(y, z)


@pytest.mark.parametrize("M,N,K,tile", [(130, 16, 512, (32, 1)), (300, 48, 64, (64, 1)), (301, 112, 1024, (64, 1)),
                                        (4097, 1040, 512, (128, 1)), (4352, 2320, 1024, (256, 1)), (4352, 4112, 4096, (256, 2)),
                                        (8192, 2064, 4096, (240, 2))])
def test_residual_on_the_persistent_tiles(cuda, M, N, K, tile):
    """Every width that sizes lead to, the last tile cut inside a 64-column line of the residual: the residual added, also
    where it is the output, with a bias and without."""
    from dli_b200 import ops

    if ops.sm_count() == 148:  # the choice counts SMs
        assert ops.gemm_plan(M, N, K) == ("persistent", *tile)
    g, x, w, acc, slack = _inputs(M, N, K, M + N)
    r = torch.randn(M, N, device=cuda, generator=g).to(BF)
    bias = torch.randn(N, device=cuda, generator=g).to(BF)
    for b in (None, bias):
        z = acc if b is None else acc + b.double()
        y = ops.gemm(x, w, bias=b, residual=r)
        _within(y, z + r.double(), slack + HALF_ULP * (z.abs() + slack) + HALF_ULP * (z + r.double()).abs() * 1.01)
        out = r.clone()
        ops.gemm(x, w, bias=b, residual=out, out=out)
        assert torch.equal(y, out)


@pytest.mark.parametrize("off", [1, 2, 4, 7])
@pytest.mark.parametrize("M,N,K", [(3, 48, 64), (17, 208, 1088), (128, 768, 768), (200, 2304, 4096), (9, 8192, 4096)])
def test_bias_that_starts_anywhere(cuda, M, N, K, off):
    """A slice of a packed bias vector: the same bits as an aligned copy of it, and right against float64."""
    from dli_b200 import ops

    g, x, w, acc, slack = _inputs(M, N, K, M + N + off)
    bias = torch.randn(N + 8, device=cuda, generator=g).to(BF)[off:off + N]
    assert bias.data_ptr() % 16
    z = acc + bias.double()
    for call in (ops.gemm, ops.linear, lambda *a, **k: ops.linear_splitk(*a, None, **k)):
        y = call(x, w, bias=bias)
        _within(y, z, slack + HALF_ULP * (z.abs() + slack))
        assert torch.equal(y, call(x, w, bias=bias.clone()))
