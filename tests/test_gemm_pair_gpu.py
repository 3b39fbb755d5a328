"""Projections on pairs of SMs (csrc/gemm_pair.cu) at the edges of their tiles, against float64; bounds as in
test_gemm_rows_gpu.py.  Sizes: the last row tile with one row, with the peer's half empty, and full; tails of narrower tiles;
more tiles than pairs, and fewer."""
import pytest
from test_gemm_rows_gpu import BF, HALF_ULP, _inputs, _within

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _on_pairs(ops, *sizes):
    if ops.sm_count() == 148:  # the choice counts SMs
        assert ops.gemm_plan(*sizes)[0] == "pairs"


@pytest.mark.parametrize("M,N,K", [(1281, 4096, 4096), (768, 6144, 512), (1000, 2560, 2048), (1409, 5632, 64), (4097, 1920, 192),
                                   (2176, 8192, 1024), (5000, 768, 768)])
def test_projection(cuda, M, N, K):
    from dli_b200 import ops

    _on_pairs(ops, M, N, K)
    g, x, w, acc, slack = _inputs(M, N, K, M + N)
    bias, res = torch.randn(N + 8, device=cuda, generator=g).to(BF), torch.randn(M, N, device=cuda, generator=g).to(BF)
    y = ops.gemm(x, w)
    _within(y, acc, slack + HALF_ULP * acc.abs())
    assert torch.equal(y, ops.gemm(x, w))
    for b in (bias[:N], bias[3:N + 3]):  # a bias may start anywhere
        z = acc + b.double()
        ref = z + res.double()
        inplace = res.clone()
        ops.gemm(x, w, bias=b, residual=inplace, out=inplace)
        _within(inplace, ref, slack + HALF_ULP * (z.abs() + slack + ref.abs() + 2.0 ** -7))
        assert torch.equal(inplace, ops.gemm(x, w, bias=b, residual=res))
    ref = torch.nn.functional.gelu(z, approximate="tanh")
    _within(ops.gemm(x, w, bias=b, epilogue=ops.EPI_GELU_NEW), ref,
            1.2 * (slack + HALF_ULP * z.abs()) + HALF_ULP * 1.1 * ref.abs() + 2e-6)


@pytest.mark.parametrize("M,F,K", [(513, 8192, 512), (1000, 14336, 512), (900, 5632, 2048), (3000, 1024, 1024), (1500, 5632, 1088)])
def test_gated_projection(cuda, M, F, K):
    from dli_b200 import ops

    _on_pairs(ops, M, 2 * F, K, True)
    g, x, wg, gate, s1 = _inputs(M, F, K, M + F)
    wu = (torch.randn(F, K, device=cuda, generator=g) * K ** -0.5).to(BF)
    up, s2 = x.double() @ wu.double().T, 2 * K * 2.0 ** -24 * (x.double().abs() @ wu.double().abs().T)
    y = ops.gemm_gated_silu(x, ops.pack_gate_up(wg, wu))
    act = torch.nn.functional.silu(gate)
    e_gate, e_up = s1 + HALF_ULP * gate.abs(), s2 + HALF_ULP * up.abs()
    e_act = 1.1 * e_gate + HALF_ULP * (act.abs() + 1.1 * e_gate)  # silu's slope is below 1.1
    _within(y, act * up, e_act * (up.abs() + e_up) + act.abs() * e_up + HALF_ULP * 1.1 * (act * up).abs() + 1e-6)


@pytest.mark.parametrize("hd,H,KV,d,B,T,bias,rotate", [(64, 32, 4, 2048, 1, 1777, None, True), (64, 32, 4, 2048, 2, 700, 1, True),
                                                       (128, 32, 8, 4096, 3, 300, None, True), (128, 31, 1, 1024, 1, 1500, 0, True),
                                                       (64, 24, 24, 1536, 2, 900, 2, False)])
def test_qkv_epilogue_equals_the_separate_steps(cuda, hd, H, KV, d, B, T, bias, rotate):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(B * T + d)
    rnd = lambda *s, std=1.0: (std * torch.randn(*s, device=cuda, generator=g)).to(BF)  # noqa: E731
    rows, N, ff, page, prefix, pages = B * T, (H + 2 * KV) * hd, 256, 16, 5, (T + 5 + 15) // 16
    _on_pairs(ops, rows, N, d)
    L = {"ln1": rnd(d), "ln2": rnd(d), "wqkv": rnd(N, d, std=0.05), "wo": rnd(d, H * hd, std=0.05), "wdown": rnd(d, ff, std=0.05),
         "wgu": ops.pack_gate_up(rnd(ff, d, std=0.05), rnd(ff, d, std=0.05))}
    if bias is not None:
        L["bqkv"] = rnd(N + bias)[bias:]
    cos = sin = None
    if rotate:
        ang = torch.rand(T + prefix, hd // 2, device=cuda, generator=g) * 6.28
        cos, sin = ang.cos().to(BF), ang.sin().to(BF)
    table = torch.randperm((B + 1) * pages, device=cuda, generator=g).int().view(B + 1, pages)
    positions, seq_ids, last = (torch.empty(rows, device=cuda, dtype=torch.int32) for _ in range(3))
    ops.prompt_rows(positions, seq_ids, last, B, T, prefix, 1)
    h_in = rnd(rows, d)
    kc, vc = (torch.zeros((B + 1) * pages, KV, page, hd, device=cuda, dtype=BF) for _ in range(2))
    h, x, qkv, attn, act = (torch.empty(rows, w, device=cuda, dtype=BF) for w in (d, d, N, H * hd, ff))
    ops.prompt_layers([L], [kc], [vc], table, table[1:], h_in, h, x, qkv, attn, act, cos, sin, positions, seq_ids, B, T, prefix,
                      H, KV, hd, 1e-5, hd ** -0.5)
    ops.add_rmsnorm(h_in, L["ln1"], 1e-5, out=x)
    want = ops.gemm(x, L["wqkv"], bias=L.get("bqkv"))
    k2, v2 = torch.zeros_like(kc), torch.zeros_like(vc)
    ops.rope_kv_append(want, cos, sin, positions, seq_ids, table, k2, v2, H, KV, hd)
    assert torch.equal(qkv, want) and torch.equal(kc, k2) and torch.equal(vc, v2)
