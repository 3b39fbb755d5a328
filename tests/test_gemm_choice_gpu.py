"""Which kernel a prompt's projections take (csrc/gemm_tcgen05.cu): sizes at which one of the three was measured to be faster than the
others by 4 % and more, around where the choice has its borders.  The times are the fastest kernel's and what the others took."""
import pytest
from test_gemm_rows_gpu import HALF_ULP, _inputs, _within

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
BF = torch.bfloat16

MEASURED = [  # rows, outputs, K, gated, kernel; us of the persistent kernel, the clusters and the pairs
    (1777, 8192, 28672, False, "pairs"),   # 680 / 713 / 545
    (2048, 8192, 28672, False, "pairs"),   # 774 / 856 / 696
    (900, 57344, 8192, True, "pairs"),     # 710 / 787 / 636
    (2048, 57344, 8192, True, "pairs"),    # 1455 / 1717 / 1345
    (4096, 57344, 8192, True, "pairs"),    # 2922 / 3556 / 2741
    (301, 28672, 4096, True, "rows"),      # 84 / 76 / 82
    (336, 28672, 4096, True, "persistent"),  # 85 / 95 / 83
    (400, 28672, 4096, True, "pairs"),     # 112 / 112 / 91
    (301, 8192, 8192, False, "rows"),      # 60 / 41 / 44
    (400, 4096, 14336, False, "rows"),     # 90 / 44 / 50
    (450, 4096, 4096, False, "pairs"),     # 32 / 22 / 19
    (2048, 256, 4096, False, "rows"),      # narrow: the pairs 27 % slower
    # qkv projections, with the rotation in the epilogue (without it they take the same kernel)
    (129, 10240, 8192, False, "rows"),     # 67 / 37 / 49
    (129, 15360, 5120, False, "rows"),     # 66 / 43 / 50
    (301, 6144, 4096, False, "rows"),      # 38 / 22 / 28
    (384, 6144, 4096, False, "rows"),      # 38 / 23 / 28
    (600, 6144, 4096, False, "pairs"),     # 38 / 30 / 29
    (1024, 6144, 4096, False, "pairs"),    # 59 / 54 / 39
    (512, 10240, 8192, False, "pairs"),    # 104 / 92 / 72
]


@pytest.mark.parametrize("M,N,K,gated,kernel", MEASURED)
def test_the_kernel_measured_to_be_faster(cuda, M, N, K, gated, kernel):
    from dli_b200 import ops

    if ops.sm_count() != 148:
        pytest.skip("the choice counts SMs")
    assert ops.gemm_plan(M, N, K, gated)[0] == kernel


@pytest.mark.parametrize("M,kernel", [(301, "rows"), (336, "persistent"), (400, "pairs"), (560, "persistent")])
def test_gated_forms_on_each_kernel(cuda, M, kernel):
    """silu, the clamped activation and gelu of 14 336 gates from 4 096 inputs, against float64.  Bounds as in test_gemm_rows_gpu.py:
    gate and up carry the sum's slack and a rounding, the activation's slope is below 1.1 (gelu 1.13), silu is rounded before the
    product."""
    from dli_b200 import ops

    F, K, limit, alpha = 14336, 4096, 1.1, 1.702
    if ops.sm_count() == 148:
        assert ops.gemm_plan(M, 2 * F, K, True)[0] == kernel
    g, x, wg, gate, s1 = _inputs(M, F, K, M)
    wu = (torch.randn(F, K, device=cuda, generator=g) * K ** -0.5).to(BF)
    up, s2 = x.double() @ wu.double().T, 2 * K * 2.0 ** -24 * (x.double().abs() @ wu.double().abs().T)
    w, e_gate, e_up = ops.pack_gate_up(wg, wu), s1 + HALF_ULP * gate.abs(), s2 + HALF_ULP * up.abs()
    act = torch.nn.functional.silu(gate)
    e_act = 1.1 * e_gate + HALF_ULP * (act.abs() + 1.1 * e_gate)
    _within(ops.linear_gated_silu(x, w), act * up, e_act * (up.abs() + e_up) + act.abs() * e_up + HALF_ULP * 1.1 * (act * up).abs() + 1e-6)
    held = gate.clamp(max=limit)
    act, u1 = held * torch.sigmoid(alpha * held), up.clamp(-limit, limit) + 1
    got = ops.linear_gated_act(x, w, torch.tensor([limit, alpha], device=cuda))
    _within(got, act * u1, 1.1 * e_gate * (u1.abs() + e_up) + act.abs() * e_up + HALF_ULP * 1.1 * (act * u1).abs() + 1e-6)
    act = torch.nn.functional.gelu(gate, approximate="tanh")
    got = ops.linear_gated_act(x, w, torch.zeros(2, device=cuda))
    _within(got, act * up, 1.13 * e_gate * (up.abs() + e_up) + act.abs() * e_up + HALF_ULP * 1.1 * (act * up).abs() + 1e-6)


@pytest.mark.parametrize("hd,H,KV,bias,kernel", [(128, 64, 8, False, "gemm_prefill_kernel"), (128, 64, 8, True, "gemm_pair_kernel"),
                                                 (128, 78, 1, False, "gemm_pair_kernel"), (64, 128, 16, False, "gemm_pair_kernel")])
def test_qkv_where_the_persistent_kernel_is_chosen(cuda, hd, H, KV, bias, kernel):
    """The rotation and the cache append in the persistent kernel's epilogue where it has them, else in the pairs': the bits of the
    projection on the persistent kernel and the separate rotation either way."""
    from dli_b200 import ops

    T, d, ff, page, prefix = 350, 8192, 256, 16, 5
    g = torch.Generator(device="cuda").manual_seed(H)
    rnd = lambda *s, std=1.0: (std * torch.randn(*s, device=cuda, generator=g)).to(BF)  # noqa: E731
    N, pages = (H + 2 * KV) * hd, (T + prefix + 15) // 16
    if ops.sm_count() == 148:
        assert ops.gemm_plan(T, N, d)[0] == "persistent"
    L = {"ln1": rnd(d), "ln2": rnd(d), "wqkv": rnd(N, d, std=0.02), "wo": rnd(d, H * hd, std=0.02), "wdown": rnd(d, ff, std=0.02),
         "wgu": ops.pack_gate_up(rnd(ff, d, std=0.02), rnd(ff, d, std=0.02))}
    if bias:
        L["bqkv"] = rnd(N)
    ang = torch.rand(T + prefix, hd // 2, device=cuda, generator=g) * 6.28
    cos, sin = ang.cos().to(BF), ang.sin().to(BF)
    table = torch.randperm(pages, device=cuda, generator=g).int().view(1, pages)
    positions, seq_ids, last = (torch.empty(T, device=cuda, dtype=torch.int32) for _ in range(3))
    ops.prompt_rows(positions, seq_ids, last, 1, T, prefix, 0)
    h_in = rnd(T, d)
    kc, vc = (torch.zeros(pages, KV, page, hd, device=cuda, dtype=BF) for _ in range(2))
    h, x, qkv, attn, act = (torch.empty(T, w, device=cuda, dtype=BF) for w in (d, d, N, H * hd, ff))
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
        ops.prompt_layers([L], [kc], [vc], table, table, h_in, h, x, qkv, attn, act, cos, sin, positions, seq_ids, 1, T, prefix,
                          H, KV, hd, 1e-5, hd ** -0.5)
        torch.cuda.synchronize()
    names = [e.name for e in prof.events()]
    assert not any("rope_kv_append" in n for n in names)
    if ops.sm_count() == 148:
        assert kernel in next(n for n in names if "gemm_" in n)  # the first projection
    ops.add_rmsnorm(h_in, L["ln1"], 1e-5, out=x)
    want = ops.gemm(x, L["wqkv"], bias=L.get("bqkv"))
    k2, v2 = torch.zeros_like(kc), torch.zeros_like(vc)
    ops.rope_kv_append(want, cos, sin, positions, seq_ids, table, k2, v2, H, KV, hd)
    assert torch.equal(qkv, want) and torch.equal(kc, k2) and torch.equal(vc, v2)
