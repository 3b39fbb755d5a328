"""The activations in the projections' epilogues, over every bf16 value they can be given."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
BF = torch.bfloat16


def _normal_values(cuda):
    v = torch.arange(65536, device=cuda, dtype=torch.int32).to(torch.int16).view(BF)
    return v[torch.isfinite(v) & (v.float().abs() >= 2.0 ** -126)]  # the tensor cores' sums know no -0


def test_silu_of_every_gate(cuda):
    """The bits of x / (1 + exp(-x)) in fp32 with CUDA's exp and division, rounded to bf16 (torch's silu)."""
    from dli_b200 import ops

    gates = _normal_values(cuda)
    want = torch.nn.functional.silu(gates)
    n = (gates.numel() + 127) // 128 * 128
    wg, wu = torch.zeros(n, 64, device=cuda, dtype=BF), torch.zeros(n, 64, device=cuda, dtype=BF)
    wg[:gates.numel(), 0] = gates
    wu[:, 1] = 1
    w = ops.pack_gate_up(wg, wu)
    x = torch.zeros(700, 64, device=cuda, dtype=BF)
    x[:, :2] = 1
    for rows in (1, 8, 40, 700):
        y = ops.linear_gated_silu(x[:rows], w)
        for r in (0, rows - 1):
            assert torch.equal(y[r, :gates.numel()].view(torch.int16), want.view(torch.int16))


def test_gelu_of_every_value(cuda):
    """Within half a bf16 ulp (2^-8 of a value just above a power of two) and the fp32 error of the exponent (2^-17 at the far end)
    of the exact value; 1 + tanh would lose all of it below -5.  Results below the normal range are only held to be as small."""
    from dli_b200 import ops

    v = _normal_values(cuda)
    n = (v.numel() + 127) // 128 * 128
    w = torch.zeros(n, 64, device=cuda, dtype=BF)
    w[:v.numel(), 0] = v
    x = torch.zeros(700, 64, device=cuda, dtype=BF)
    x[:, 0] = 1
    z = v.double()
    want = z * torch.sigmoid(2 * (2 / torch.pi) ** 0.5 * (z + 0.044715 * z ** 3))
    for rows in (1, 8, 40, 700):
        y = ops.linear(x[:rows], w, epilogue=ops.EPI_GELU_NEW)
        for r in (0, rows - 1):
            got = y[r, :v.numel()].double()
            assert ((got - want).abs() <= (2.0 ** -8 + 2.0 ** -16) * want.abs() + 2.0 ** -120).all()


def _every_value(cuda):
    return torch.arange(65536, device=cuda, dtype=torch.int32).to(torch.int16).view(BF)


def _gated(cuda, K):
    """The weights of a gated projection whose gates are all 65 536 values, whose ups are 1, and the rows to feed it."""
    from dli_b200 import ops

    wg, wu = torch.zeros(65536, K, device=cuda, dtype=BF), torch.zeros(65536, K, device=cuda, dtype=BF)
    wg[:, 0] = _every_value(cuda)
    wu[:, 1] = 1
    x = torch.zeros(700, K, device=cuda, dtype=BF)
    x[:, :2] = 1
    return wg, ops.pack_gate_up(wg, wu), x


@pytest.mark.parametrize("rows,K,kernel", [(1, 64, None), (8, 64, None), (40, 64, "rows"), (700, 64, "pairs"),
                                           (350, 4096, "persistent")])
def test_silu_of_zeros_subnormals_infinities_and_nans_too(cuda, rows, K, kernel):
    """All 65 536 gates through each kernel (None: the GEMV and the stream of few rows).  The gate is what the projection by itself
    hands over: its sums know no -0."""
    from dli_b200 import ops

    wg, w, x = _gated(cuda, K)
    if kernel and ops.sm_count() == 148:
        assert ops.gemm_plan(rows, 131072, K, True)[0] == kernel
    gate = ops.linear(x[:rows], wg)[0]
    v = _every_value(cuda)
    assert torch.equal(gate[~v.isnan()], v[~v.isnan()]) and gate.isnan().equal(v.isnan())
    want = torch.nn.functional.silu(gate)
    y = ops.linear_gated_silu(x[:rows], w)
    for r in (0, rows - 1):
        assert y[r].isnan().equal(want.isnan())
        assert torch.equal(y[r].nan_to_num(0.0), want.nan_to_num(0.0))


def test_gelu_on_the_persistent_kernel(cuda):
    """As test_gelu_of_every_value, at a width that keeps the projection off the pairs."""
    from dli_b200 import ops

    v = _normal_values(cuda)
    n = (v.numel() + 127) // 128 * 128 + 16
    w = torch.zeros(n, 64, device=cuda, dtype=BF)
    w[:v.numel(), 0] = v
    x = torch.zeros(4097, 64, device=cuda, dtype=BF)
    x[:, 0] = 1
    assert ops.gemm_plan(4097, n, 64)[0] == "persistent"
    z = v.double()
    want = z * torch.sigmoid(2 * (2 / torch.pi) ** 0.5 * (z + 0.044715 * z ** 3))
    y = ops.linear(x, w, epilogue=ops.EPI_GELU_NEW)
    for r in (0, 4096):
        assert ((y[r, :v.numel()].double() - want).abs() <= (2.0 ** -8 + 2.0 ** -16) * want.abs() + 2.0 ** -120).all()
