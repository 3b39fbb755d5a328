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
