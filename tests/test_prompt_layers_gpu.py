"""A prompt pass through a shard's layers in one native call (csrc/prompt.cu) and what ShardEngine.prefill hands to it."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
BF = torch.bfloat16


def test_no_layers_hand_the_input_on(cuda):
    from dli_b200 import ops

    B, T, d, H, hd = 2, 5, 128, 2, 64
    rows = B * T
    h_in = torch.randn(rows, d, device=cuda).to(BF)
    h, x, attn, act = (torch.zeros(rows, d, device=cuda, dtype=BF) for _ in range(4))
    qkv = torch.zeros(rows, 3 * H * hd, device=cuda, dtype=BF)
    positions, seq_ids = (torch.zeros(rows, device=cuda, dtype=torch.int32) for _ in range(2))
    table = torch.zeros(B, 1, device=cuda, dtype=torch.int32)
    for src in (h_in, h):  # the second time in place
        out = ops.prompt_layers([], [], [], table, table, src, h, x, qkv, attn, act, None, None, positions, seq_ids, B, T,
                                None, H, H, hd, 1e-5, hd ** -0.5)
        assert out is h and torch.equal(h, h_in)
