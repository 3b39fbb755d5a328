"""Prompt attention at head size 64 on the tcgen05 kernel (and both head sizes on either side of the kernel rule) against
float64.  Bound: the probabilities are rounded to bf16 (2^-9 each, relative), sums are fp32, the result is rounded to bf16
once: 2^-9 sum |p v| / l + 2^-9 |out|, the exponential's 2^-20 beside it."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
BF = torch.bfloat16


def _ref(q, k, v, scale, prefix, window):
    T, S = q.shape[0], k.shape[0]
    i = torch.arange(T, device=q.device)[:, None] + prefix
    j = torch.arange(S, device=q.device)[None]
    hide = (j > i) | ((j <= i - window) if window else torch.zeros_like(j > i))
    p = torch.softmax((q @ k.T * scale).masked_fill(hide, -float("inf")), dim=-1)
    return p @ v, p @ v.abs()


def _check(out, q, k, v, H, KV, hd, prefix, window):
    for h in range(H):
        ref, mag = _ref(q[:, h], k[:, h * KV // H], v[:, h * KV // H], hd ** -0.5, prefix, window)
        bound = 2.0 ** -8 * (mag + ref.abs()) + 1e-6
        assert ((out[:, h] - ref).abs() <= bound).all()


@pytest.mark.parametrize("hd,B,T,H,KV,window", [(64, 1, 447, 4, 2, 0), (64, 1, 448, 4, 1, 0), (64, 2, 513, 3, 3, 0),
                                                (64, 1, 1777, 2, 1, 300), (64, 3, 640, 12, 12, 0), (128, 2, 64, 4, 2, 0),
                                                (128, 2, 65, 4, 2, 0), (64, 1, 2, 2, 2, 0)])
def test_whole_prompts(cuda, hd, B, T, H, KV, window):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T + hd)
    qkv = (1.3 * torch.randn(B * T, (H + 2 * KV) * hd, device=cuda, generator=g)).to(BF)
    out = torch.full((B * T, H * hd), float("nan"), device=cuda, dtype=BF)
    ops.attn_prefill(qkv, out, B, T, H, KV, hd, hd ** -0.5, window=window)
    q, k, v = (x.double().view(B, T, -1, hd) for x in qkv.split([H * hd, KV * hd, KV * hd], dim=1))
    for b in range(B):
        _check(out.double().view(B, T, H, hd)[b], q[b], k[b], v[b], H, KV, hd, 0, window)


@pytest.mark.parametrize("hd,B,T,prefix,H,KV,page,window", [(64, 2, 100, 400, 4, 2, 16, 0), (64, 1, 3, 1000, 2, 1, 8, 0),
                                                             (64, 1, 300, 148, 3, 3, 64, 0), (64, 2, 130, 900, 4, 1, 16, 257),
                                                             (64, 1, 40, 407, 2, 2, 16, 0), (128, 1, 20, 44, 4, 2, 16, 0),
                                                             (128, 1, 20, 45, 4, 2, 16, 0)])
def test_chunks_on_the_paged_cache(cuda, hd, B, T, prefix, H, KV, page, window):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T + prefix)
    S = prefix + T
    n = (S + page - 1) // page
    kc = (1.3 * torch.randn(B * n + 2, KV, page, hd, device=cuda, generator=g)).to(BF)
    vc = torch.randn(B * n + 2, KV, page, hd, device=cuda, generator=g).to(BF)
    table = torch.randperm(B * n + 2, device=cuda, generator=g)[:B * n].int().view(B, n).contiguous()
    for b in range(B):  # what lies past the context in its last page must not matter
        if S % page:
            kc[table[b, -1], :, S % page:], vc[table[b, -1], :, S % page:] = float("nan"), float("inf")
    qkv = (1.3 * torch.randn(B * T, (H + 2 * KV) * hd, device=cuda, generator=g)).to(BF)
    out = torch.full((B * T, H * hd), float("nan"), device=cuda, dtype=BF)
    ops.attn_prefill_paged(qkv, out, kc, vc, table, B, T, prefix, H, KV, hd, hd ** -0.5, window=window)
    q = qkv[:, :H * hd].double().view(B, T, H, hd)
    for b in range(B):
        k, v = (c[table[b].long()].double().transpose(1, 2).reshape(n * page, KV, hd)[:S] for c in (kc, vc))
        _check(out.double().view(B, T, H, hd)[b], q[b], k, v, H, KV, hd, prefix, window)


@pytest.mark.parametrize("hd,T", [(64, 450), (128, 130), (64, 40), (128, 40)])
def test_a_sequence_does_not_see_its_neighbour(cuda, hd, T):
    """The tile after a sequence's last row holds the next sequence's keys and values: infinities there stay there."""
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T)
    H = KV = 2
    qkv = torch.randn(2 * T, 3 * H * hd, device=cuda, generator=g).to(BF)
    alone, both = torch.empty(T, H * hd, device=cuda, dtype=BF), torch.empty(2 * T, H * hd, device=cuda, dtype=BF)
    ops.attn_prefill(qkv[:T].contiguous(), alone, 1, T, H, KV, hd, hd ** -0.5)
    qkv[T:, H * hd:] = float("inf")
    ops.attn_prefill(qkv, both, 2, T, H, KV, hd, hd ** -0.5)
    assert torch.equal(both[:T], alone)


@pytest.mark.parametrize("hd,T", [(64, 1100), (64, 1777), (128, 130)])
def test_the_caller_chooses_the_kernel(cuda, monkeypatch, hd, T):
    """tensor_core=False is the mma.sync kernel at either head size, whatever the rule says, and DLI_PREFILL_ATTN is looked up
    at every call.  The kernels tile the keys differently, so their bits differ: that tells them apart."""
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T)
    H, KV, page = 4, 2, 16
    n = (T + page - 1) // page
    qkv = (1.3 * torch.randn(T, (H + 2 * KV) * hd, device=cuda, generator=g)).to(BF)
    kc, vc = (c.reshape(T, KV, hd) for c in qkv[:, H * hd:].split([KV * hd, KV * hd], dim=1))
    kc, vc = (torch.nn.functional.pad(c, (0, 0, 0, 0, 0, n * page - T)).view(n, page, KV, hd).transpose(1, 2).contiguous()
              for c in (kc, vc))
    table = torch.arange(n, device=cuda).int().view(1, n)

    def whole(choice):
        return ops.attn_prefill(qkv, torch.empty(T, H * hd, device=cuda, dtype=BF), 1, T, H, KV, hd, hd ** -0.5,
                                tensor_core=choice).clone()

    def chunk():
        return ops.attn_prefill_paged(qkv, torch.empty(T, H * hd, device=cuda, dtype=BF), kc, vc, table, 1, T, 0, H, KV, hd,
                                      hd ** -0.5).clone()

    monkeypatch.delenv("DLI_PREFILL_ATTN", raising=False)
    by_rule, mma, paged = whole(None), whole(False), chunk()
    assert not torch.equal(by_rule, mma) and torch.equal(by_rule, paged)
    monkeypatch.setenv("DLI_PREFILL_ATTN", "mma")
    assert torch.equal(whole(None), mma) and torch.equal(chunk(), mma)
    monkeypatch.delenv("DLI_PREFILL_ATTN")
    assert torch.equal(whole(None), by_rule) and torch.equal(chunk(), paged)


@pytest.mark.parametrize("B,T,H,KV,window", [(1, 1025, 2, 1, 0), (1, 1151, 4, 2, 0), (2, 1280, 3, 3, 0), (8, 1025, 2, 2, 257),
                                             (1, 1777, 2, 1, 1000), (3, 450, 12, 12, 0), (16, 512, 8, 8, 0)])
def test_whole_prompts_of_head_size_64_on_tcgen05(cuda, B, T, H, KV, window):
    """Sizes that the rule gives to the tcgen05 kernel (its bits are not those of the mma.sync kernel)."""
    from dli_b200 import ops

    hd, g = 64, torch.Generator(device="cuda").manual_seed(T + B)
    qkv = (1.3 * torch.randn(B * T, (H + 2 * KV) * hd, device=cuda, generator=g)).to(BF)
    out, mma = (torch.full((B * T, H * hd), float("nan"), device=cuda, dtype=BF) for _ in range(2))
    ops.attn_prefill(qkv, out, B, T, H, KV, hd, hd ** -0.5, window=window)
    ops.attn_prefill(qkv, mma, B, T, H, KV, hd, hd ** -0.5, window=window, tensor_core=False)
    assert not torch.equal(out, mma)
    q, k, v = (x.double().view(B, T, -1, hd) for x in qkv.split([H * hd, KV * hd, KV * hd], dim=1))
    for b in range(B):
        for o in (out, mma):
            _check(o.double().view(B, T, H, hd)[b], q[b], k[b], v[b], H, KV, hd, 0, window)


@pytest.mark.parametrize("B,T,prefix,H,KV,page,window", [(1, 1, 1000, 2, 1, 8, 0), (2, 100, 900, 2, 2, 16, 0), (1, 100, 900, 2, 2, 64, 600),
                                                         (2, 40, 900, 3, 3, 16, 0), (2, 513, 407, 2, 2, 32, 0), (1, 130, 2000, 4, 2, 16, 0),
                                                         (4, 100, 407, 32, 8, 16, 600), (1, 3, 2000, 2, 2, 128, 0)])
def test_chunks_of_head_size_64_on_tcgen05(cuda, monkeypatch, B, T, prefix, H, KV, page, window):
    from dli_b200 import ops

    hd, g = 64, torch.Generator(device="cuda").manual_seed(T + prefix)
    S = prefix + T
    n = (S + page - 1) // page
    kc = (1.3 * torch.randn(B * n + 2, KV, page, hd, device=cuda, generator=g)).to(BF)
    vc = torch.randn(B * n + 2, KV, page, hd, device=cuda, generator=g).to(BF)
    table = torch.randperm(B * n + 2, device=cuda, generator=g)[:B * n].int().view(B, n).contiguous()
    for b in range(B):
        if S % page:
            kc[table[b, -1], :, S % page:], vc[table[b, -1], :, S % page:] = float("nan"), float("inf")
    qkv = (1.3 * torch.randn(B * T, (H + 2 * KV) * hd, device=cuda, generator=g)).to(BF)
    outs = []
    for choice in ("tc", "mma"):
        monkeypatch.setenv("DLI_PREFILL_ATTN", choice)
        outs.append(torch.full((B * T, H * hd), float("nan"), device=cuda, dtype=BF))
        ops.attn_prefill_paged(qkv, outs[-1], kc, vc, table, B, T, prefix, H, KV, hd, hd ** -0.5, window=window)
    assert not torch.equal(*outs)
    q = qkv[:, :H * hd].double().view(B, T, H, hd)
    for b in range(B):
        k, v = (c[table[b].long()].double().transpose(1, 2).reshape(n * page, KV, hd)[:S] for c in (kc, vc))
        for o in outs:
            _check(o.double().view(B, T, H, hd)[b], q[b], k, v, H, KV, hd, prefix, window)


@pytest.mark.parametrize("T", [1030, 1800])
def test_long_prompts_of_head_size_64_do_not_see_their_neighbours(cuda, T):
    test_a_sequence_does_not_see_its_neighbour(cuda, 64, T)
