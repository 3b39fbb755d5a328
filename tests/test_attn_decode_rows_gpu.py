"""Decode attention of large batches: sequences of every length around the tile, page and stage edges, each form of the
kernel (csrc/attn_decode.cu), against float64.  Bound: probabilities and the result are rounded to bf16 (2^-9 relative
each), sums are fp32, the online softmax's exponentials good to 2^-20."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
BF = torch.bfloat16


def _rope(x, c, s):
    a, b = x.chunk(2, dim=-1)
    r = lambda t: t.to(BF).float()  # noqa: E731
    return torch.cat((r(r(a * c) + r(-b * s)), r(r(b * c) + r(a * s))), dim=-1)


# (heads of 128: 2 stages x 6 warps up to 296 CTAs, 2 x 4 between; heads of 64: 2 x 8, then 3 x 4)
@pytest.mark.parametrize("hd,B,H,KV,page,window", [(128, 40, 16, 4, 16, 0), (128, 48, 8, 8, 8, 0), (128, 75, 8, 2, 64, 100),
                                                   (64, 40, 32, 4, 16, 0), (64, 80, 8, 8, 8, 33), (64, 50, 16, 16, 32, 0)])
def test_lengths_around_every_edge(cuda, hd, B, H, KV, page, window):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(B)
    edges = [1, 2, 15, 16, 17, 63, 64, 65, 95, 96, 97, 127, 128, 129, 191, 192, 193, 255, 256, 257, 288, 289, 300, 0, 511, 33]
    lens = [edges[i % len(edges)] for i in range(B)]
    top = max(lens)
    n = (top + page - 1) // page
    pool = B * n + 1
    kc = (1.3 * torch.randn(pool, KV, page, hd, device=cuda, generator=g)).to(BF)
    vc = torch.randn(pool, KV, page, hd, device=cuda, generator=g).to(BF)
    table = torch.randperm(pool, device=cuda, generator=g)[:B * n].int().view(B, n).contiguous()
    for b, L in enumerate(lens):  # nothing past a sequence's end may be read into the result
        if L % page:
            kc[table[b, L // page], :, L % page:] = float("nan")
            vc[table[b, L // page], :, L % page:] = float("inf")
    ang = 6.28 * torch.rand(top, hd // 2, device=cuda, generator=g)
    cos, sin = ang.cos().to(BF), ang.sin().to(BF)
    qkv = (1.3 * torch.randn(B, (H + 2 * KV) * hd, device=cuda, generator=g)).to(BF)
    out = torch.full((B, H * hd), 7.0, device=cuda, dtype=BF)
    k0, v0 = kc.clone(), vc.clone()
    ops.paged_attn_decode_fused(qkv, cos, sin, kc, vc, table, torch.tensor(lens, dtype=torch.int32, device=cuda), out, H, KV,
                                hd, hd ** -0.5, num_splits=1, window=window)
    for b, L in enumerate(lens):
        if L == 0:
            continue
        q, k, v = (x.view(-1, hd).float() for x in qkv[b].split([H * hd, KV * hd, KV * hd]))
        c, s = cos[L - 1].float(), sin[L - 1].float()
        q, k = _rope(q, c, s), _rope(k, c, s)
        at = (int(table[b, (L - 1) // page]), slice(None), (L - 1) % page)
        assert torch.equal(kc[at].float(), k) and torch.equal(vc[at].float(), v)
        k0[at], v0[at] = k.to(BF), v.to(BF)
        keys, vals = (x[table[b].long()].double().transpose(1, 2).reshape(n * page, KV, hd)[:L] for x in (kc, vc))
        lo = max(0, L - window) if window else 0
        keys, vals = keys[lo:], vals[lo:]
        p = torch.softmax(torch.einsum("gjd,tgd->gjt", q.double().view(KV, H // KV, hd), keys) * hd ** -0.5, dim=-1)
        ref = torch.einsum("gjt,tgd->gjd", p, vals).reshape(H * hd)
        mag = torch.einsum("gjt,tgd->gjd", p, vals.abs()).reshape(H * hd)
        assert ((out[b].double() - ref).abs() <= 2.0 ** -8 * (mag + ref.abs()) + 1e-6).all(), (b, L)
    assert torch.equal(torch.nan_to_num(kc, nan=9.0), torch.nan_to_num(k0, nan=9.0))  # only the new rows were written
    assert torch.equal(vc, v0)
