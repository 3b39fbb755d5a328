"""Key splits of ragged decode rows that add their sums over a cluster: numbers of splits around what a cluster may have (17: two
kernels), rows with fewer keys than splits, value sizes that the splits do not divide, against the row in one piece.  Bound: both
sum fp32 products of the same rounded keys, in other orders, and round once."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("splits", [2, 3, 8, 9, 12, 16, 17])
@pytest.mark.parametrize("D,V,H,G,extra", [(128, 128, 16, 4, "sink gate"), (64, 72, 6, 2, "turn"), (32, 512, 2, 2, "window sink"),
                                           (40, 2, 3, 3, "cap channel")])
def test_as_in_one_piece(cuda, D, V, H, G, extra, splits, dt):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(D + splits)
    rnd = lambda *s: torch.randn(*s, device=cuda, generator=g)  # noqa: E731
    lens, page = [333, 1, 5, 64], 16
    rows, per = len(lens), 22
    qbuf, proj = rnd(rows, H, D), rnd(rows, H * V + H + 3).to(dt)
    kc, vc = rnd(rows * per, G, page, D).to(dt), rnd(rows * per, G, page, V).to(dt)
    table = torch.randperm(rows * per, device=cuda, generator=g).int().view(rows, per)
    ent = torch.tensor([[r, r, 1, n - 1] for r, n in enumerate(lens)], device=cuda, dtype=torch.int32).view(-1)
    row_ent = torch.arange(rows, device=cuda).int()
    kw = {}
    if "sink" in extra:
        kw["sink"] = rnd(H)
    if "gate" in extra:
        kw["g_off"] = 2
    if "channel" in extra:
        kw.update(g_off=1, g_chan=True, cap=20.0)
    if "window" in extra:
        kw.update(window=40, first=3)
    if "turn" in extra:
        ang = rnd(400, V // 2)
        kw.update(cos_v=ang.cos().contiguous(), sin_v=ang.sin().contiguous())
    outs = []
    for n in (1, splits, splits):
        out = torch.full((rows, H * V), float("nan"), device=cuda, dtype=dt)
        part = torch.empty(rows * H * n * (V + 2), device=cuda) if n > 1 else None
        ops.attn_ragged(qbuf, kc, vc, proj, out, row_ent, ent, table, H, G, D, V, D ** -0.5, splits=n, part=part, **kw)
        outs.append(out.float())
    assert torch.equal(outs[1], outs[2])
    mag = vc.float().abs().amax() * (2 if "turn" in extra else 1)
    ulp = 2.0 ** -7 if dt == torch.bfloat16 else 2.0 ** -22
    assert ((outs[1] - outs[0]).abs() <= 2.0 ** -16 * mag + ulp * outs[0].abs()).all()
