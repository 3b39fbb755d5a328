"""Prompt attention with two query tiles per CTA (csrc/attn_prefill_streams.cu), at sizes where the rule takes it, against float64.

Bound per output: probabilities are rounded to bf16 (8 bits: 2^-8 relative each, the sum is of the unrounded ones), the output once more; the
fp32 scores move a probability by less than 2e-4 of itself."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
BF = torch.bfloat16


PROMPTS = [
    (1, 2048, 32, 8, 0),      # pairs of heads
    (1, 2177, 32, 32, 0),     # pairs of query tiles of one head, 18 tiles, one row in the last
    (1, 4097, 14, 2, 0),      # groups of 7: both kinds, 33 tiles: the last one alone
    (3, 1500, 32, 8, 0),      # rows behind a sequence are the next one's
    (1, 4000, 32, 8, 1000),   # windows: key tiles that only one of the two needs
    (1, 4224, 32, 32, 900),
]
CHUNKS = [(1, 1024, 3072, 32, 8, 16, 0), (2, 907, 1500, 32, 8, 8, 0), (4, 515, 1021, 32, 4, 128, 0), (2, 1025, 2047, 14, 2, 32, 0),
          (1, 2048, 2048, 32, 32, 16, 1100)]
# in a process of its own: a profile taken here would be one of several of a test run
ROUTE = """
import torch
from test_attn_streams_gpu import CHUNKS, PROMPTS
from dli_b200 import ops
z = lambda *s: torch.zeros(*s, device="cuda", dtype=torch.bfloat16)
with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as p:
    for hd in (64, 128):
        for B, T, H, KV, w in PROMPTS:
            ops.attn_prefill(z(B * T, (H + 2 * KV) * hd), z(B * T, H * hd), B, T, H, KV, hd, 1.0, w)
        for B, T, prefix, H, KV, page, w in CHUNKS:
            n = (prefix + T + page - 1) // page
            cache, table = z(B * n, KV, page, hd), torch.arange(B * n, device="cuda", dtype=torch.int32).view(B, n)
            ops.attn_prefill_paged(z(B * T, (H + 2 * KV) * hd), z(B * T, H * hd), cache, cache, table, B, T, prefix, H, KV, hd, 1.0, w)
    torch.cuda.synchronize()
print("streams", sum("attn_streams_kernel" in e.name for e in p.events()), "of", 2 * (len(PROMPTS) + len(CHUNKS)))
"""


def test_the_rule_takes_these_sizes(cuda):
    from dli_b200 import ops

    if ops.sm_count() != 148:
        pytest.skip("the rule counts SMs")
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([here, os.path.dirname(here), os.environ.get("PYTHONPATH", "")]))
    out = subprocess.run([sys.executable, "-c", ROUTE], env=env, capture_output=True, text=True, timeout=300)
    n = 2 * (len(PROMPTS) + len(CHUNKS))
    assert f"streams {n} of {n}" in out.stdout, out.stdout + out.stderr


def _check(out, q, k, v, rows, pos, window, H, KV):
    """out [R, H, hd] of query rows q [R, H, hd] at positions pos [R] over keys k, v [N, KV, hd]."""
    hd = q.shape[-1]
    for r, p in zip(rows, pos):
        lo = max(0, p - window + 1) if window else 0
        kk, vv = (t[lo:p + 1].double().repeat_interleave(H // KV, 1) for t in (k, v))
        w = torch.softmax(torch.einsum("hd,nhd->hn", q[r].double(), kk) * hd ** -0.5, -1)
        y, size = torch.einsum("hn,nhd->hd", w, vv), torch.einsum("hn,nhd->hd", w, vv.abs())
        bad = (out[r].double() - y).abs() > (2.0 ** -8 + 2e-4) * size + 2.0 ** -8 * 1.01 * y.abs() + 1e-6
        assert not bad.any(), (r, p, int(bad.sum()))


def _rows(T):
    return sorted({r for r in (0, 1, 63, 127, 128, 129, 255, 256, T // 2, T - 130, T - 129, T - 128, T - 2, T - 1) if 0 <= r < T})


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,T,H,KV,window", PROMPTS)
def test_prompt(cuda, hd, B, T, H, KV, window):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T + hd)
    qkv = torch.randn(B * T, (H + 2 * KV) * hd, device=cuda, generator=g).to(BF)
    qkv[:, :H * hd] *= 2  # maxima that move
    x = qkv.view(B, T, H + 2 * KV, hd)
    x[-1, T // 2:T // 2 + 3, H] *= 4
    out = torch.empty(B * T, H * hd, device=cuda, dtype=BF)
    run = lambda: ops.attn_prefill(qkv, out, B, T, H, KV, hd, hd ** -0.5, window)  # noqa: E731
    run()
    first = out.clone()
    run()
    assert torch.equal(out, first)
    for b in {0, B - 1}:
        rows = _rows(T)
        _check(out.view(B, T, H, hd)[b], x[b, :, :H], x[b, :, H:H + KV], x[b, :, H + KV:], rows, rows, window, H, KV)
    if B > 1:  # the values behind a sequence's end have probability 0, but may be anything
        clean = out.view(B, T, H, hd)[0].clone()
        x[1, :4, H + KV:] = float("inf")
        run()
        assert torch.equal(out.view(B, T, H, hd)[0], clean)


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("B,T,prefix,H,KV,page,window", CHUNKS)
def test_chunk(cuda, hd, B, T, prefix, H, KV, page, window):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T + prefix + hd)
    total = prefix + T
    per = (total + page - 1) // page
    k, v = (torch.randn(B, per * page, KV, hd, device=cuda, generator=g).to(BF) for _ in range(2))
    v[:, total:] = float("inf")  # the rest of the last page
    table = torch.randperm(B * per, device=cuda, generator=g).int().view(B, per)
    kc, vc = (torch.empty(B * per, KV, page, hd, device=cuda, dtype=BF) for _ in range(2))
    for c, t in ((kc, k), (vc, v)):
        c[table.long().view(-1)] = t.view(B * per, page, KV, hd).transpose(1, 2)
    qkv = torch.randn(B * T, (H + 2 * KV) * hd, device=cuda, generator=g).to(BF)
    out = torch.empty(B * T, H * hd, device=cuda, dtype=BF)
    run = lambda: ops.attn_prefill_paged(qkv, out, kc, vc, table, B, T, prefix, H, KV, hd, hd ** -0.5, window)  # noqa: E731
    run()
    for b in {0, B - 1}:
        rows = _rows(T)
        _check(out.view(B, T, H, hd)[b], qkv.view(B, T, H + 2 * KV, hd)[b, :, :H], k[b], v[b], rows, [prefix + r for r in rows], window, H, KV)
