"""The sampler's row split (csrc/sample.cu): rows of every size and alignment, ties, masked rows, k beyond the fast path.

The kept set is exact: tokens in descending order of the bf16 logit (ties by id), the top k with all ties at the k-th, then
those whose exclusive prefix sum of probabilities is below top_p.  Probabilities are fp32: __expf and sums of up to 2 048
terms, 1e-5 relative; a token whose prefix sum lies within 1e-5 of top_p may go either way."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
BF = torch.bfloat16
CAP = 2048


def _kept(row, top_k, top_p, t):
    x = row.double().cpu()
    order = torch.argsort(-x, stable=True)
    k = min(top_k, len(x)) if top_k else len(x)
    n = int((x >= x[order[k - 1]]).sum())
    order = order[:n]
    p = torch.softmax(x[order] / t, dim=0)
    before = torch.cumsum(p, 0) - p
    return order, p, before


def _check(logits, top_k=50, top_p=0.95, t=0.8):
    from dli_b200 import ops

    B, V = logits.shape
    seed = torch.tensor([7], dtype=torch.int64, device="cuda")
    step = torch.tensor([3], dtype=torch.int32, device="cuda")
    out, probs, ids = ops.sample(logits, temperature=t, top_k=top_k, top_p=top_p, seed=seed, step=step, debug_cap=CAP)
    again = ops.sample(logits, temperature=t, top_k=top_k, top_p=top_p, seed=seed, step=step)
    assert torch.equal(out, again)
    for b in range(B):
        order, p, before = _kept(logits[b], top_k, top_p, t)
        got = ids[b][ids[b] >= 0].long().cpu()
        n = len(got)
        assert n >= 1 and torch.equal(got, order[:n])
        assert n == 1 or before[n - 1] < top_p + 1e-5
        assert n == len(order) or before[n] > top_p - 1e-5
        torch.testing.assert_close(probs[b, :n].double().cpu(), p[:n] / p[:n].sum(), rtol=1e-4, atol=1e-7)
        assert int(out[b]) in got.tolist()


@pytest.mark.parametrize("V", [1, 7, 50, 65, 511, 4097, 16384, 16391, 32000, 50257, 128256, 131080, 262151])
def test_rows_of_every_size(cuda, V):
    g = torch.Generator(device="cuda").manual_seed(V)
    _check((2.5 * torch.randn(3, V, device=cuda, generator=g)).to(BF))


@pytest.mark.parametrize("stride,start", [(32003, 0), (32008, 1), (33001, 5)])
def test_rows_that_start_anywhere(cuda, stride, start):
    g = torch.Generator(device="cuda").manual_seed(stride)
    wide = (2.5 * torch.randn(4, stride, device=cuda, generator=g)).to(BF)
    _check(wide[:, start:start + 32000])


@pytest.mark.parametrize("top_k,top_p", [(1, 0.95), (512, 1.0), (513, 0.99), (2000, 1.0)])
def test_any_k(cuda, top_k, top_p):
    g = torch.Generator(device="cuda").manual_seed(top_k)
    # distinct values around the k-th (a permutation of all finite bf16 values above 1), so ties do not exceed the cap
    base = torch.arange(0x3F80, 0x3F80 + 8000, dtype=torch.int16, device=cuda).view(BF).float().log2().to(BF)
    V = 20000
    x = torch.full((2, V), -30.0, device=cuda, dtype=BF)
    for b in range(2):
        x[b, torch.randperm(V, device=cuda, generator=g)[:8000]] = base
    _check(x, top_k=top_k, top_p=top_p)


def test_ties_and_masks(cuda):
    V = 40000
    x = torch.full((5, V), -float("inf"), device=cuda, dtype=BF)
    x[0, [5, 39999, 17000]] = torch.tensor([1.0, 2.0, 2.0], device=cuda, dtype=BF)     # fewer than k finite logits
    x[1] = torch.finfo(BF).min
    x[1, 100:160] = 3.0                                                                  # 60 equal values above all
    x[2] = 0.0
    x[2, ::2] = -0.0
    x[2, 30000:30060] = 1.0
    x[3, :] = torch.linspace(-4, 4, V, device=cuda).to(BF)                               # long runs of equal values
    x[4, 8:16384:16] = 1.5                                                               # all in the first slice
    x[4, 20000] = 9.0
    from dli_b200 import ops
    for b, n in ((1, 60), (2, 60)):
        _check(x[b:b + 1], top_p=1.0)
    _check(x[3:4])
    _check(x[4:5], top_k=3)
    seed = torch.tensor([1], dtype=torch.int64, device=cuda)
    _, probs, ids = ops.sample(x[:1], top_k=50, top_p=1.0, seed=seed, debug_cap=64)
    got = ids[0][probs[0] > 0].tolist()
    assert got == [17000, 39999, 5]


def test_rows_keep_their_draws_in_any_batch(cuda):
    """A row's token depends on its own seed and step only; masked rows keep theirs."""
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(2)
    x = (2 * torch.randn(9, 50257, device=cuda, generator=g)).to(BF)
    seeds = torch.arange(9, device=cuda) + 11
    steps = torch.arange(9, device=cuda, dtype=torch.int32) * 3
    mask = torch.tensor([1, 0, 1, 1, 1, 0, 1, 1, 1], dtype=torch.int32, device=cuda)
    out = torch.full((9,), -5, dtype=torch.int32, device=cuda)
    ops.sample_rows(x, out, seeds, steps, mask)
    for b in range(9):
        one = torch.full((1,), -5, dtype=torch.int32, device=cuda)
        ops.sample_rows(x[b:b + 1], one, seeds[b:b + 1], steps[b:b + 1], mask[b:b + 1])
        assert int(one) == int(out[b])


@pytest.mark.parametrize("V", [16400, 50257, 128256])
def test_ctas_of_a_row_that_start_apart(cuda, V):
    """The CTAs of a cluster write into each other's shared memory: the same kept sets and tokens on a device whose SMs free up
    one by one (another stream keeps them busy with kernels of uneven length)."""
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(V)
    x = (2.5 * torch.randn(40, V, device=cuda, generator=g)).to(BF)
    seed = torch.tensor([5], dtype=torch.int64, device=cuda)
    want = ops.sample(x, seed=seed, debug_cap=64)
    other, load = torch.cuda.Stream(), [torch.randn(n, n, device=cuda) for n in (300, 900, 1700)]
    torch.cuda.synchronize()
    for _ in range(10):
        with torch.cuda.stream(other):
            for m in load:
                m @ m
        got = [ops.sample(x, seed=seed, debug_cap=64) for _ in range(4)]
        assert all(torch.equal(a, b) for r in got for a, b in zip(r, want))


@pytest.mark.parametrize("V,k", [(300, 300), (512, 512), (513, 512), (2048, 400), (2100, 128), (5000, 65), (5000, 129), (40000, 400),
                                 (128256, 200), (128256, 256), (262151, 200), (262151, 128)])
def test_either_side_of_the_rules(cuda, V, k):
    """k where candidates are put in order by counting, by the network, and where a row stays with one CTA."""
    g = torch.Generator(device="cuda").manual_seed(V + k)
    _check((2.5 * torch.randn(2, V, device=cuda, generator=g)).to(BF), top_k=k, top_p=1.0)


@pytest.mark.parametrize("zeros", [40, 150, 700])
def test_signed_zeros_and_nan(cuda, zeros):
    """-0 and 0 stand by token id (put in order by counting, by the network, with one CTA); a NaN before every number."""
    from dli_b200 import ops

    x = torch.full((1, 5000), -3.0, device=cuda, dtype=BF)
    x[0, 7:7 + zeros] = 0.0
    x[0, 8:7 + zeros:2] = -0.0
    x[0, [4000, 2, 3000]] = torch.tensor([-1.0, -1.5, 2.0], device=cuda, dtype=BF)
    _check(x, top_k=zeros + 3, top_p=1.0)
    x[0, 3] = float("nan")
    seed = torch.tensor([1], dtype=torch.int64, device=cuda)
    _, _, ids = ops.sample(x, top_k=zeros + 3, top_p=1.0, seed=seed, debug_cap=8)
    assert int(ids[0, 0]) == 3
