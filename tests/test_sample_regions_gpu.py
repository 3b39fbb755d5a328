"""The sampler's clusters (csrc/sample.cu): their size follows the number of rows, the token does not; candidates that crowd one
CTA's region of the gathering; draws at the last kept token.  The kept set is checked as in test_sample_cluster_gpu.py."""
import pytest
from test_sample_cluster_gpu import BF, _check

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("V", [50257, 128256])
def test_a_rows_token_does_not_depend_on_the_batch(cuda, V):
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(V)
    x = (2.5 * torch.randn(150, V, device=cuda, generator=g)).to(BF)
    seeds = torch.arange(150, device=cuda) * 7919 + 1
    steps = torch.arange(150, device=cuda, dtype=torch.int32)
    tokens = lambda lo, n: ops.sample_rows(x[lo:lo + n], torch.zeros(n, dtype=torch.int32, device=cuda), seeds[lo:lo + n],  # noqa: E731
                                           steps[lo:lo + n])
    one = torch.cat([tokens(i, 1) for i in range(150)])
    for n in (2, 17, 31, 40, 67, 75, 149):
        assert torch.equal(torch.cat([tokens(i, min(n, 150 - i)) for i in range(0, 150, n)]), one)


@pytest.mark.parametrize("crowd", [60, 500, 520, 2100])
@pytest.mark.parametrize("at", [0, 70003])
def test_candidates_in_one_place(cuda, crowd, at):
    """`crowd` neighbouring logits above all others, equal in groups: more than a region holds, or a row's candidates."""
    g = torch.Generator(device="cuda").manual_seed(crowd)
    x = torch.randn(2, 128256, device=cuda, generator=g)
    x[:, at:at + crowd] = 9.0 + (torch.arange(crowd, device=cuda) % 7) * 0.0625
    _check(x.to(BF), top_p=1.0)
    _check(x.to(BF), top_k=400)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65])
def test_a_few_tokens_left(cuda, n):
    """As many kept tokens as one warp holds, and one more, over the draws of 400 seeds: tokens of probability 0.6 / n and more, so
    that all but a few are drawn (expected to miss: n e^(-240/n), 1.6 of 65)."""
    from dli_b200 import ops

    x = torch.full((1, 4000), -30.0, device=cuda)
    x[0, torch.arange(n, device=cuda) * 50 + 3] = torch.linspace(2.0, 2.5, n, device=cuda)
    x = x.to(BF)
    _check(x, top_k=n, top_p=1.0)
    out = torch.full((400,), -1, dtype=torch.int32, device=cuda)
    ops.sample_rows(x.repeat(400, 1), out, torch.arange(400, device=cuda), torch.zeros(400, dtype=torch.int32, device=cuda), top_k=n,
                    top_p=1.0)
    drawn = set(out.tolist())
    assert all((i - 3) % 50 == 0 and (i - 3) // 50 < n for i in drawn)
    assert len(drawn) >= n - 10


@pytest.mark.parametrize("V", [300, 512, 513, 1000, 1024, 1025, 1500, 2000, 2048])
def test_every_number_of_keys_a_thread(cuda, V):
    """Short rows are candidates as a whole: one to four keys a thread in the search for the threshold, full and not."""
    g = torch.Generator(device="cuda").manual_seed(V)
    x = torch.randn(3, V, device=cuda, generator=g).to(BF)
    for k in (1, 257, 300):
        _check(x, top_k=min(k, V), top_p=1.0)
