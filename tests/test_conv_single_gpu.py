"""The decode form of post-norm + add + norm + input convolution: equal to the separate steps, and to itself whatever the
launch before it still writes (programmatic dependent launch on, as engines have it)."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.fixture(autouse=True)
def _pdl():
    from dli_b200 import ops

    before = ops.set_pdl(True)
    yield
    ops.set_pdl(before)


def _state(rows, d, taps, dt, seed, slots=7):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape):
        return torch.randn(*shape, device="cuda", generator=g)

    slot = torch.randperm(slots, device="cuda", generator=g)[:rows].int()
    ent = torch.stack([slot, torch.arange(rows, device="cuda").int(), torch.ones_like(slot),
                       torch.arange(rows, device="cuda").int()], dim=1).contiguous().view(-1)  # positions 0 ..: short tails too
    return randn(rows, d).to(dt), 3 * randn(rows, d), randn(slots, max(taps - 1, 1), d), randn(d, taps), ent


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("d", [8, 1000, 2048, 4096, 4100])
@pytest.mark.parametrize("taps", [2, 4, 5])
@pytest.mark.parametrize("post", [True, False])
def test_equals_the_separate_steps(cuda, d, taps, post, dt):
    """Bound: fp32 sums of d squares and of the taps, the result rounded to the element type."""
    from dli_b200 import ops

    rows = 5
    y, x, tail, w, ent = _state(rows, d, taps, dt, d + taps)
    row_ent = torch.arange(rows, device="cuda").int()
    x2, t2, hn, want = x.clone(), tail.clone(), torch.empty_like(x), torch.empty_like(y)
    if post:
        ops.postnorm_add_norm(y, x2, 0.7, 1e-5, hn, 1.3)
    else:
        ops.scalar_rmsnorm(x2, 1.3, 1e-5, hn)
    ops.causal_conv_ragged(hn, t2, w, row_ent, ent, want)
    mag = hn.abs().amax(0) * w.abs().sum(1) + tail.abs().amax((0, 1)) * w.abs().sum(1) + hn.abs().amax(0)
    for ahead in (False, True):
        torch.cuda.synchronize()  # nothing before it writes what `ahead` reads early
        xa, ta, out = x.clone(), tail.clone(), torch.empty_like(y)
        torch.cuda.synchronize()
        ops.postnorm_add_norm_conv_single(y if post else None, xa, ta, w, ent, out, 0.7, 1.3, 1e-5, ahead=ahead)
        step = 2.0 ** -18 * mag
        assert ((xa - x2).abs() <= 2.0 ** -20 * (x2.abs() + 1)).all()
        assert ((ta - t2).abs() <= 2.0 ** -18 * (t2.abs() + hn.abs().amax() * 2.0 ** -4)).all()
        ulp = 2.0 ** -7 if dt == torch.bfloat16 else 2.0 ** -22
        assert ((out.float() - want.float()).abs() <= step + ulp * want.float().abs()).all()


@pytest.mark.parametrize("d,taps", [(2048, 4), (1000, 3), (4096, 2)])
@pytest.mark.parametrize("post", [True, False])
def test_calls_in_a_row_on_the_same_slots(cuda, d, taps, post):
    """Every call reads the tail and the row of x that the launch just before it writes: the same as with the stream
    drained in between."""
    from dli_b200 import ops

    rows, steps = 3, 40
    y, x, tail, w, ent = _state(rows, d, taps, torch.float32, d)
    ent.view(rows, 4)[:, 3] += taps  # every tail entry counts
    runs = []
    for wait in (True, False):
        xa, ta, outs = x.clone(), tail.clone(), [torch.empty_like(y) for _ in range(steps)]
        torch.cuda.synchronize()
        for out in outs:
            ops.postnorm_add_norm_conv_single(y if post else None, xa, ta, w, ent, out, 0.7, 1.3, 1e-5)
            if wait:
                torch.cuda.synchronize()
        runs.append(outs + [xa, ta])
    assert all(torch.equal(a, b) for a, b in zip(*runs))


@pytest.mark.parametrize("n", [1, 3])
def test_right_after_the_convolution_that_writes_its_tail(cuda, n):
    """A portion of n rows per sequence through causal_conv_ragged, then a decode row on the same tails."""
    from dli_b200 import ops

    rows, d, taps = 3, 2048, 4
    y, x, tail, w, ent = _state(rows, d, taps, torch.float32, n)
    ent.view(rows, 4)[:, 3] += 9
    first = ent.clone().view(rows, 4)
    first[:, 1], first[:, 2], first[:, 3] = torch.arange(rows, device="cuda") * n, n, first[:, 3] - n
    first = first.contiguous().view(-1)
    row_ent = torch.arange(rows, device="cuda").int().repeat_interleave(n).contiguous()
    h = torch.randn(rows * n, d, device="cuda")
    runs = []
    for wait in (True, False):
        for _ in range(20):
            xa, ta, mid, out = x.clone(), tail.clone(), torch.empty_like(h), torch.empty_like(y)
            torch.cuda.synchronize()
            ops.causal_conv_ragged(h, ta, w, row_ent, first, mid)
            if wait:
                torch.cuda.synchronize()
            ops.postnorm_add_norm_conv_single(y, xa, ta, w, ent, out, 0.7, 1.3, 1e-5)
            runs.append([mid, out, xa, ta])
    assert all(torch.equal(a, b) for r in runs[1:] for a, b in zip(runs[0], r))


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("d", [4, 72, 1024, 1028, 2052])
def test_four_channels_a_thread_as_one(cuda, d, dt):
    """The 16-byte form of the input convolution and the scalar one (which a tail that starts off 16 bytes takes): the same
    bits, in portions shorter and longer than the taps, at a sequence's start and later."""
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(d)
    ns, starts = [1, 2, 9, 40, 3], [0, 1, 0, 77, 2]
    rows, at, ent, row_ent = sum(ns), 0, [], []
    for i, (n, s) in enumerate(zip(ns, starts)):
        ent += [len(ns) - 1 - i, at, n, s]
        row_ent += [i] * n
        at += n
    ent, row_ent = (torch.tensor(v, device=cuda, dtype=torch.int32) for v in (ent, row_ent))
    h, w = torch.randn(rows, d, device=cuda, generator=g), torch.randn(d, 4, device=cuda, generator=g)
    tail = torch.randn(len(ns), 3, d, device=cuda, generator=g)
    flat = torch.empty(tail.numel() + 1, device=cuda)
    flat[1:] = tail.view(-1)
    outs = []
    for t in (tail, flat[1:].view_as(tail)):
        out = torch.full((rows, d), float("nan"), device=cuda, dtype=dt)
        ops.causal_conv_ragged(h, t, w, row_ent, ent, out)
        outs.append((out, t))
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
