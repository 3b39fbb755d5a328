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


@pytest.fixture(scope="module")
def stages():
    from dli_b200.engine import ModelSpec, ShardEngine
    from oracle import decoder_ref as R

    spec = ModelSpec("llama", 3, 256, 4, 2, 64, 512, 512, 1e-5, 10000.0, 0, 128)
    sd = R.seeded_state_dict(R.ModelSpec(**spec.__dict__), seed=7, std=0.06)
    first, last = ShardEngine(spec, 0, 0, device="cuda:0", max_batch=2, max_seq_len=64), ShardEngine(
        spec, 1, 2, device="cuda:0", max_batch=2, max_seq_len=64)
    for e in (first, last):
        e.load_state_dict(sd)
    return first, last


def test_hidden_states_in_any_form(cuda, stages):
    """What a later stage is given: a buffer of its own, strided, unaligned, of another type, or the stage's own workspace
    under another shape — the same logits; a buffer that overlaps the workspace is refused as a copy of it always was."""
    first, last = stages
    B, T, d = 2, 11, 256
    for e in stages:
        e.start_batch(B, T, T + 4)
    ids = torch.randint(0, 512, (B * T,), device=cuda, dtype=torch.int32)
    hidden = first.prefill(B, T, ids=ids).clone()

    def logits(h):
        last.prefill(B, T, hidden=h)
        return last._state(B, 0)["logits"].clone()

    want, kept = logits(hidden), hidden.clone()
    assert torch.equal(hidden, kept)  # read only
    flat = torch.empty(B * T * d + 1, device=cuda, dtype=BF)
    flat[1:] = hidden.view(-1)
    wide = torch.zeros(B * T, 2 * d, device=cuda, dtype=BF)
    wide[:, ::2] = hidden
    forms = [flat[1:].view(B * T, d), wide[:, ::2], hidden.float()]
    own = last._h[:B * T]
    for h in forms + [own, own.view(B, T, d)]:
        if h.data_ptr() == own.data_ptr():
            own.copy_(hidden)
        assert torch.equal(logits(h), want)
    last._workspace(B * T + 1)
    with pytest.raises(RuntimeError):
        last.prefill(B, T, hidden=last._h[1:B * T + 1])


@pytest.mark.parametrize("name", ["llama", "gpt2"])
def test_rotation_as_a_kernel_of_its_own(cuda, monkeypatch, name):
    """DLI_FUSE_QKV_ROPE=0: one launch more per layer, the same caches and logits."""
    from dli_b200 import ops
    from dli_b200.engine import ModelSpec, ShardEngine
    from oracle import decoder_ref as R

    spec = ModelSpec("llama", 2, 256, 4, 2, 64, 512, 512, 1e-5, 10000.0, 0, 128) if name == "llama" else ModelSpec(
        "gpt2", 2, 256, 4, 4, 64, 1024, 512, 1e-5, 0.0, 0, 128, True)
    sd = R.seeded_state_dict(R.ModelSpec(**spec.__dict__), seed=3, std=0.06)
    B, T = 2, 21
    ids = torch.randint(0, 512, (B * T,), device=cuda, dtype=torch.int32)
    runs = []
    for switch in ("1", "0"):
        monkeypatch.setenv("DLI_FUSE_QKV_ROPE", switch)
        e = ShardEngine(spec, device="cuda:0", max_batch=B, max_seq_len=64)
        e.load_state_dict(sd)
        e.start_batch(B, T, T + 4)
        n0 = ops.launch_count
        e.prefill(B, T, ids=ids)
        runs.append((ops.launch_count - n0, [e._state(B, 0)["logits"].clone()] + [t.clone() for t in e.kv.k + e.kv.v]))
    assert runs[1][0] == runs[0][0] + spec.n_layers
    assert all(torch.equal(a, b) for a, b in zip(runs[0][1], runs[1][1]))


def test_buffers_that_are_too_small(cuda):
    """Refused on the host: nothing is launched on buffers that do not cover the prompts."""
    from dli_b200 import ops

    B, T, d, H, hd = 2, 5, 128, 2, 64
    rows = B * T
    mat = lambda n, w: torch.zeros(n, w, device=cuda, dtype=BF)  # noqa: E731
    ints = lambda *n: torch.zeros(*n, device=cuda, dtype=torch.int32)  # noqa: E731
    good = dict(layers=[], k_pools=[], v_pools=[], page_table=ints(B, 3), page_rows=ints(B, 3), h_in=mat(rows, d), h=mat(rows, d),
                x=mat(rows, d), qkv=mat(rows, 3 * H * hd), attn=mat(rows, H * hd), act=mat(rows, d), cos=None, sin=None,
                positions=ints(rows), seq_ids=ints(rows), B=B, T=T, prefix=None, H=H, KV=H, hd=hd, eps=1e-5, scale=0.125)
    ops.prompt_layers(**good)
    for bad in (dict(positions=ints(rows - 1)), dict(seq_ids=ints(rows - 1)), dict(page_rows=ints(B - 1, 3)),
                dict(page_rows=ints(B, 2)), dict(page_rows=ints(B * 3)), dict(layers=[{}]), dict(h_in=mat(rows + 1, d)),
                dict(qkv=mat(rows, 64)), dict(attn=mat(rows - 1, H * hd))):
        n0 = ops.launch_count
        with pytest.raises(ValueError):
            ops.prompt_layers(**{**good, **bad})
        assert ops.launch_count == n0
    with pytest.raises(ValueError):
        ops.prompt_rows(ints(rows), ints(rows - 1), None, B, T, 0, 0)
    with pytest.raises(ValueError):
        ops.prompt_rows(ints(rows), ints(rows), ints(B - 1), B, T, 0, 0)


@pytest.mark.parametrize("B,T,prefix,seq0", [(1, 1, 0, 0), (3, 7, 5, 6), (2, 200, 1000, 2)])
def test_prompt_rows(cuda, B, T, prefix, seq0):
    from dli_b200 import ops

    n = B * T
    pos, seq, last = (torch.full((n + 3,), -7, device=cuda, dtype=torch.int32) for _ in range(3))
    ops.prompt_rows(pos, seq, last, B, T, prefix, seq0)
    b, t = torch.arange(n, device=cuda) // T, torch.arange(n, device=cuda) % T
    assert torch.equal(pos[:n].long(), prefix + t) and torch.equal(seq[:n].long(), seq0 + b)
    assert torch.equal(last[:B].long(), (torch.arange(B, device=cuda) + 1) * T - 1)
    assert (pos[n:] == -7).all() and (seq[n:] == -7).all() and (last[B:] == -7).all()


def _shift(t, off):
    """The same values starting `off` elements into a buffer."""
    flat = torch.empty(t.numel() + off, device=t.device, dtype=t.dtype)
    flat[off:] = t.view(-1)
    return flat[off:].view(t.shape)


@pytest.mark.parametrize("arch,hd,H,KV,d,bias", [("llama", 64, 4, 2, 256, None), ("llama", 64, 3, 3, 768, 0), ("llama", 64, 32, 4, 2048, 1),
                                                 ("llama", 128, 3, 1, 512, None), ("llama", 128, 4, 2, 512, 0), ("llama", 128, 5, 1, 640, 3),
                                                 ("gpt2", 64, 12, 12, 768, 0), ("gpt2", 64, 4, 4, 256, 5), ("gpt2", 128, 2, 2, 256, 0)])
@pytest.mark.parametrize("B,T", [(1, 3), (1, 19), (2, 64), (2, 65), (1, 700), (3, 1400)])
def test_qkv_epilogue_equals_the_separate_steps(cuda, arch, hd, H, KV, d, bias, B, T):
    """Projection, rotation and cache append of a prompt pass against gemm + rope_kv_append: the same bits, with one and two
    heads per tile, an odd number of heads, a bias (aligned or not) and none, with rotation and without."""
    from dli_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(B * T + d)
    rnd = lambda *s, std=1.0: (std * torch.randn(*s, device=cuda, generator=g)).to(BF)  # noqa: E731
    rows, N, ff, page, prefix, pages = B * T, (H + 2 * KV) * hd, 256, 16, 5, (T + 5 + 15) // 16
    L = {"ln1": rnd(d), "ln2": rnd(d), "wqkv": rnd(N, d, std=0.05), "wo": rnd(d, H * hd, std=0.05), "wdown": rnd(d, ff, std=0.05)}
    if arch == "gpt2":
        L.update(ln1b=rnd(d), ln2b=rnd(d), wfc=rnd(ff, d, std=0.05))
    else:
        L.update(wgu=ops.pack_gate_up(rnd(ff, d, std=0.05), rnd(ff, d, std=0.05)))
    if bias is not None:
        L["bqkv"] = _shift(rnd(N), bias)
    cos = sin = None
    if arch == "llama":
        ang = torch.rand(T + prefix, hd // 2, device=cuda, generator=g) * 6.28
        cos, sin = ang.cos().to(BF), ang.sin().to(BF)
    table = torch.randperm((B + 1) * pages, device=cuda, generator=g).int().view(B + 1, pages)
    positions, seq_ids, last = (torch.empty(rows, device=cuda, dtype=torch.int32) for _ in range(3))
    ops.prompt_rows(positions, seq_ids, last, B, T, prefix, 1)
    h_in = rnd(rows, d)
    kc, vc = (torch.zeros((B + 1) * pages, KV, page, hd, device=cuda, dtype=BF) for _ in range(2))
    h, x, qkv, attn, act = (torch.empty(rows, w, device=cuda, dtype=BF) for w in (d, d, N, H * hd, ff))
    ops.prompt_layers([L], [kc], [vc], table, table[1:], h_in, h, x, qkv, attn, act, cos, sin, positions, seq_ids, B, T, prefix,
                      H, KV, hd, 1e-5, hd ** -0.5)
    if arch == "gpt2":
        ops.add_layernorm(h_in, L["ln1"], L["ln1b"], 1e-5, out=x)
    else:
        ops.add_rmsnorm(h_in, L["ln1"], 1e-5, out=x)
    want = ops.gemm(x, L["wqkv"], bias=L.get("bqkv"))
    k2, v2 = torch.zeros_like(kc), torch.zeros_like(vc)
    ops.rope_kv_append(want, cos, sin, positions, seq_ids, table, k2, v2, H, KV, hd)
    assert torch.equal(qkv, want) and torch.equal(kc, k2) and torch.equal(vc, v2)
    assert torch.isfinite(h.float()).all()
