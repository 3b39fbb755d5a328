"""The work this framework is timed on: what serving a decoder on one GPU has it do, through its public entry points.

A uniform stack (Llama / Mistral / TinyLlama / GPT-2 shapes) spends its time in prompt passes through a shard's layers,
in the kernels of a batched decode step, in the sampler and, at batch 1, in whole `generate` calls; the layer-by-layer
family spends it in ragged steps.  The sizes are those of the named specs of the engine and of the benchmark.

Weights and inputs are random: weights with the standard deviation of a fresh initialisation (0.02), hidden states of
unit size as a normed residual stream has them, logits with a few tokens far above the rest as a trained model gives.
"""
import math

import numpy as np
import torch

from dli_b200 import ops, sokevik
from dli_b200.engine import NAMED_SPECS, ModelSpec, ShardEngine, rope_tables
from dli_b200.ragged_engine import RaggedEngine

BF = torch.bfloat16
F64 = torch.float64
DEV = "cuda"
PAGE = 16  # tokens per cache page: the engines' default


# ---------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # the token of one request: the default /inference call samples (temperature 0.8, top-k 50, top-p 0.95)
        {"name": "sample_one", "kind": "sample", "rows": 1, "vocab": 128256},
        # the tokens of a full continuous batch, each row with its own request's seed
        {"name": "sample_batch", "kind": "sample", "rows": 48, "vocab": 128256},
        # a one-line question through two layers of an 8B shard: few rows, the weights are the cost
        {"name": "prompt_short", "kind": "prompt", "spec": "llama-3-8b", "layers": 2, "batch": 1, "tokens": 19, "chunk": 0},
        # a chat turn of a few hundred tokens, an odd count
        {"name": "prompt_chat", "kind": "prompt", "spec": "llama-3-8b", "layers": 2, "batch": 1, "tokens": 301, "chunk": 0},
        # two 2k prompts at once: the benchmark's context, the largest prompt pass
        {"name": "prompt_long", "kind": "prompt", "spec": "llama-3-8b", "layers": 2, "batch": 2, "tokens": 2048, "chunk": 0},
        # a document fed in chunks past the sliding window, the last chunk ragged
        {"name": "prompt_chunks", "kind": "prompt", "spec": "mistral-7b", "layers": 1, "batch": 1, "tokens": 5003, "chunk": 1024},
        # a smaller model (head size 64) at an odd prompt length
        {"name": "prompt_tiny", "kind": "prompt", "spec": "tinyllama-1.1b", "layers": 4, "batch": 1, "tokens": 1777, "chunk": 0},
        # the reference's default model: LayerNorm, biases, GELU, head size 64, three prompts together
        {"name": "prompt_gpt2", "kind": "prompt", "spec": "gpt2", "layers": 4, "batch": 3, "tokens": 450, "chunk": 0},
        # attention of a batched decode step: 32 sequences of different lengths up to 2k on the paged cache
        {"name": "attention_decode", "kind": "attention", "spec": "llama-3-8b", "rows": 32, "max_len": 2048, "window": 0},
        # everything after the attention of a batched decode step: output projection, norm, gated feed-forward
        {"name": "mlp_decode", "kind": "mlp", "spec": "llama-3-8b", "rows": 24},
        # one whole request on the smaller model, the reference's default sampling call
        {"name": "generate", "kind": "generate", "spec": "tinyllama-1.1b", "batch": 1, "tokens": 100, "new": 40},
        # the layer-by-layer family: portions of three prompts, then decode steps of all three
        {"name": "ragged", "kind": "ragged", "rows": 3, "max_len": 333, "steps": 6},
    ]


def draw(rng):
    """One more case of the same ranges."""
    def span(lo, hi):
        return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))

    kind = rng.choice(["sample", "prompt", "prompt", "prompt", "attention", "mlp", "generate", "ragged"])
    if kind == "sample":
        return {"kind": kind, "rows": span(1, 64), "vocab": rng.choice([32000, 50257, 128256])}
    if kind == "prompt":
        name = rng.choice(["llama-3-8b", "llama-3-8b", "mistral-7b", "tinyllama-1.1b", "gpt2"])
        longest = 1024 if name == "gpt2" else 2048 if name == "tinyllama-1.1b" else 4096
        tokens = span(2, longest)
        batch = min(span(1, 8), max(1, 4096 // tokens))
        chunk = rng.choice([512, 1000, 2048]) if rng.random() < 0.25 else 0
        return {"kind": kind, "spec": name, "layers": rng.choice([1, 2]), "batch": batch, "tokens": tokens,
                "chunk": chunk if chunk < tokens else 0}
    if kind == "attention":
        name = rng.choice(["llama-3-8b", "llama-3-8b", "mistral-7b", "tinyllama-1.1b"])
        rows = span(1, 64)
        return {"kind": kind, "spec": name, "rows": rows, "max_len": span(40, min(4096, 65536 // rows)),
                "window": rng.choice([0, 0, 1000])}
    if kind == "mlp":
        return {"kind": kind, "spec": rng.choice(["llama-3-8b", "mistral-7b", "tinyllama-1.1b"]), "rows": span(3, 128)}
    if kind == "generate":
        batch = span(1, 16)
        return {"kind": kind, "spec": "tinyllama-1.1b", "batch": batch, "tokens": span(4, 1024 // batch + 4),
                "new": span(4, 40)}
    return {"kind": kind, "rows": rng.randint(1, 4), "max_len": span(2, 400), "steps": rng.randint(1, 8)}


# ---------------------------------------------------------------------------------------------- inputs
def _gen(seed, tag):
    return torch.Generator(device=DEV).manual_seed(seed * 1009 + tag)


def _normal(g, *shape, std=1.0, mean=0.0):
    return (mean + std * torch.randn(*shape, device=DEV, generator=g)).to(BF)


def _lengths(case):
    """Lengths of a batch of sequences, spread between an eighth of the longest and it (a decode batch: the new token
    included)."""
    n, top = case["rows"], case["max_len"]
    return [top - (i * 7919 % n) * (top - max(1, top // 8)) // n for i in range(n)]


def _spec(case):
    return NAMED_SPECS[case["spec"]]


def _shard_spec(case):
    """A stack with one layer before and one after the shard's: the shard takes and returns hidden states."""
    return ModelSpec(**{**_spec(case).__dict__, "n_layers": case["layers"] + 2})


def _layer_weights(spec, i, seed):
    """One layer's tensors under the checkpoint's names, bf16 on the GPU."""
    g, d, hd, ff = _gen(seed, 10 + i), spec.d_model, spec.head_dim, spec.d_ff
    if spec.arch == "gpt2":
        p = f"transformer.h.{i}."
        sd = {}
        for n in ("ln_1", "ln_2"):
            sd[p + n + ".weight"], sd[p + n + ".bias"] = _normal(g, d, std=0.1, mean=1.0), _normal(g, d, std=0.05)
        for n, a, b in (("attn.c_attn", d, 3 * d), ("attn.c_proj", d, d), ("mlp.c_fc", d, ff), ("mlp.c_proj", ff, d)):
            sd[p + n + ".weight"], sd[p + n + ".bias"] = _normal(g, a, b, std=0.04), _normal(g, b, std=0.05)
        return sd
    p, kv = f"model.layers.{i}.", spec.n_kv_heads * hd
    return {p + "input_layernorm.weight": _normal(g, d, std=0.1, mean=1.0),
            p + "post_attention_layernorm.weight": _normal(g, d, std=0.1, mean=1.0),
            p + "self_attn.q_proj.weight": _normal(g, spec.n_heads * hd, d, std=0.02),
            p + "self_attn.k_proj.weight": _normal(g, kv, d, std=0.02),
            p + "self_attn.v_proj.weight": _normal(g, kv, d, std=0.02),
            p + "self_attn.o_proj.weight": _normal(g, d, spec.n_heads * hd, std=0.02),
            p + "mlp.gate_proj.weight": _normal(g, ff, d, std=0.02),
            p + "mlp.up_proj.weight": _normal(g, ff, d, std=0.02),
            p + "mlp.down_proj.weight": _normal(g, d, ff, std=0.02)}


def _prompt_inputs(case, seed):
    spec = _shard_spec(case)
    sd = {}
    for i in range(1, case["layers"] + 1):
        sd.update(_layer_weights(spec, i, seed))
    return spec, sd, _normal(_gen(seed, 1), case["batch"] * case["tokens"], spec.d_model)


def _attention_inputs(case, seed):
    spec, g = _spec(case), _gen(seed, 2)
    lens = _lengths(case)
    pages = [(n + PAGE - 1) // PAGE for n in lens]
    pool = sum(pages)
    table = torch.zeros(case["rows"], max(pages), dtype=torch.int32)
    order = torch.randperm(pool, generator=torch.Generator().manual_seed(seed)).to(torch.int32)
    at = 0
    for b, n in enumerate(pages):
        table[b, :n] = order[at:at + n]
        at += n
    shape = (pool, spec.n_kv_heads, PAGE, spec.head_dim)
    width = (spec.n_heads + 2 * spec.n_kv_heads) * spec.head_dim
    return {"k": _normal(g, *shape, std=1.2), "v": _normal(g, *shape, std=1.2),
            "qkv": _normal(g, case["rows"], width, std=1.2), "table": table.to(DEV),
            "lens": torch.tensor(lens, dtype=torch.int32, device=DEV), "pages": pages}


def _mlp_inputs(case, seed):
    spec, g = _spec(case), _gen(seed, 3)
    d, ff, n = spec.d_model, spec.d_ff, case["rows"]
    return {"attn": _normal(g, n, spec.n_heads * spec.head_dim, std=0.3), "h": _normal(g, n, d),
            "ln": _normal(g, d, std=0.1, mean=1.0), "wo": _normal(g, d, spec.n_heads * spec.head_dim, std=0.02),
            "gate": _normal(g, ff, d, std=0.02), "up": _normal(g, ff, d, std=0.02), "down": _normal(g, d, ff, std=0.02)}


def _sample_inputs(case, seed):
    g = _gen(seed, 4)
    n, V = case["rows"], case["vocab"]
    x = 1.5 * torch.randn(n, V, device=DEV, generator=g)
    top = torch.randint(0, V, (n, 12), device=DEV, generator=g)
    x.scatter_add_(1, top, 6.0 + 2.0 * torch.randn(n, 12, device=DEV, generator=g))
    seeds = torch.randint(0, 1 << 31, (n,), generator=torch.Generator().manual_seed(seed))
    steps = torch.randint(0, 4096, (n,), generator=torch.Generator().manual_seed(seed + 1)).to(torch.int32)
    return x.to(BF), seeds, steps


def _generate_inputs(case, seed):
    """A model whose next token stands well above the rest, as a trained one's does: the head is the embedding under a
    permutation of the tokens, the layers add to it.  Projections back to the residual stream are smaller, as usual."""
    spec = _spec(case)
    sd = {}
    for i in range(spec.n_layers):
        sd.update(_layer_weights(spec, i, seed))
        for n in ("self_attn.o_proj", "mlp.down_proj"):
            sd[f"model.layers.{i}.{n}.weight"] *= 0.5
    g = _gen(seed, 5)
    embed = torch.randn(spec.vocab, spec.d_model, device=DEV, generator=g)
    perm = torch.randperm(spec.vocab, device=DEV, generator=g)
    head = torch.empty_like(embed)
    head[perm] = 0.02 * embed
    sd["model.embed_tokens.weight"], sd["lm_head.weight"] = embed.to(BF), head.to(BF)
    sd["model.norm.weight"] = _normal(g, spec.d_model, std=0.1, mean=1.0)
    ids = torch.randint(0, spec.vocab, (case["batch"], case["tokens"]),
                        generator=torch.Generator().manual_seed(seed), dtype=torch.int64)
    return spec, sd, ids, perm


def _ragged_config():
    """The benchmark's smaller layer-by-layer stack: attention and matrix-memory layers by turns, two of each."""
    att = {"type": "attention", "mlp": {"kind": "dense", "ff": 8192},
           "mixer": {"heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 2048},
                     "rot": {"base": 500000.0, "dims": 128,
                             "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}}
    rec = {"type": "mlstm", "mlp": {"kind": "dense", "ff": 8192},
           "mixer": {"heads": 8, "dim": 128, "vdim": 256, "gate_cap": 15.0}}
    return {"architecture": "Sokevik", "vocab": 32000, "width": 2048, "norm": {"eps": 1e-6}, "canon": {"taps": 4},
            "layers": [att, rec, att, rec]}


def _ragged_inputs(case, seed):
    cfg = _ragged_config()
    W, g, sd = cfg["width"], _gen(seed, 6), {}
    sd["embed"], sd["head"] = _normal(g, cfg["vocab"], W), _normal(g, cfg["vocab"], W, std=0.02)
    one = lambda: _normal(g, 1, std=0.1, mean=1.0)[0]  # noqa: E731
    sd["final.norm"] = one()
    for i, L in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", L["mixer"], L["mlp"]["ff"]
        H, D, V, att = m["heads"], m["dim"], m["vdim"], L["type"] == "attention"
        G = m.get("kv_heads", H)
        for n in ("norm1", "norm1b", "norm2", "norm2b"):
            sd[p + n] = one()
        sd[p + "canon1"], sd[p + "canon2"] = _normal(g, W, 4, std=0.2), _normal(g, W, 4, std=0.2)
        for n, rows in (("q", H * D), ("k", G * D), ("v", G * V), ("g", H if att else H * V)):
            sd[p + "mix." + n] = _normal(g, rows, W, std=0.02)
        if att:
            sd[p + "mix.q.norm"], sd[p + "mix.k.norm"] = _normal(g, D, std=0.2, mean=1.0), _normal(g, D, std=0.2, mean=1.0)
            sd[p + "mix.sink"] = _normal(g, H)
        else:
            sd[p + "mix.norm"] = _normal(g, H * V, std=0.2, mean=1.0)
            sd[p + "mix.i"], sd[p + "mix.f"] = _normal(g, H, W, std=0.02), _normal(g, H, W, std=0.02)
            sd[p + "mix.i.b"], sd[p + "mix.f.b"] = _normal(g, H), _normal(g, H, mean=2.0)
        sd[p + "mix.o"] = _normal(g, W, H * V, std=0.02)
        sd[p + "mlp.gate"], sd[p + "mlp.up"] = _normal(g, ff, W, std=0.02), _normal(g, ff, W, std=0.02)
        sd[p + "mlp.down"] = _normal(g, W, ff, std=0.02)
    host = torch.Generator().manual_seed(seed)
    prompts = [torch.randint(0, cfg["vocab"], (n,), generator=host).tolist() for n in _lengths(case)]
    fed = torch.randint(0, cfg["vocab"], (case["steps"], len(prompts)), generator=host).tolist()
    return cfg, sd, prompts, fed


# ---------------------------------------------------------------------------------------------- one pass
def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "sample":
        x, seeds, steps = _sample_inputs(case, seed)
        st.update(logits=x, out=torch.zeros(case["rows"], dtype=torch.int32, device=DEV), seeds=seeds.to(DEV),
                  steps=steps.to(DEV))
    elif kind == "prompt":
        spec, sd, hidden = _prompt_inputs(case, seed)
        eng = ShardEngine(spec, start_layer=1, end_layer=case["layers"], max_batch=case["batch"],
                          max_seq_len=max(64, case["tokens"] + 1), page_size=PAGE)
        eng.load_state_dict(sd)
        eng.start_batch(case["batch"], case["tokens"], case["tokens"] + 1)
        st.update(eng=eng, hidden=hidden)
    elif kind == "attention":
        spec = _spec(case)
        st.update(_attention_inputs(case, seed), spec=spec)
        # key splits: about two blocks per multiprocessor, no split shorter than four 64-token tiles (the engine's rule)
        tiles = (case["max_len"] + 63) // 64
        splits = max(1, min((tiles + 3) // 4, 2 * ops.sm_count() // (case["rows"] * spec.n_kv_heads), 64))
        nbytes = ops.attn_decode_scratch_bytes(case["rows"], spec.n_heads, spec.head_dim, splits)
        cos, sin = rope_tables(spec, case["max_len"], DEV)
        st.update(splits=splits, scratch=torch.empty(max(nbytes // 4, 1), dtype=torch.float32, device=DEV), cos=cos, sin=sin,
                  out=torch.empty(case["rows"], spec.n_heads * spec.head_dim, dtype=BF, device=DEV))
    elif kind == "mlp":
        spec, d = _spec(case), _mlp_inputs(case, seed)
        st.update(spec=spec, attn=d["attn"], h=d["h"], ln=d["ln"], wo=d["wo"], down=d["down"],
                  wgu=ops.pack_gate_up(d["gate"], d["up"]),
                  scratch=torch.zeros(ops.gemm_splitk_scratch_bytes(128, 2 * spec.d_ff), dtype=torch.uint8, device=DEV))
        n = case["rows"]
        st.update({k: torch.empty(n, w, dtype=BF, device=DEV)
                   for k, w in (("mid", spec.d_model), ("x", spec.d_model), ("act", spec.d_ff), ("out", spec.d_model))})
    elif kind == "generate":
        spec, sd, ids, _ = _generate_inputs(case, seed)
        eng = ShardEngine(spec, max_batch=case["batch"], max_seq_len=case["tokens"] + case["new"], page_size=PAGE)
        eng.load_state_dict(sd)
        st.update(eng=eng, ids=ids, seed=seed)
    else:
        cfg, sd, prompts, fed = _ragged_inputs(case, seed)
        spec = sokevik.spec_from_config(cfg)
        eng = RaggedEngine(spec, max_batch=max(4, len(prompts)), max_seq_len=512, page_size=PAGE)
        eng.load_tensors(sokevik.model_tensors(spec, sd))
        st.update(eng=eng, prompts=prompts, fed=fed)
    return st


@torch.no_grad()
def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "sample":
        if case["rows"] == 1:
            return ops.sample(st["logits"], out=st["out"], seed=st["seeds"], step=st["steps"])
        return ops.sample_rows(st["logits"], st["out"], st["seeds"], st["steps"])
    if kind == "prompt":
        if case["chunk"]:
            return st["eng"].prefill_chunked(case["batch"], case["tokens"], case["chunk"], hidden=st["hidden"])
        return st["eng"].prefill(case["batch"], case["tokens"], hidden=st["hidden"])
    if kind == "attention":
        s = st["spec"]
        ops.paged_attn_decode_fused(st["qkv"], st["cos"], st["sin"], st["k"], st["v"], st["table"], st["lens"], st["out"],
                                    s.n_heads, s.n_kv_heads, s.head_dim, s.head_dim ** -0.5, num_splits=st["splits"],
                                    scratch=st["scratch"], window=case["window"])
        return st["out"], st["k"], st["v"]
    if kind == "mlp":
        s, sk = st["spec"], st["scratch"]
        ops.linear_splitk(st["attn"], st["wo"], sk, residual=st["h"], out=st["mid"])
        ops.add_rmsnorm(st["mid"], st["ln"], s.eps, out=st["x"])
        ops.linear_splitk_gated_silu(st["x"], st["wgu"], sk, out=st["act"])
        ops.linear_splitk(st["act"], st["down"], sk, residual=st["mid"], out=st["out"])
        return st["out"]
    if kind == "generate":
        ids = st["eng"].generate(st["ids"], case["tokens"] + case["new"], do_sample=True, seed=st["seed"])
        return ids, st["eng"].last_logits
    eng, prompts = st["eng"], st["prompts"]
    slots = [eng.open_sequence() for _ in prompts]
    outs = [eng.step([(s, p) for s, p in zip(slots, prompts)])]
    for toks in st["fed"]:
        outs.append(eng.step([(s, [t]) for s, t in zip(slots, toks)]))
    for s in slots:
        eng.close_sequence(s)
    return outs


# ---------------------------------------------------------------------------------------------- cost and accuracy
def _pairs(tokens, window=0):
    """Query-key pairs of causal attention over a prompt."""
    if not window or tokens <= window:
        return tokens * (tokens + 1) // 2
    return window * (window + 1) // 2 + (tokens - window) * window


def work(case):
    kind = case["kind"]
    if kind == "sample":
        n = case["rows"] * case["vocab"]
        return {"bytes": 2 * n + 16 * case["rows"], "flops": n}
    if kind == "ragged":
        cfg = _ragged_config()
        rows, steps, live = sum(_lengths(case)), case["steps"], case["rows"]
        W = cfg["width"]
        params, pair_flops = 0, 0
        for L in cfg["layers"]:
            m = L["mixer"]
            H, D, V, G = m["heads"], m["dim"], m["vdim"], m["kv_heads"] if "kv_heads" in m else m["heads"]
            gates = H if L["type"] == "attention" else H * V + 2 * H
            params += W * (H * D + G * (D + V) + gates + H * V) + 3 * W * L["mlp"]["ff"]
            if L["type"] == "attention":
                pair_flops += 2 * H * (D + V) * sum(_pairs(n + steps) for n in _lengths(case))
            else:
                pair_flops += 4 * H * D * V * (rows + steps * live)  # state update and read-out per position
        head = W * cfg["vocab"]
        return {"bytes": 2 * (1 + steps) * (params + head) + 2 * W * (rows + steps * live),
                "flops": 2 * params * (rows + steps * live) + 2 * head * (1 + steps) * live + pair_flops}
    s = _spec(case)
    d, hd, H, KV = s.d_model, s.head_dim, s.n_heads, s.n_kv_heads
    per_layer = s.layer_weight_bytes() // 2
    if kind == "prompt":
        rows = case["batch"] * case["tokens"]
        chunks = math.ceil(case["tokens"] / case["chunk"]) if case["chunk"] else 1
        pairs = case["batch"] * _pairs(case["tokens"], s.sliding_window)
        out_rows = rows if chunks == 1 else case["batch"] * (case["tokens"] - (chunks - 1) * case["chunk"])
        return {"bytes": case["layers"] * (2 * per_layer + 4 * KV * hd * rows) + 2 * d * (rows + out_rows),
                "flops": case["layers"] * (2 * per_layer * rows + 4 * H * hd * pairs)}
    if kind == "attention":
        seen = sum(min(n, case["window"]) if case["window"] else n for n in _lengths(case))
        rows = case["rows"]
        return {"bytes": 4 * KV * hd * seen + 2 * rows * hd * (2 * H + 4 * KV), "flops": 4 * H * hd * seen}
    if kind == "mlp":
        params = d * H * hd + 3 * d * s.d_ff
        return {"bytes": 2 * params + 2 * case["rows"] * (H * hd + 2 * d), "flops": 2 * params * case["rows"]}
    n, T, B = case["new"], case["tokens"], case["batch"]
    params, head = s.n_layers * per_layer, d * s.vocab
    kv = 4 * KV * hd * s.n_layers
    return {"bytes": n * 2 * (params + head) + B * kv * (T + sum(range(T, T + n))) + 2 * B * d * (T + n),
            "flops": 2 * params * B * (T + n - 1) + 2 * head * B * n + 4 * H * hd * s.n_layers * B * _pairs(T + n - 1)}


def tolerance(case):
    """Two to four times what the paths show against 64 bits (prompts 0.4-1.1e-2, attention 4e-3, feed-forward 6e-3,
    whole models 1.3-2e-2, all of it bf16 rounding); sampled tokens are a function of the logits and the seed."""
    return {"sample": "exact", "prompt": {"rel": 2.5e-2}, "attention": {"rel": 1.2e-2}, "mlp": {"rel": 2e-2},
            "generate": {"rel": 5e-2}, "ragged": {"rel": 5e-2}}[case["kind"]]


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(x, w, eps):
    return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def _ln(x, w, b, eps):
    m = x.mean(-1, keepdim=True)
    return (x - m) / torch.sqrt((x - m).pow(2).mean(-1, keepdim=True) + eps) * w + b


def _rope(x, cos, sin):
    """Rotate the halves of x [T, heads, hd]; the tables are bf16 by the model's definition."""
    a, b = x.chunk(2, dim=-1)
    c, s = cos[:, None], sin[:, None]
    return torch.cat((a * c - b * s, b * c + a * s), dim=-1)


def _attend(q, k, v, scale, window=0):
    """Causal attention of one sequence, [T, H, hd] against [T, KV, hd], head by head in blocks of queries."""
    T, H, _ = q.shape
    group = H // k.shape[1]
    out = torch.empty(T, H, v.shape[-1], dtype=F64, device=q.device)
    j = torch.arange(T, device=q.device)
    for t0 in range(0, T, 2048):
        i = j[t0:t0 + 2048, None]
        hide = j[None, :] > i
        if window:
            hide = hide | (j[None, :] <= i - window)
        for h in range(H):
            s = q[t0:t0 + 2048, h] @ k[:, h // group].T * scale
            out[t0:t0 + 2048, h] = torch.softmax(s.masked_fill_(hide, -math.inf), dim=-1) @ v[:, h // group]
    return out


def _inv_freq(base, dims):
    return 1.0 / (base ** (torch.arange(0, dims, 2, device=DEV, dtype=F64) / dims))


def _tables(spec, T):
    """The bf16 rotation tables transformers multiplies by (fp32 angles)."""
    inv = 1.0 / (spec.rope_theta ** (torch.arange(0, spec.head_dim, 2, dtype=torch.int64).float() / spec.head_dim))
    ang = torch.arange(T, dtype=torch.float32)[:, None] * inv[None]
    return ang.cos().to(BF).to(DEV).to(F64), ang.sin().to(BF).to(DEV).to(F64)


def _layer64(spec, sd, i, h, B):
    """One decoder layer on hidden states [B * T, d] in 64 bits."""
    T, H, KV, hd = h.shape[0] // B, spec.n_heads, spec.n_kv_heads, spec.head_dim
    if spec.arch == "gpt2":
        p = f"transformer.h.{i}."
        w = lambda n: sd[p + n].to(F64)  # noqa: E731
        lin = lambda x, n: x @ w(n + ".weight") + w(n + ".bias")  # noqa: E731
        qkv = lin(_ln(h, w("ln_1.weight"), w("ln_1.bias"), spec.eps), "attn.c_attn")
    else:
        p = f"model.layers.{i}."
        w = lambda n: sd[p + n + ".weight"].to(F64)  # noqa: E731
        x = _rms(h, w("input_layernorm"), spec.eps)
        qkv = torch.cat([x @ w(f"self_attn.{n}_proj").T for n in "qkv"], dim=1)
        cos, sin = _tables(spec, T)
    outs = []
    for b in range(B):
        q, k, v = (t.reshape(T, -1, hd) for t in qkv[b * T:(b + 1) * T].split([H * hd, KV * hd, KV * hd], dim=1))
        if spec.arch != "gpt2":
            q, k = _rope(q, cos, sin), _rope(k, cos, sin)
        outs.append(_attend(q, k, v, hd ** -0.5, spec.sliding_window).reshape(T, H * hd))
    a = torch.cat(outs)
    if spec.arch == "gpt2":
        h = h + lin(a, "attn.c_proj")
        u = lin(_ln(h, w("ln_2.weight"), w("ln_2.bias"), spec.eps), "mlp.c_fc")
        u = 0.5 * u * (1 + torch.tanh(math.sqrt(2 / math.pi) * (u + 0.044715 * u ** 3)))
        return h + lin(u, "mlp.c_proj")
    h = h + a @ w("self_attn.o_proj").T
    x = _rms(h, w("post_attention_layernorm"), spec.eps)
    return h + (torch.nn.functional.silu(x @ w("mlp.gate_proj").T) * (x @ w("mlp.up_proj").T)) @ w("mlp.down_proj").T


def _philox(seed, step):
    """First word of Philox4x32-10 for counter (step, 0) and key `seed` as a uniform number in [0, 1)."""
    c = [step, 0, 0x6A09E667, 0xBB67AE85]
    k = [seed & 0xFFFFFFFF, seed >> 32]
    for _ in range(10):
        a, b = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [(b >> 32) ^ c[1] ^ k[0], b & 0xFFFFFFFF, (a >> 32) ^ c[3] ^ k[1], a & 0xFFFFFFFF]
        k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
    return (c[0] >> 8) / 16777216.0


def _sample64(row, seed, step, temperature=0.8, top_k=50, top_p=0.95):
    x = row.astype(np.float64) / temperature
    kept = np.flatnonzero(x >= np.sort(x)[-top_k])
    kept = kept[np.lexsort((kept, -x[kept]))]
    p = np.exp(x[kept] - x[kept[0]])
    p /= p.sum()
    n = max(1, int(((np.cumsum(p) - p) < top_p).sum()))
    return int(kept[min(n - 1, int((np.cumsum(p[:n]) <= _philox(seed, step) * p[:n].sum()).sum()))])


def _ragged64(cfg, P, tokens):
    """Logits of every position of one sequence of the layer-by-layer stack."""
    eps, x = cfg["norm"]["eps"], P["embed"][tokens]
    T = len(tokens)
    pos = torch.arange(T, device=DEV, dtype=F64)

    def conv(h, w):
        pad = torch.cat((torch.zeros(3, h.shape[1], dtype=F64, device=DEV), h))
        return h + sum(w[:, j] * pad[j:j + T] for j in range(4))

    def turn(z, ang):
        a, b = z[..., 0::2], z[..., 1::2]
        return torch.stack((a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()), dim=-1).flatten(-2)

    for i, L in enumerate(cfg["layers"]):
        p, m = f"l{i}.", L["mixer"]
        H, D, V = m["heads"], m["dim"], m["vdim"]
        w = lambda n: P[p + n]  # noqa: E731
        h = conv(_rms(x, w("norm1"), eps), w("canon1"))
        q, k, v = (h @ w("mix." + n).T for n in "qkv")
        if L["type"] == "attention":
            G, sc = m["kv_heads"], m["rot"]["scaling"]
            inv = _inv_freq(m["rot"]["base"], D)
            wave = 2 * math.pi / inv
            mix = (sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])
            mid = (1 - mix) * inv / sc["factor"] + mix * inv
            far, near = wave > sc["original"] / sc["low"], wave < sc["original"] / sc["high"]
            ang = pos[:, None, None] * torch.where(far, inv / sc["factor"], torch.where(near, inv, mid))
            ang_v = pos[:, None, None] * _inv_freq(m["rot"]["base"], V)
            q = turn(_rms(q.reshape(T, H, D), w("mix.q.norm"), eps), ang)
            k = turn(_rms(k.reshape(T, G, D), w("mix.k.norm"), eps), ang)
            v = turn(v.reshape(T, G, V), ang_v)
            hide = pos[None, :] > pos[:, None]
            o = torch.empty(T, H, V, dtype=F64, device=DEV)
            for hh in range(H):
                s = (q[:, hh] @ k[:, hh * G // H].T * m["scale"]).masked_fill_(hide, -math.inf)
                s = torch.cat((s, w("mix.sink")[hh].expand(T, 1)), dim=1)
                o[:, hh] = torch.softmax(s, dim=-1)[:, :T] @ v[:, hh * G // H]
            o = turn(o, -ang_v) * torch.sigmoid(h @ w("mix.g").T)[:, :, None]
        else:
            cap = lambda t: m["gate_cap"] * torch.tanh(t / m["gate_cap"])  # noqa: E731
            q, k, v = q.reshape(T, H, D) / math.sqrt(D), k.reshape(T, H, D), v.reshape(T, H, V)
            li = cap(h @ w("mix.i").T + w("mix.i.b"))
            cf = torch.cumsum(torch.nn.functional.logsigmoid(cap(h @ w("mix.f").T + w("mix.f.b"))), dim=0)
            # weight of position j in the state at t: exp(cf_t - cf_j + li_j); the stabiliser is its running maximum
            # against the empty state's exp(cf_t)
            top = cf + torch.clamp(torch.cummax(li - cf, dim=0).values, min=0.0)
            o = torch.empty(T, H, V, dtype=F64, device=DEV)
            for hh in range(H):
                e = cf[:, hh, None] - cf[None, :, hh] + li[None, :, hh] - top[:, hh, None]
                a = (q[:, hh] @ k[:, hh].T) * torch.exp(e).tril()
                den = torch.maximum(a.sum(dim=1).abs(), torch.exp(-top[:, hh])) + 1e-6
                o[:, hh] = a @ v[:, hh] / den[:, None]
            o = _rms(o, w("mix.norm").reshape(H, V), eps) * torch.sigmoid(h @ w("mix.g").T).reshape(T, H, V)
        x = x + _rms(o.reshape(T, H * V) @ w("mix.o").T, w("norm1b"), eps)
        h = conv(_rms(x, w("norm2"), eps), w("canon2"))
        y = (torch.nn.functional.silu(h @ w("mlp.gate").T) * (h @ w("mlp.up").T)) @ w("mlp.down").T
        x = x + _rms(y, w("norm2b"), eps)
    return _rms(x, P["final.norm"], eps) @ P["head"].T


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        x, seeds, steps = _sample_inputs(case, seed)
        rows = x.float().cpu().numpy()
        return torch.tensor([_sample64(rows[b], int(seeds[b]), int(steps[b])) for b in range(case["rows"])],
                            dtype=torch.int32)
    if kind == "prompt":
        spec, sd, hidden = _prompt_inputs(case, seed)
        h = hidden.to(F64)
        for i in range(1, case["layers"] + 1):
            h = _layer64(spec, sd, i, h, case["batch"])
        if case["chunk"]:  # the last chunk of every prompt
            last = (case["tokens"] - 1) // case["chunk"] * case["chunk"]
            h = h.view(case["batch"], case["tokens"], -1)[:, last:].reshape(-1, spec.d_model)
        return h
    if kind == "attention":
        spec, st = _spec(case), _attention_inputs(case, seed)
        H, KV, hd = spec.n_heads, spec.n_kv_heads, spec.head_dim
        cos, sin = _tables(spec, case["max_len"])
        kc, vc = st["k"].to(F64), st["v"].to(F64)
        outs = []
        for b, n in enumerate(_lengths(case)):
            q, k, v = (t.reshape(1, -1, hd) for t in st["qkv"][b:b + 1].to(F64).split([H * hd, KV * hd, KV * hd], dim=1))
            q, k = _rope(q, cos[n - 1:n], sin[n - 1:n]), _rope(k, cos[n - 1:n], sin[n - 1:n])
            page = int(st["table"][b, (n - 1) // PAGE])
            kc[page, :, (n - 1) % PAGE], vc[page, :, (n - 1) % PAGE] = k[0], v[0]
            pages = st["table"][b, :st["pages"][b]].long()
            keys, vals = (c[pages].transpose(1, 2).reshape(-1, KV, hd)[:n] for c in (kc, vc))
            if case["window"]:
                keys, vals = keys[-case["window"]:], vals[-case["window"]:]
            s = torch.einsum("gjd,tgd->gjt", q.reshape(KV, H // KV, hd), keys) * hd ** -0.5
            outs.append(torch.einsum("gjt,tgd->gjd", torch.softmax(s, dim=-1), vals).reshape(H * hd))
        return torch.stack(outs), kc, vc
    if kind == "mlp":
        spec, d = _spec(case), {k: v.to(F64) for k, v in _mlp_inputs(case, seed).items()}
        h = d["h"] + d["attn"] @ d["wo"].T
        x = _rms(h, d["ln"], spec.eps)
        return h + (torch.nn.functional.silu(x @ d["gate"].T) * (x @ d["up"].T)) @ d["down"].T
    if kind == "generate":
        spec, sd, ids, perm = _generate_inputs(case, seed)
        seqs = [ids.to(DEV)]
        for _ in range(case["new"]):
            seqs.append(perm[seqs[-1][:, -1:]])
        full = torch.cat(seqs, dim=1)
        B, T = case["batch"], full.shape[1] - 1
        h = sd["model.embed_tokens.weight"][full[:, :-1].reshape(-1)].to(F64)
        for i in range(spec.n_layers):
            h = _layer64(spec, sd, i, h, B)
        h = _rms(h.view(B, T, -1)[:, -1], sd["model.norm.weight"].to(F64), spec.eps)
        return full.cpu(), h @ sd["lm_head.weight"].to(F64).T
    cfg, sd, prompts, fed = _ragged_inputs(case, seed)
    P = {k: v.to(F64) for k, v in sd.items()}
    per_seq = [_ragged64(cfg, P, torch.tensor(p + [t[i] for t in fed], device=DEV)) for i, p in enumerate(prompts)]
    return [torch.stack([per_seq[i][len(p) - 1 + n] for i, p in enumerate(prompts)]) for n in range(len(fed) + 1)]
