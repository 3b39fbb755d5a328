"""What a batched decode step takes from the allocator once its workspaces exist: nothing beyond its outputs."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _growth(step):
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    out = step()
    torch.cuda.synchronize()
    grown = torch.cuda.memory_allocated() - before
    return grown, out


def test_uniform_stack(cuda):
    from dli_b200.engine import ModelSpec, ShardEngine
    from oracle import decoder_ref as R

    spec = ModelSpec("llama", 2, 256, 4, 2, 64, 512, 512, 1e-5, 10000.0, 0, 128)
    e = ShardEngine(spec, device="cuda:0", max_batch=4, max_seq_len=64, use_cuda_graph=False)
    e.load_state_dict(R.seeded_state_dict(R.ModelSpec(**spec.__dict__), seed=7, std=0.06))
    e.start_batch(4, 8, 16)
    e.prefill(4, 8, ids=torch.randint(0, 512, (32,), device=cuda, dtype=torch.int32))
    grown, _ = _growth(lambda: e.decode_step(4))
    assert grown < 1 << 20, grown


def test_ragged_stack(cuda, monkeypatch):
    from test_hybrid_engine_gpu import build, cfg_a

    monkeypatch.setenv("DLI_RAGGED_GRAPH", "0")
    e, _ = build(cfg_a(), torch.bfloat16)
    slots = [e.open_sequence() for _ in range(3)]
    e.step([(s, [1]) for s in slots[:2]])  # makes the workspaces (of 64 rows)
    grown, _ = _growth(lambda: e.step([(s, [4]) for s in slots]))  # three rows: the tensor-core projections
    assert grown < 1 << 20, grown
