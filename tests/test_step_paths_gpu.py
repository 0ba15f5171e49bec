"""Paths a step takes around its operators: replayed forward passes, staging of the batch, the loss read back."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from flexflow_train_b200 import _ffcore as core  # noqa: E402
from flexflow_train_b200 import api  # noqa: E402
from flexflow_train_b200.ops import kernels as K  # noqa: E402
from flexflow_train_b200.runtime.executor import ExecConfig, Executable  # noqa: E402

LM = {"num_features": 128, "sequence_length": 48, "batch_size": 3, "dim_feedforward": 256, "num_heads": 2, "num_decoder_layers": 2,
      "dropout": 0.0, "vocab_size": 200}


@pytest.mark.parametrize("model,cfg,shape,hi", [("transformer_lm", LM, (3, 48, 1), 200), ("mlp", {"batch_size": 5, "input_dim": 30}, (5, 30), 0)])
def test_replayed_forward_matches_eager(model, cfg, shape, hi):
    g = core.build_model(model, cfg)
    eager = Executable(g, ExecConfig(training=False, use_cuda_graph=False))
    replay = Executable(g, ExecConfig(training=False, use_cuda_graph=True))
    name = next(n["name"] for n in g.nodes() if n["type"] == "INPUT")
    gen = torch.Generator(device="cuda").manual_seed(0)
    kept = []
    for _ in range(4):  # eager call, capture, two replays: each on inputs of its own
        x = torch.randint(0, hi, shape, generator=gen, device="cuda", dtype=torch.int32) if hi else torch.randn(shape, generator=gen, device="cuda")
        kept.append((eager.infer({name: x}), replay.infer({name: x})))
    for a, b in kept:  # every call returned a tensor of its own
        assert torch.equal(a, b)
    assert not torch.equal(kept[0][1], kept[3][1])


def test_forward_inside_a_callers_capture():
    m = api.compile("mlp", {"batch_size": 4, "input_dim": 16}, training=False)
    x = torch.randn(4, 16, device="cuda")
    want = m.forward({"input": x}).clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = m.forward({"input": x})
    g.replay()
    assert torch.equal(y, want)


def test_capturing_the_forward_leaves_the_process_alone(monkeypatch):
    """The call that captures neither synchronises the device nor empties the allocator's cache under other threads."""
    m = api.compile("mlp", {"batch_size": 4, "input_dim": 16}, training=False)
    x = torch.randn(4, 16, device="cuda")
    want, calls = m.forward({"input": x}).clone(), []
    for name in ("synchronize", "empty_cache"):
        monkeypatch.setattr(torch.cuda, name, lambda *a, name=name, **k: calls.append(name))
    got = m.forward({"input": x}).clone()
    monkeypatch.undo()
    assert not calls and torch.equal(got, want) and torch.equal(m.forward({"input": x}), want)
    assert m.executable._fwd_graph


def test_forward_stays_eager_without_memory_for_a_graph(monkeypatch):
    """Operators that allocate as they go find their memory in the cache; a graph's pool, which has to have its own, may not."""
    m = api.compile("mlp", {"batch_size": 4, "input_dim": 16}, training=False)
    eager = Executable(m.graph, ExecConfig(training=False, use_cuda_graph=False))
    eager.load_state_dict(m.state_dict())
    op = next(o for o in m.executable.ops.values() if o.type == "LINEAR")
    plain = op.forward

    def allocates():
        plain()
        if torch.cuda.is_current_stream_capturing():
            raise torch.cuda.OutOfMemoryError("no memory left")

    monkeypatch.setattr(op, "forward", allocates)
    for _ in range(3):
        x = torch.randn(4, 16, device="cuda")
        assert torch.equal(m.forward({"input": x}), eager.infer({"input": x}))
    assert torch.randn(3, device="cuda").isfinite().all()  # the generator is not left inside a capture


@pytest.mark.parametrize("n", [1, 7, 4096, 4099, 16384 * 3 + 5])
@pytest.mark.parametrize("offset", [0, 1])  # 1: no 16-byte alignment
def test_stage_batch_copies_and_casts_like_copy(n, offset):
    gen = torch.Generator(device="cuda").manual_seed(n)
    f = torch.randn(n + offset, generator=gen, device="cuda")[offset:]
    i = torch.randint(-2**31, 2**31 - 1, (n + offset,), generator=gen, device="cuda", dtype=torch.int64)[offset:]
    pairs = []
    for src, dt in ((f, torch.bfloat16), (f, torch.float32), (i, torch.int32), (i, torch.int64), (i.int(), torch.int64), (f.half(), torch.float16),
                    (i.int(), torch.int32), (f > 0, torch.bool), (f.double(), torch.float32), (f.cpu(), torch.bfloat16)):
        pairs.append((src, torch.zeros(n + offset, dtype=dt, device="cuda")[offset:]))
    alpha, seed = torch.zeros(1, device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda")
    K.stage_batch(pairs * 2, (0.25, alpha, 2**62 + 3, seed))  # 20 pairs: more than one launch holds
    for src, dst in pairs:
        assert torch.equal(dst, src.to("cuda").to(dst.dtype)), (src.dtype, dst.dtype)
    assert alpha.item() == 0.25 and seed.item() == 2**62 + 3


@pytest.mark.parametrize("n", [1, 33, 4096, 32771])
def test_loss_mean(n):
    rows, out = torch.rand(n, device="cuda") + 1, torch.zeros(1).pin_memory()
    K.loss_mean(rows, out)
    torch.cuda.current_stream().synchronize()
    assert abs(out.item() - rows.double().mean().item()) < 1e-6 * 2  # 32 partial sums of n / 1024 terms each
