"""Paths a step takes around its operators: replayed forward passes, staging of the batch, the loss read back."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from flexflow_train_b200 import _ffcore as core  # noqa: E402
from flexflow_train_b200 import api  # noqa: E402
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
