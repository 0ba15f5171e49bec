"""Scratch an operator reserves at planning covers what its kernels write."""
from types import SimpleNamespace

import pytest
import torch

from flexflow_train_b200.ops import kernels as K
from flexflow_train_b200.runtime.executor import AttentionOp, ExecConfig, Executable, _Buf

pytestmark = pytest.mark.skipif(not K.available(), reason="kernel library not built")


def _reserved(rows, embed, heads, d, shards):
    """Bytes of scratch a self-attention operator reserves when it is planned for the GPU (its tensors stay on the CPU)."""
    q_in, h = 8, heads // shards
    asked = [0]
    ex = SimpleNamespace(cfg=ExecConfig(training=True, fused_attention=False), device=torch.device("cpu"), on_gpu=True, values={},
                         head_shards=lambda op: shards, use_bias=lambda op, slot: True, next_salt=lambda: 1,
                         need_scratch=lambda n: asked.append(n), need_big_scratch=lambda n, slots: None, wgrad_splits=Executable.wgrad_splits,
                         torch_dtype=lambda name: torch.bfloat16,
                         allocator=SimpleNamespace(allocate=lambda shape, dt: torch.empty(shape, dtype=dt)))
    node = {"attrs": {"num_heads": heads, "kdim": d, "vdim": d, "embed_dim": embed, "dropout": 0.0}, "type": "MULTIHEAD_ATTENTION",
            "inputs": [(s, (0, "OUTPUT")) for s in ("QUERY", "KEY", "VALUE")] + [("WEIGHT", (1, "OUTPUT")), ("INPUT_BIAS", (2, "OUTPUT")),
                                                                               ("OUTPUT_BIAS", (3, "OUTPUT"))],
            "outputs": [("OUTPUT", SimpleNamespace(piece_sizes=(rows, 1, embed), dtype="FLOAT"), None)]}
    new = lambda *shape: _Buf(torch.empty(*shape, dtype=torch.bfloat16))  # noqa: E731
    ex.values.update({(0, "OUTPUT"): new(rows, 1, q_in), (1, "OUTPUT"): new(h * d * 3 * q_in + embed * h * d), (2, "OUTPUT"): new(3 * h * d),
                      (3, "OUTPUT"): new(embed), (4, "OUTPUT"): _Buf()})
    AttentionOp(ex, 4, node).setup()
    return max(asked)


@pytest.mark.parametrize("rows,embed,heads,d,shards", [(2400, 256, 4, 24, 1), (800, 1024, 16, 64, 4), (4096, 512, 5, 48, 1), (64, 1024, 16, 64, 1),
                                                       (1, 8, 1, 8, 1), (8192, 2048, 16, 128, 1)])
def test_attention_reserves_both_bias_gradients(rows, embed, heads, d, shards):
    have = _reserved(rows, embed, heads, d, shards)
    for cols in (embed, heads // shards * 3 * d):
        assert have >= 4 * K.bias_act_bwd_scratch(rows, cols), cols
