"""Every float32 product of a model's parts gets the device status word: the GEMM's waits are bounded, and one that is given
up has to be told of.  (The launches are replaced; no GPU.)"""
from types import SimpleNamespace

import torch

from velox_b200.ops import kernels
from velox_b200.parts.io import LinearHead
from velox_b200.parts.mlp import SwiGLU


def test_head_and_feed_forward_hand_the_status_on(monkeypatch):
    seen = []
    monkeypatch.setattr(kernels, "gemm_f32", lambda *args, status=None: seen.append(status))
    monkeypatch.setattr(kernels, "swiglu", lambda *args: None)
    buffers = SimpleNamespace(max_tokens=4, max_logit_rows=4, get=lambda name, shape, dtype: torch.zeros(shape, dtype=dtype))
    status = torch.zeros(4, dtype=torch.int32)
    ctx = SimpleNamespace(num_tokens=3, workspace=buffers, status=status, residual=torch.zeros(4, 8))
    x = torch.zeros(4, 8)
    head = LinearHead({"vocab_size": 16, "hidden_size": 8}, {"weight": torch.zeros(16, 8)}, torch.float32, "cpu")
    head.forward(x, 3, ctx)
    part = SwiGLU({"hidden_size": 8, "intermediate_size": 16},
                  {"gate_up.weight": torch.zeros(32, 8), "down.weight": torch.zeros(8, 16)}, torch.float32, "cpu")
    part.forward(x, ctx)
    assert len(seen) == 3 and all(word is status for word in seen)
