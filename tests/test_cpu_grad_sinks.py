"""Where weight gradients may be added by a kernel in place of autograd: decided on the host, tested on the CPU."""

import pytest
import torch

from rl_engine.kernels.registry import kernel_registry
from rl_engine.models.config import ModelConfig
from rl_engine.models.grpo import _head_logps
from rl_engine.models.llama import LlamaModel


def test_sinks_go_only_to_operators_that_take_them(monkeypatch):
    """With the registry's native operators (forced by the environment, or its fallback) the passes of a trainer run as
    without sinks: autograd adds the gradients."""
    from rl_engine.kernels.ops.sm100.linear_logp import FusedLinearLogpSM100Op
    from rl_engine.kernels.ops.sm100.model_ops import FusedEmbeddingSM100Op

    assert FusedEmbeddingSM100Op.supports_grad_sink and FusedLinearLogpSM100Op.supports_grad_sink
    for name in ("embedding", "linear_logp"):
        assert not getattr(kernel_registry.get_op(name), "supports_grad_sink", False)
    model = LlamaModel(ModelConfig("sinks", 64, 32, 1, 2, 1, 16, 32), dtype=torch.float32, device="cpu")
    buffers = {}
    monkeypatch.setattr(model, "_grad_sink", lambda name: buffers.setdefault(name, torch.zeros_like(model.view(name))))
    ids = torch.tensor([3, 5, 3])
    logps = _head_logps(model, model.embed_tokens(ids), ids)
    grads = torch.autograd.grad(logps.sum(), [model.view("embed"), model.view("lm_head")])
    assert all(float(g.norm()) > 0 for g in grads)
    assert all(float(b.norm()) == 0 for b in buffers.values())
