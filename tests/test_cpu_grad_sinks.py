"""Where weight gradients may be added by a kernel in place of autograd: decided on the host, tested on the CPU."""

import pytest
import torch

from rl_engine.kernels.ops.base import _C, _EXT_AVAILABLE
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


@pytest.mark.skipif(not _EXT_AVAILABLE, reason="the native extension is not built")
def test_every_kind_of_gradient_hook_is_seen():
    """Hooks on the parameter, after its accumulation and on its AccumulateGrad node (how wrappers attach); a node that exists
    without hooks is not one."""
    node_of = lambda p: p.expand_as(p).grad_fn.next_functions[0][0]
    attach = [lambda p: p.register_hook(lambda g: g), lambda p: p.register_post_accumulate_grad_hook(lambda p: None),
              lambda p: node_of(p).register_hook(lambda *a: None), lambda p: node_of(p).register_prehook(lambda g: None),
              lambda p: torch.autograd.graph.register_multi_grad_hook([p], lambda g: None)]
    for add in attach:
        p = torch.nn.Parameter(torch.zeros(4, 8))
        node = node_of(p)  # noqa: F841  (kept alive, as a graph would)
        assert not _C.grad_is_watched(p)
        handle = add(p)  # noqa: F841
        assert _C.grad_is_watched(p)
