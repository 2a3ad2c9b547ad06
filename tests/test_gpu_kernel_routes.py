"""Sizes at which the dispatch of a kernel changes, the edges of its tiles and the splits inside it: results against plain
PyTorch in higher precision, and the same bits where a row must not depend on its neighbours."""

from dataclasses import replace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF16 = 2.0 ** -8  # relative spacing of bf16: half of it is the rounding of one stored value


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(*shape, seed, scale=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, device=DEV, generator=_gen(seed)) * scale).to(dtype)


def _rel(got, want):
    return ((got.double() - want.double()).norm() / want.double().norm().clamp_min(1e-300)).item()


# ------------------------------------------------------------------------------------------------ embedding gradient
@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 1000])
@pytest.mark.parametrize("kind", ["one", "distinct", "few", "border"])
@pytest.mark.parametrize("d,dtype", [(200, torch.bfloat16), (13, torch.float32), (1032, torch.bfloat16)])
def test_embedding_gradient_runs_across_chunks(n, kind, d, dtype):
    from rl_engine.kernels.ops.sm100.model_ops import FusedEmbeddingSM100Op

    vocab = 2000
    ids = {"one": torch.zeros(n, dtype=torch.long), "distinct": torch.randperm(vocab)[:n], "few": torch.arange(n) % 3,
           "border": torch.arange(n) // 64}[kind].to(DEV)
    ids = ids[torch.randperm(n, generator=torch.Generator().manual_seed(n)).to(DEV)]
    table = _randn(vocab, d, seed=1, dtype=dtype).requires_grad_(True)
    dy = _randn(n, d, seed=2, dtype=dtype)
    op = FusedEmbeddingSM100Op()
    op(ids, table).backward(dy)
    want = torch.zeros(vocab, d, dtype=torch.float64, device=DEV).index_add_(0, ids, dy.double())
    assert _rel(table.grad, want) < (BF16 / 2 if dtype == torch.bfloat16 else 1e-5)
    first, table.grad = table.grad, None
    op(ids, table).backward(dy)
    assert torch.equal(first, table.grad)


def test_embedding_gradient_refuses_ids_outside_the_table():
    from rl_engine.kernels.ops.sm100.model_ops import FusedEmbeddingSM100Op

    table = _randn(10, 64, seed=1).requires_grad_(True)
    for bad in (-1, 10):
        out = FusedEmbeddingSM100Op()(torch.tensor([1, bad, 2], device=DEV), table)
        with pytest.raises(ValueError):
            out.sum().backward()


@pytest.mark.parametrize("p,g,l,hq,hkv", [(1, 2, 33, 4, 1), (300, 5, 70, 8, 2), (129, 40, 64, 2, 2), (700, 3, 200, 16, 2)])
def test_attention_gradient_with_split_block_lists(p, g, l, hq, hkv):
    """Key tiles whose query-block lists are cut into pieces of 4 and more, against the fp32 restatement of the packed
    attention (P and dS are rounded to bf16 once each)."""
    from rl_engine.kernels.ops.sm100.attention import _reference_backward, grpo_group_layout, packed_attention_forward
    from rl_engine.kernels.ops.sm100.attention_bwd_kernels import fused_backward

    t = p + g * l
    q, k, v = _randn(t, hq, 128, seed=1), _randn(t, hkv, 128, seed=2), _randn(t, hkv, 128, seed=3)
    dout = _randn(t, hq, 128, seed=4)
    layout = grpo_group_layout(p, g, l, torch.device(DEV))
    out, lse = packed_attention_forward(q, k, v, layout)
    scale = 128 ** -0.5
    got = fused_backward(q, k, v, out, lse, dout, layout, scale)
    for a, b in zip(got, _reference_backward(q, k, v, out, lse, dout, layout, scale)):
        assert _rel(a, b) < 2 * BF16
    assert all(torch.equal(a, b) for a, b in zip(got, fused_backward(q, k, v, out, lse, dout, layout, scale)))
