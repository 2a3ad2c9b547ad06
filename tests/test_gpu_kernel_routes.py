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


# ------------------------------------------------------------------------------------------------ linear log-prob
@pytest.mark.parametrize("n", [1, 127, 128, 129, 300, 777, 5000])
@pytest.mark.parametrize("v", [300, 513, 9000])
def test_linear_logp_rows_on_both_engines(n, v):
    """Single CTAs up to one row tile, CTA pairs above: values against fp64, and each row the same bits on its own."""
    from rl_engine.kernels.ops.sm100.linear_logp import FusedLinearLogpSM100Op

    h, w = _randn(n, 192, seed=n), _randn(v, 192, seed=v, scale=0.1)
    t = torch.randint(0, v, (n,), device=DEV, generator=_gen(3))
    op = FusedLinearLogpSM100Op()
    lp, ent = op.with_entropy(h, w, t)
    z = torch.log_softmax(h.double() @ w.double().t(), -1)
    assert torch.allclose(lp.double(), z.gather(1, t[:, None])[:, 0], atol=2e-5, rtol=1e-5)  # 32-bit sums over v terms
    assert torch.allclose(ent.double(), -(z.exp() * z).sum(-1), atol=2e-5, rtol=1e-5)
    rows = slice(n // 2, n // 2 + 1)
    assert torch.equal(op(h[rows], w, t[rows]), lp[rows])


def test_linear_logp_with_masked_vocabulary_and_replayed_graph():
    """Whole records of -inf (a masked stretch of the vocabulary, also the first one) leave the row finite; a captured call
    gives new results on every replay."""
    from rl_engine.kernels.ops.sm100.linear_logp import FusedLinearLogpSM100Op

    n, v = 200, 3000
    h, w = _randn(n, 128, seed=1), _randn(v, 128, seed=2, scale=0.1)
    bias = torch.zeros(v, device=DEV)
    bias[:1100] = float("-inf")
    bias[2000:2600] = float("-inf")
    t = torch.randint(1100, 2000, (n,), device=DEV, generator=_gen(4))
    op = FusedLinearLogpSM100Op()
    want = torch.log_softmax(h.double() @ w.double().t() + bias.double(), -1).gather(1, t[:, None])[:, 0]
    with torch.no_grad():
        assert torch.allclose(op(h, w, t, bias).double(), want, atol=2e-5, rtol=1e-5)
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            op(h, w, t, bias)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = op(h, w, t, bias)
        for seed in (5, 6, 7):
            h.copy_(_randn(n, 128, seed=seed))
            graph.replay()
            want = torch.log_softmax(h.double() @ w.double().t() + bias.double(), -1).gather(1, t[:, None])[:, 0]
            assert torch.allclose(out.double(), want, atol=2e-5, rtol=1e-5)


@pytest.mark.parametrize("n,chunk", [(100, 4096), (700, 128), (700, 4096), (513, 256)])
@pytest.mark.parametrize("v", [1001, 1024])
def test_linear_logp_weight_gradient_in_one_and_several_chunks(n, chunk, v):
    """First chunk writes, later ones add, the last one rounds: against fp64 of the same bf16 dz (rounding of dz: 2^-9 per
    term, of the stored gradient 2^-9), bias column sums included."""
    from rl_engine.kernels.ops.sm100.linear_logp import FusedLinearLogpSM100Op

    d = 64
    h, w = _randn(n, d, seed=n).requires_grad_(True), _randn(v, d, seed=v, scale=0.1).requires_grad_(True)
    b = (0.1 * torch.randn(v, device=DEV, generator=_gen(8))).requires_grad_(True)
    t = torch.randint(0, v, (n,), device=DEV, generator=_gen(9))
    g = torch.randn(n, device=DEV, generator=_gen(10))
    FusedLinearLogpSM100Op(bwd_chunk_tokens=chunk)(h, w, t, b).backward(g)
    hd, wd, bd = (x.detach().double().requires_grad_(True) for x in (h, w, b))
    torch.log_softmax(hd @ wd.t() + bd, -1).gather(1, t[:, None])[:, 0].backward(g.double())
    for got, want in ((h.grad, hd.grad), (w.grad, wd.grad), (b.grad, bd.grad)):
        assert _rel(got, want) < BF16


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
