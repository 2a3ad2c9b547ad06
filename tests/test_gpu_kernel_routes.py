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


@pytest.mark.parametrize("n,chunk", [(300, 128), (512, 256), (513, 512)])
def test_linear_logp_weight_gradient_adds_its_chunks_in_order(n, chunk):
    """The sum of the chunks' products, each formed apart in 32 bits, rounded once: the same bits, also where one longer
    contraction over the whole batch would fit."""
    from rl_engine.kernels.ops.base import require_ext
    from rl_engine.kernels.ops.sm100.linear_logp import FusedLinearLogpSM100Op, _forward_local

    ext, d, v = require_ext(), 192, 1024
    h, w = _randn(n, d, seed=n).requires_grad_(True), _randn(v, d, seed=v, scale=0.1).requires_grad_(True)
    t = torch.randint(0, v, (n,), device=DEV, generator=_gen(9))
    g = torch.randn(n, device=DEV, generator=_gen(10))
    FusedLinearLogpSM100Op(bwd_chunk_tokens=chunk)(h, w, t).backward(g)
    _, lse, _ = _forward_local(h.detach(), w.detach(), t, None, True, False)
    want = torch.zeros(v, d, device=DEV)
    for i in range(0, n, chunk):
        rows = slice(i, min(i + chunk, n))
        dz = torch.empty(rows.stop - i, v, dtype=torch.bfloat16, device=DEV)
        ext.linear_logp_dz(h.detach()[rows], w.detach(), t[rows], None, lse[rows], g[rows], 0, dz)
        want += ext.gemm(dz, h.detach()[rows], True, True, None, True)
    assert torch.equal(w.grad, want.to(torch.bfloat16))


def test_linear_logp_backward_passes_on_two_streams():
    """Each stream's gradients are those of the pass on its own."""
    from rl_engine.kernels.ops.sm100.linear_logp import FusedLinearLogpSM100Op

    n, d, v = 1500, 256, 20000
    op, streams = FusedLinearLogpSM100Op(bwd_chunk_tokens=512), [torch.cuda.Stream() for _ in range(2)]
    w = _randn(v, d, seed=1, scale=0.1).requires_grad_(True)
    hs = [_randn(n, d, seed=2 + i).requires_grad_(True) for i in range(2)]
    t = torch.randint(0, v, (n,), device=DEV, generator=_gen(4))
    g = torch.randn(n, device=DEV, generator=_gen(5))
    want = [torch.autograd.grad(op(h, w, t), [h, w], g) for h in hs]
    torch.cuda.synchronize()
    for _ in range(4):
        logps, got = [], []
        for s, h in zip(streams, hs):
            with torch.cuda.stream(s):
                logps.append(op(h, w, t))
        for s, lp, h in zip(streams, logps, hs):
            with torch.cuda.stream(s):
                got.append(torch.autograd.grad(lp, [h, w], g))
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


@pytest.mark.parametrize("rows", [8, 24, 1024, 1032, 4000])
@pytest.mark.parametrize("d", [40, 264])
def test_rmsnorm_weight_gradient_adds_its_chunks_in_order(rows, d):
    """Eight rows a chunk at these sizes: the chunks on their own, added one after the other in 32 bits, are the same bits."""
    from rl_engine.kernels.ops.base import require_ext

    ext = require_ext()
    x, dy = _randn(rows, d, seed=1), _randn(rows, d, seed=2)
    w = torch.randn(d, device=DEV, generator=_gen(3))
    rstd = torch.rand(rows, device=DEV, generator=_gen(4)) + 0.5
    parts = [ext.rmsnorm_bwd(x[i : i + 8], w, dy[i : i + 8], rstd[i : i + 8])[1] for i in range(0, rows, 8)]
    want = torch.zeros(d, device=DEV)
    for part in parts:
        want = want + part
    assert torch.equal(ext.rmsnorm_bwd(x, w, dy, rstd)[1], want)


# ------------------------------------------------------------------------------------------------ decoding step
@pytest.mark.parametrize("n", [1, 16, 17, 33, 64, 128])
@pytest.mark.parametrize("rows,k", [(128, 64), (200, 200), (2560, 1088), (12800, 320), (128 * 149, 136), (128 * 300 - 8, 72)])
@pytest.mark.parametrize("tile", [0, 64, 128])
def test_decode_linear(n, rows, k, tile):
    """Tiles of 64 and 128 rows: fewer of them than SMs, a CTA per tile with two per SM, more tiles than that; ragged last
    tile, k tail; residual add and SwiGLU epilogues with the bits of the GEMM and the kernels that follow it."""
    from rl_engine.kernels.ops.base import require_ext
    from rl_engine.kernels.ops.sm100.gemm import gemm

    ext = require_ext()
    x, w = _randn(n, k, seed=n), _randn(rows, k, seed=rows, scale=k ** -0.5)
    res = _randn(n, rows, seed=5)
    y = x.double() @ w.double().t()
    product = gemm(torch.cat([x, _randn(200, k, seed=7)]), w)[:n]  # the engine of many rows
    plain = ext.decode_linear(x, w, False, None, tile)
    assert _rel(plain, y) < BF16 / 2
    assert torch.equal(plain, product)
    assert torch.equal(ext.decode_linear(x, w, False, res, tile), res + product)
    if rows % 128 == 0:
        assert torch.equal(ext.decode_linear(x, w, True, None, tile), ext.swiglu_packed_fwd(product.contiguous()))


@pytest.mark.parametrize("n", [1, 16, 33, 128])
@pytest.mark.parametrize("hq,hkv,bias", [(4, 2, False), (8, 1, True), (2, 2, True)])
@pytest.mark.parametrize("tile", [0, 64, 128])
def test_decode_qkv(n, hq, hkv, bias, tile):
    """Projection, bias, rotation, packing of the queries and cache write: the bits of the separate kernels."""
    from rl_engine.kernels.ops.base import require_ext
    from rl_engine.kernels.ops.sm100.gemm import gemm

    ext, k, heads = require_ext(), 200, hq + 2 * hkv
    x, w = _randn(n, k, seed=1), _randn(heads * 128, k, seed=2, scale=0.1)
    b = _randn(heads * 128, seed=3, scale=0.1) if bias else None
    angle = torch.rand(50, 64, device=DEV, generator=_gen(4)) * 6
    cos, sin = angle.cos(), angle.sin()
    positions = torch.randint(0, 50, (n,), device=DEV, generator=_gen(5))
    slots = torch.randperm(200, device=DEV, generator=_gen(6))[:n]
    ck, cv = _randn(200, hkv, 128, seed=7), _randn(200, hkv, 128, seed=8)
    got_k, got_v = ck.clone(), cv.clone()
    q = ext.decode_qkv(x, w, b, cos, sin, positions, slots, got_k, got_v, hq, tile)
    qkv = gemm(torch.cat([x, _randn(200, k, seed=9)]), w)[:n]
    qkv = (qkv if b is None else qkv + b).view(n, heads, 128)
    qk = ext.rope(qkv[:, : hq + hkv].contiguous(), positions, cos, sin)
    ck.index_copy_(0, slots, qk[:, hq:])
    cv.index_copy_(0, slots, qkv[:, hq + hkv :])
    rep = hq // hkv
    assert torch.equal(q, qk[:, :hq].reshape(n, hkv, rep, 128).permute(0, 2, 1, 3).reshape(n * rep, hkv, 128))
    assert torch.equal(got_k, ck) and torch.equal(got_v, cv)


@pytest.mark.parametrize("m", [1, 17, 100, 128])
@pytest.mark.parametrize("rows,k", [(200, 208), (4096, 4096), (128 * 149, 272), (128 * 300, 144)])
def test_few_row_fp8_gemm_has_the_bits_of_the_tall_engines(m, rows, k):
    from rl_engine.kernels.ops.sm100.gemm_fp8 import gemm_fp8, quantize_rows

    (x, sx), (w, sw) = quantize_rows(_randn(300, k, seed=1)), quantize_rows(_randn(rows, k, seed=2))
    full = gemm_fp8(x, sx, w, sw)
    assert torch.equal(gemm_fp8(x[:m], sx[:m].contiguous(), w, sw), full[:m])


@pytest.mark.parametrize("n,p,own,heads,kv,bias", [(1, 1, 1, 4, 2, False), (3, 300, 5, 8, 2, True), (40, 1500, 130, 8, 2, False),
                                                   (128, 200, 3, 4, 4, False)])
def test_decode_step_on_the_decode_kernels_matches_the_general_ones(n, p, own, heads, kv, bias):
    """One prefix range and many, one query tile and several, own keys across a tile; the cache rows that are written are
    the same up to one rounding.  Each route rounds about ten intermediate tensors per layer to bf16: 2 layers, 2^-8."""
    from rl_engine.models.config import ModelConfig
    from rl_engine.models.llama import LlamaModel

    cfg = ModelConfig("decode", 512, 256, 2, heads, kv, 128, 448, qkv_bias=bias)
    model = LlamaModel(cfg, dtype=torch.bfloat16, device=DEV, seed=3)
    rows = own + 2
    cache = model.new_kv_cache(p + n * rows)
    for i, (k, v) in enumerate(cache):
        k.copy_(_randn(*k.shape, seed=10 + i))
        v.copy_(_randn(*v.shape, seed=20 + i))
        if bias:
            with torch.no_grad():
                model.view(f"l{i}.bqkv").copy_(_randn(*model.view(f"l{i}.bqkv").shape, seed=30 + i, scale=0.1))
    tokens = torch.randint(0, 512, (n,), device=DEV, generator=_gen(1))
    positions = torch.full((n,), p + own - 1, dtype=torch.long, device=DEV)
    slots = p + torch.arange(n, device=DEV) * rows + own - 1
    prefix, layout = model.decode_layouts(n, p, rows, own)
    other = [(k.clone(), v.clone()) for k, v in cache]
    got = model.decode_step(tokens, positions, cache, slots, prefix, layout)
    want = model.decode_step(tokens, positions, other, slots, prefix, replace(layout, step=None))
    assert _rel(got, want) < 4 * BF16
    for (k, v), (k2, v2) in zip(cache, other):
        assert _rel(k, k2) < 4 * BF16 and _rel(v, v2) < 4 * BF16
    layout.seqs[:, 5] += 1  # advanced in place by the caller: both tables follow
    assert torch.equal(layout.step.seqs[layout.step.own_begin :, 5], layout.seqs[:, 5])


@pytest.mark.parametrize("p", [1, 200, 3000])
@pytest.mark.parametrize("heads,kv", [(8, 2), (4, 4)])
def test_decode_step_rows_have_the_same_bits_at_any_number_of_sequences(p, heads, kv):
    """Query tiles, prefix ranges, both routes of the projections, row maxima that grow by more than the kernel's lazy step: a
    sequence's hidden state and cache rows do not depend on who decodes with it."""
    from rl_engine.models.config import ModelConfig
    from rl_engine.models.llama import LlamaModel

    cfg, most, own = ModelConfig("rows", 512, 256, 2, heads, kv, 128, 448), 300, 3
    model = LlamaModel(cfg, dtype=torch.bfloat16, device=DEV, seed=3)
    start = [(_randn(p + most * own, kv, 128, seed=10 + i, scale=8.0), _randn(p + most * own, kv, 128, seed=20 + i)) for i in range(2)]
    with torch.no_grad():
        for i in range(2):
            model.view(f"l{i}.wqkv")[: heads * 128].mul_(4)
    tokens = torch.randint(0, 512, (most,), device=DEV, generator=_gen(1))
    seen = {}
    for n in (300, 257, 256, 129, 128, 65, 64, 33, 32, 31, 5, 1):
        cache = [(k[: p + n * own].clone(), v[: p + n * own].clone()) for k, v in start]
        positions = torch.full((n,), p + own - 1, dtype=torch.long, device=DEV)
        slots = p + torch.arange(n, device=DEV) * own + own - 1
        prefix, layout = model.decode_layouts(n, p, own, own)
        with torch.no_grad():
            got = model.decode_step(tokens[:n], positions, cache, slots, prefix, layout)
        rows = [got] + [t[slots] for pair in cache for t in pair]
        if not seen:
            seen = rows
        for a, b in zip(rows, seen):
            assert torch.equal(a, b[:n]), n


def test_rollout_does_not_read_what_the_cache_memory_held():
    """Rows of a key tile behind a sequence's last key are multiplied with zero weights; memory that held NaN must not get in."""
    from rl_engine.executors.native_rollout import NativeRolloutEngine
    from rl_engine.models.config import ModelConfig
    from rl_engine.models.llama import LlamaModel

    model = LlamaModel(ModelConfig("cache", 512, 256, 2, 4, 2, 128, 448), dtype=torch.bfloat16, device=DEV, seed=5)
    prompt = torch.randint(0, 512, (40,), device=DEV, generator=_gen(1))
    rows = 40 + 3 * 6
    poison = [torch.full((rows, 2, 128), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(64)]
    del poison
    for k, v in model.new_kv_cache(rows):
        assert bool((k == 0).all()) and bool((v == 0).all())
    out = NativeRolloutEngine(model, seed=5).generate(prompt, num_generations=3, max_new_tokens=6, top_k=20)
    assert torch.isfinite(out["rollout_logps"]).all()


@pytest.mark.parametrize("fp8", [False, True])
def test_decode_step_applies_the_head_norms(fp8):
    """A model with per-head q / k norms: teacher-forced steps against the rows of the packed forward, which normalises the heads.
    Weights far from one: a step without the norms misses by 1.03 of the hidden state's norm.  bf16 rounds about ten tensors per
    layer on either side; e4m3 codes are 2^-3 apart, rounded to within 2^-4, in four products a layer whose errors add up like
    independent ones: 2^-4 * sqrt(16) at most."""
    from rl_engine.kernels.ops.sm100.attention import grpo_group_layout
    from rl_engine.models.config import ModelConfig
    from rl_engine.models.llama import LlamaModel

    cfg = ModelConfig("norms", 512, 256, 2, 4, 2, 128, 448, qk_norm=True)
    model = LlamaModel(cfg, dtype=torch.bfloat16, device=DEV, seed=5)
    p, g, l = 70, 3, 5
    ids = torch.randint(0, 512, (p + g * l,), device=DEV, generator=_gen(6))
    prompt, comp = ids[:p], ids[p:].view(g, l)
    with torch.no_grad():
        for i in range(2):
            for j, name in enumerate(("q_norm", "k_norm")):
                model.view(f"l{i}.{name}").copy_(3 * torch.rand(128, device=DEV, generator=_gen(7 + j)))
        positions = torch.cat([torch.arange(p, device=DEV), (p + torch.arange(l, device=DEV)).repeat(g)])
        full = model.hidden_states(ids, positions, grpo_group_layout(p, g, l, DEV))[p:].view(g, l, -1)
        if fp8:
            model.enable_fp8_inference()
        cache = model.new_kv_cache(p + g * l)
        for (ck, cv), (pk, pv) in zip(cache, model.prefix_states(prompt)[1]):
            ck[:p].copy_(pk)
            cv[:p].copy_(pv)
        prefix, own = model.decode_layouts(g, p, l)
        for t in range(l):
            pos = torch.full((g,), p + t, dtype=torch.long, device=DEV)
            got = model.decode_step(comp[:, t].contiguous(), pos, cache, p + torch.arange(g, device=DEV) * l + t, prefix, own)
            own.seqs[:, 5] += 1
            assert _rel(got, full[:, t]) < (0.25 if fp8 else 8 * BF16)


@pytest.mark.parametrize("m", [1, 32, 100, 128])
def test_wide_gemm_rows_have_the_same_bits_at_any_number_of_rows(m):
    from rl_engine.kernels.ops.sm100.gemm import gemm

    x, w = _randn(300, 200, seed=1), _randn(128 * 148 + 72, 200, seed=2, scale=0.1)
    full = gemm(x, w)
    assert torch.equal(gemm(x[:m], w), full[:m])
    assert _rel(full, x.double() @ w.double().t()) < BF16 / 2


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


@pytest.mark.parametrize("n,kind", [(64, "one"), (65, "one"), (1000, "one"), (20000, "one"), (700, "mixed"), (131, "last")])
@pytest.mark.parametrize("d,dtype", [(200, torch.bfloat16), (13, torch.float32), (72, torch.float32), (5, torch.float16)])
def test_embedding_gradient_adds_a_row_in_batch_order(n, kind, d, dtype):
    """A table row is one 32-bit sum in the order of the batch, however its run lies in the chunks: the same bits."""
    from rl_engine.kernels.ops.sm100.model_ops import FusedEmbeddingSM100Op

    ids = {"one": torch.full((n,), 3), "mixed": (torch.arange(n) * 7) % 5, "last": (torch.arange(n) > 2) * 6 + 1}[kind].to(DEV)
    table = _randn(8, d, seed=1, dtype=dtype).requires_grad_(True)
    dy = _randn(n, d, seed=2, dtype=dtype)
    FusedEmbeddingSM100Op()(ids, table).backward(dy)
    want = torch.zeros(8, d)
    for i, row in zip(ids.tolist(), dy.float().cpu().unbind()):
        want[i] += row
    assert torch.equal(table.grad.cpu(), want.to(dtype))


def test_embedding_gradient_refuses_ids_outside_the_table():
    from rl_engine.kernels.ops.sm100.model_ops import FusedEmbeddingSM100Op

    table = _randn(10, 64, seed=1).requires_grad_(True)
    for bad in (-1, 10):
        out = FusedEmbeddingSM100Op()(torch.tensor([1, bad, 2], device=DEV), table)
        with pytest.raises(ValueError):
            out.sum().backward()


@pytest.mark.parametrize("n", [3, 200])
@pytest.mark.parametrize("bad", [-1, 10])
def test_refused_ids_leave_the_gradient_buffer_as_it_was(n, bad):
    """A run inside a chunk and one across a border beside the id outside the table, into a sink that holds a gradient."""
    from rl_engine.kernels.ops.sm100.model_ops import FusedEmbeddingSM100Op

    table = _randn(10, 64, seed=1).requires_grad_(True)
    sink = _randn(10, 64, seed=2)
    before = sink.clone()
    ids = torch.full((n,), 3, device=DEV)
    ids[n // 2] = bad
    out = FusedEmbeddingSM100Op()(ids, table, grad_sink=sink)
    with pytest.raises(ValueError):
        out.sum().backward()
    torch.cuda.synchronize()
    assert torch.equal(sink, before)


# ------------------------------------------------------------------------------------------------ sampler
def _draws(z, k, p, seed, offset):
    """The kernel's rule in fp64 on the host; a draw within 1e-5 of the border between two tokens allows both."""
    from rl_engine.kernels.ops.sm100.sampler import philox_uniform

    out = []
    for row, x in enumerate(z.double().cpu()):
        order = torch.argsort(x, descending=True, stable=True)
        kth = x[order[min(k, x.numel()) - 1]]
        order = order[: int((x >= kth).sum())]
        e = torch.exp(x[order] - x[order[0]])
        c = e.cumsum(0)
        keep = 1 + int((c[:-1] <= p * c[-1]).sum())
        at = philox_uniform(seed, offset, row) * c[keep - 1]
        near = lambda s: int(order[min(int(torch.searchsorted(c[:keep], at * s, right=True)), keep - 1)])
        out.append({near(1 - 1e-5), near(1.0), near(1 + 1e-5)})
    return out


@pytest.mark.parametrize("rows,vocab", [(1, 140000), (3, 40001), (75, 33000), (200, 4096), (5, 37)])
@pytest.mark.parametrize("k", [1, 50, 513, 1000])
@pytest.mark.parametrize("shape", ["normal", "rising", "ties"])
def test_top_k_sampler_over_splits_and_fallbacks(rows, vocab, k, shape):
    """1 to 8 CTAs per row, unaligned rows, k above the vocabulary, a row whose head is far below its tail (the candidates
    overflow) and masses of ties at the k-th place."""
    from rl_engine.kernels.ops.sm100.sampler import sample_topk_topp

    z = torch.randn(rows, vocab, device=DEV, generator=_gen(rows + k)) * 2
    if shape == "rising":
        z = z * 0.01 + torch.linspace(0, 40, vocab, device=DEV)
    elif shape == "ties":
        z = torch.round(z)
        if int((z[0] == z[0].kthvalue(vocab - min(k, vocab) + 1).values).sum()) > 1000:
            z[:, ::3] = z[:, ::3] + 0.25  # at most 2048 candidates are ordered
    if k >= vocab:
        pytest.skip("top_k >= vocab is the full-vocabulary kernel")
    ids, _ = sample_topk_topp(z, top_k=k, top_p=0.95, temperature=1.0, seed=7, offset=11)
    kth = z.kthvalue(vocab - k + 1, dim=-1).values
    if int((z >= kth[:, None]).sum(-1).max()) > 2048:
        assert bool((z.gather(1, ids[:, None])[:, 0] >= kth).all())
        return
    allowed = _draws(z, k, 0.95, 7, 11)
    assert all(int(i) in a for i, a in zip(ids.cpu(), allowed))


@pytest.mark.parametrize("rows,vocab", [(1, 140001), (3, 66000), (20, 50257), (75, 33001), (149, 9000), (160, 101000), (5, 300), (200, 64)])
@pytest.mark.parametrize("k", [1, 20, 63, 200, 256, 257, 700, 1024])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_top_k_draws_do_not_depend_on_the_kernel(rows, vocab, k, dtype):
    """A CTA per row (both instances), slices with either bound, one to eight of them: the same ids and log-probs, with ties, rows whose
    head is far below their tail (candidates overflow) and masked stretches; and what the sizes select is one of them."""
    from rl_engine.kernels.ops.base import require_ext

    ext = require_ext()
    z = (2 * torch.randn(rows, vocab, device=DEV, generator=_gen(rows + k)))
    z[rows // 2] += torch.linspace(0, 40, vocab, device=DEV)
    z[0, : vocab // 2] = float("-inf")
    z = z.to(dtype)
    if min(k, vocab) > int((z[0] > float("-inf")).sum()):
        pytest.skip("ties at -inf fill the buffer")
    want = ext.sample(z, k, 0.95, 0.8, 7, 11, True, 0)
    for route in (-1, 1, 2):
        if route == 1 and k > 256:
            continue
        ids, logprob = ext.sample(z, k, 0.95, 0.8, 7, 11, True, route)
        assert torch.equal(ids, want[0]) and torch.equal(logprob, want[1]), route
    # the same rows in a batch of another size
    part = ext.sample(z[:1].contiguous(), k, 0.95, 0.8, 7, 11, True)
    assert torch.equal(part[0], want[0][:1]) and torch.equal(part[1], want[1][:1])


# ------------------------------------------------------------------------------------------------ log-prob gradient
@pytest.mark.parametrize("v", [5, 1024, 4099, 8192])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("pitch", [0, 1, 8])
def test_selected_logprob_gradient_alignment(v, dtype, pitch):
    """Rows that share their offset from a 16-byte boundary with the gradient's (peeled) and rows that do not."""
    from rl_engine.kernels.ops.sm100.logp_autograd import selected_logprobs

    n = 9
    store = _randn(n, v + pitch, seed=v, dtype=dtype)
    z = store[:, :v].detach().requires_grad_(True)
    ids = torch.randint(0, v, (n,), device=DEV, generator=_gen(2))
    ids[:2] = torch.tensor([0, v - 1], device=DEV)
    mask = torch.ones(n, dtype=torch.bool, device=DEV)
    mask[3] = False
    g = torch.randn(n, device=DEV, generator=_gen(3))
    (grad,) = torch.autograd.grad(selected_logprobs(z, ids, mask), [z], g)
    want = -torch.softmax(z.detach().double(), -1)
    want[torch.arange(n), ids] += 1
    want *= (g * mask).double()[:, None]
    assert _rel(grad, want) < {torch.float32: 1e-6, torch.bfloat16: BF16 / 2, torch.float16: 2.0 ** -11}[dtype] * 2
    assert bool((grad[3] == 0).all())


# ------------------------------------------------------------------------------------------------ experts, attention backward
@pytest.mark.parametrize("tokens", [1, 5, 130, 700])
@pytest.mark.parametrize("h,e,k,f", [(256, 32, 4, 64), (128, 8, 2, 192), (512, 4, 1, 128)])
def test_moe_with_empty_experts_and_ragged_blocks(tokens, h, e, k, f):
    """Experts without a token (their weight gradient is exactly zero), blocks of any length, per-expert gradients with and
    without 256-row tiles: against the oracle in fp32.  Every stored tensor on the way is rounded to bf16 once."""
    from rl_engine.kernels.ops.sm100.moe import FusedMoESM100Op, NativeMoEOp

    x, r = _randn(tokens, h, seed=1), _randn(e, h, seed=2, scale=h ** -0.5)
    w1, w2 = _randn(e * 2 * f, h, seed=3, scale=0.05), _randn(e * h, f, seed=4, scale=0.05)
    args = [t.requires_grad_(True) for t in (x, r, w1, w2)]
    oracle = [t.detach().float().requires_grad_(True) for t in args]
    dout = _randn(tokens, h, seed=5)
    torch.full((1 << 24,), float("nan"), device=DEV)  # rows that no kernel writes would otherwise look harmless
    out = FusedMoESM100Op()(*args, k)
    want = NativeMoEOp()(*oracle, k)
    assert _rel(out.detach(), want.detach()) < 2 * BF16
    grads, wanted = torch.autograd.grad(out, args, dout), torch.autograd.grad(want, oracle, dout.float())
    # the router's gradient is made of differences w_i w_j (dw_i - dw_j) of dot products of rounded rows: with few tokens each
    # rounding counts up to |dw_i| + |dw_j| over their difference times, here up to four
    for i, (got, ref) in enumerate(zip(grads, wanted)):
        assert _rel(got, ref) < (12 if i == 1 else 3) * BF16
    hit = wanted[3].view(e, -1).abs().sum(1) > 0
    assert bool((grads[3].view(e, -1)[~hit] == 0).all()) and bool((grads[2].view(e, -1)[~hit] == 0).all())


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


@pytest.mark.parametrize("rows,vocab", [(3, 40001), (160, 4096), (2, 150000), (4, 5)])
@pytest.mark.parametrize("p", [0.5, 0.95, 1.0])
@pytest.mark.parametrize("shape", ["normal", "flat", "steep", "masked"])
def test_nucleus_sampler_integer_masses(rows, vocab, p, shape):
    """The cut and the draw on 40-bit integer masses, restated on the host; flat logits overflow the gathered step and take
    the search over the row.  A draw within 1e-5 of a token's border allows its neighbour."""
    from rl_engine.kernels.ops.sm100.sampler import philox_uniform, sample_topk_topp

    z = {"normal": 2.0, "flat": 1e-4, "steep": 12.0, "masked": 2.0}[shape] * torch.randn(rows, vocab, device=DEV, generator=_gen(vocab))
    if shape == "masked" and vocab > 8:
        z[:, : vocab // 2] = float("-inf")
    got, _ = sample_topk_topp(z, top_k=None, top_p=p, temperature=0.8, seed=3, offset=2)
    x = z.double().cpu()
    for row in range(rows):
        mass = torch.floor(torch.exp((x[row] - x[row].max()) / 0.8) * 2.0 ** 40)
        order = torch.argsort(x[row], descending=True, stable=True)
        c = mass[order].cumsum(0)
        i = int(got[row])
        first = min(int(torch.searchsorted(c, max(1.0, p * float(c[-1])) * (1 + 1e-5))), vocab - 1)
        assert x[row, i] >= x[row, order[first]]  # inside the nucleus
        cut = x[row, order[min(int(torch.searchsorted(c, max(1.0, p * float(c[-1])))), vocab - 1)]]
        kept = torch.where(x[row] >= cut, mass, torch.zeros_like(mass)).cumsum(0)
        t = philox_uniform(3, 2, row) * float(kept[-1])
        lo, hi = (0.0 if i == 0 else float(kept[i - 1])), float(kept[i])
        assert lo - 2e-5 * float(kept[-1]) <= t <= hi + 2e-5 * float(kept[-1])


@pytest.mark.parametrize("form", ["dense", "odd offset", "odd pitch", "transposed", "row", "3-d", "float32"])
def test_residuals_of_any_layout_are_added(form):
    """Residuals that the epilogue can address and those that it cannot: the sum (each rounded once, as is the
    product) and its gradient; a residual that does not broadcast with the product is refused, as by the addition."""
    from rl_engine.kernels.ops.sm100.lean_blocks import residual_linear, swiglu_linear

    n, k, m = 24, 64, 40
    x, w = _randn(n, k, seed=1).requires_grad_(True), _randn(m, k, seed=2, scale=0.2).requires_grad_(True)
    gu, wd = _randn(n, 2 * k, seed=3).requires_grad_(True), _randn(m, k, seed=4, scale=0.2)
    make = {"dense": lambda: _randn(n, m, seed=5), "odd offset": lambda: _randn(n * m + 1, seed=5)[1:].view(n, m),
            "odd pitch": lambda: _randn(n, m + 3, seed=5)[:, 1 : m + 1], "transposed": lambda: _randn(m, n, seed=5).t(),
            "row": lambda: _randn(1, m, seed=5), "3-d": lambda: _randn(2, n // 2, m, seed=5),
            "float32": lambda: _randn(n, m, seed=5, dtype=torch.float32)}[form]
    res = make().requires_grad_(True)
    for fused, product in ((lambda: residual_linear(res, x, w), lambda: x @ w.t()),
                           (lambda: swiglu_linear(gu, wd, residual=res), lambda: swiglu_linear(gu, wd))):
        if form == "3-d":
            with pytest.raises(RuntimeError):
                fused()
            continue
        got, plain = fused(), product()
        assert got.shape == (res + plain).shape and got.dtype == (res + plain).dtype
        assert _rel(got.detach(), res.detach().double() + plain.detach().double()) < BF16
        (a,), (b,) = (torch.autograd.grad(out.sum(), [res]) for out in (got, res + plain))
        assert torch.equal(a, b)


@pytest.mark.parametrize("micro", [None, 2])
@pytest.mark.parametrize("chunk", [4096, 128])
def test_gradients_added_by_the_gemms_equal_those_added_by_autograd(micro, chunk):
    """One pass, and micro-batches after a prompt pass; LM-head gradients of one chunk and of several: the same bits."""
    from rl_engine.kernels.registry import kernel_registry
    from rl_engine.models.config import ModelConfig
    from rl_engine.models.grpo import GRPOTrainer, synthetic_batch
    from rl_engine.models.llama import LlamaModel

    cfg = ModelConfig("sink", 640, 256, 2, 4, 2, 128, 384)
    batch = synthetic_batch(640, 70, 6, 90, seed=2).to(DEV)
    op = kernel_registry.get_op("linear_logp")
    before, op.bwd_chunk_tokens = op.bwd_chunk_tokens, chunk
    try:
        grads = []
        for sink in (True, False):
            trainer = GRPOTrainer(LlamaModel(cfg, dtype=torch.bfloat16, device=DEV, seed=4), micro_group=micro)
            trainer.sink_weight_grads = sink
            trainer.opt.zero_grad()
            trainer.forward_backward(batch)
            grads.append({n: p.grad.clone() for n, p in trainer.model.named_views().items()})
            assert trainer.model.sink_weight_grads is None
        for name, want in grads[1].items():
            assert torch.equal(grads[0][name], want), name
        # outside the trainer's own pass, gradients are returned
        model = trainer.model
        out = trainer.policy_logps(batch).sum()
        (g,) = torch.autograd.grad(out, [model.view("l0.wo")])
        assert float(g.float().norm()) > 0
    finally:
        op.bwd_chunk_tokens = before


@pytest.mark.parametrize("how", ["node", "tensor", "after"])
def test_hooks_on_a_parameter_see_its_gradient_in_a_trainers_pass(how):
    """A hook on the AccumulateGrad node, on the parameter or after its accumulation fires as without sinks, and the gradient is
    the same."""
    from rl_engine.models.config import ModelConfig
    from rl_engine.models.grpo import GRPOTrainer, synthetic_batch
    from rl_engine.models.llama import LlamaModel

    batch = synthetic_batch(640, 70, 6, 90, seed=2).to(DEV)
    names, grads = ("embed", "l0.wqkv", "l0.mlp_norm", "l1.w_down", "lm_head"), []
    for watch in (False, True):
        trainer = GRPOTrainer(LlamaModel(ModelConfig("hooks", 640, 256, 2, 4, 2, 128, 384), dtype=torch.bfloat16, device=DEV, seed=4))
        trainer.opt.zero_grad()
        model, seen, nodes = trainer.model, [], []
        for name in names if watch else ():
            p = model.view(name)
            if how == "node":
                nodes.append(p.expand_as(p).grad_fn.next_functions[0][0])
                nodes[-1].register_hook(lambda *a, n=name: seen.append(n))
            elif how == "tensor":
                p.register_hook(lambda g, n=name: seen.append(n))
            else:
                p.register_post_accumulate_grad_hook(lambda p, n=name: seen.append(n))
        trainer.forward_backward(batch)
        assert set(seen) == set(names if watch else ())
        grads.append({n: p.grad.clone() for n, p in model.named_views().items()})
    for name, want in grads[0].items():
        assert torch.equal(grads[1][name], want), name
