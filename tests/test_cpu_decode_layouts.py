"""Tables of a decoding step, looked at on the CPU: nothing is launched."""

from dataclasses import replace

import pytest
import torch

from rl_engine.kernels.ops.base import _EXT_AVAILABLE
from rl_engine.kernels.ops.sm100.attention import make_layout
from rl_engine.models.config import ModelConfig
from rl_engine.models.llama import LlamaModel


def _model(**kw):
    return LlamaModel(ModelConfig("layouts", 64, 256, 1, 8, 2, 128, 64, **kw), dtype=torch.float32, device="cpu")


class _Ran(Exception):
    pass


@pytest.mark.skipif(not _EXT_AVAILABLE, reason="the native extension is not built")
@pytest.mark.parametrize("n", [0, 1, 3, 4, 5, 8])
def test_decode_step_refuses_layouts_of_another_number_of_sequences(n, monkeypatch):
    """The attention kernels store a row for every query row of the tables, so tables for more sequences than the call has
    would write past its buffers, tables for fewer would leave rows unwritten: refused before anything runs."""
    model = _model()
    monkeypatch.setattr(model, "supports_prefix_cache", lambda: True)

    def embed(_ids):
        raise _Ran

    monkeypatch.setattr(model, "embed_tokens", embed)
    tokens = torch.zeros(n, dtype=torch.long)
    prefix, own = model.decode_layouts(4, 300, 16, 2)
    prefix_n, own_n = model.decode_layouts(n, 300, 16, 2)
    call = lambda p, o: model.decode_step(tokens, tokens, [], tokens, p, o)
    with pytest.raises(_Ran):
        call(prefix_n, own_n)
    with pytest.raises(_Ran):
        call(prefix_n, replace(own_n, step=None))
    if n != 4:
        for p, o in ((prefix, own), (prefix, replace(own, step=None)), (prefix_n, own), (prefix, own_n)):
            with pytest.raises(ValueError, match="was not built for"):
                call(p, o)
    # as many rows, in other places: the last one lies outside the call's
    if n == 4:
        shifted = make_layout([(1, 16, 0, 300, 0, 0)], False, "cpu")
        with pytest.raises(ValueError):
            call(shifted, own)


def test_joint_tables_name_their_query_rows():
    model = _model()
    for n, p in ((1, 1), (40, 1500), (3, 0)):
        _, own = model.decode_layouts(n, p, 16, 2)
        rows = n * 4
        assert own.step.rows == rows
        assert own.step.seqs[: own.step.own_begin, 1].eq(rows).all()
        # part i ends inside the output of `parts` times `rows` rows
        ends = own.step.seqs[:, 0] + own.step.seqs[:, 1] + own.step.seqs[:, 6]
        assert int(ends.max()) <= own.step.parts * rows


def test_joint_tables_are_built_for_models_whose_step_reads_them():
    """fp8 projections and per-head norms decode on the general kernels: a private own table, no joint one."""
    fp8 = _model()
    fp8._fp8_linears = {"l0.wqkv": object()}
    for model, joint in ((_model(), True), (fp8, False), (_model(qk_norm=True), False)):
        prefix, own = model.decode_layouts(3, 300, 16, 2)
        assert (own.step is not None) == joint
        own.seqs[:, 5] += 1
        assert model.decode_layouts(3, 300, 16, 2)[1].seqs[:, 5].eq(2).all()
