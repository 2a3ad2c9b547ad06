"""Fused linear -> log-prob: what the host decides (record cuts, buffers), looked at without a GPU."""

import pytest
import torch

from rl_engine.kernels.ops.base import _C, _EXT_AVAILABLE


@pytest.mark.skipif(not _EXT_AVAILABLE, reason="the native extension is not built")
@pytest.mark.parametrize("world", [1, 2, 8])
@pytest.mark.parametrize("vocab", [1, 8192, 8193, 50257, 128256])
def test_records_follow_from_the_vocabulary_alone(world, vocab):
    """A row's sums are cut at multiples of 8192 columns at any batch size and any number of ranks; tensor parallelism sends
    one record a cut to every peer."""
    for tokens in (1, 777, 8192):
        records, n_pad, row_tiles = _C.linear_logp_workspace_shape(tokens, vocab, world)
        assert records == -(-vocab // 8192)
        assert (n_pad, row_tiles) == (-(-tokens // 128) * 128, -(-tokens // 128))


def test_two_backward_passes_never_share_a_dz_buffer():
    """Passes on two streams run at the same time: each has a buffer of its own for as long as it holds it."""
    from rl_engine.kernels.ops.sm100 import linear_logp

    first, second = (linear_logp.dz_buffer(torch.device("cpu"), 128, 1001) for _ in range(2))
    assert first.data_ptr() != second.data_ptr()
    assert first.shape == (128, 1008) and first.dtype == torch.bfloat16
