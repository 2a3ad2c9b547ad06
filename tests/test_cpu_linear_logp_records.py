"""How the fused linear -> log-prob forward cuts the vocabulary, looked up on the host: no GPU."""

import pytest

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
