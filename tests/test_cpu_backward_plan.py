"""Work lists of the attention backward on the CPU: however the query-block lists are cut, every (key tile, query block) pair
appears once, partial slots are used once and the reduction covers them in order."""

import pytest

from rl_engine.kernels.ops.sm100.attention import grpo_group_layout, make_layout
from rl_engine.kernels.ops.sm100.attention_bwd_kernels import MAX_BLOCKS_PER_ITEM, build_plan


@pytest.mark.parametrize("p,g,l,causal", [(1, 2, 1, True), (333, 8, 211, True), (1024, 16, 512, True), (130, 3, 64, False)])
def test_pieces_cover_every_list_once(p, g, l, causal):
    if causal:
        layout = grpo_group_layout(p, g, l, "cpu")
    else:
        layout = make_layout([(i * l, l, 0, p, 0, 0) for i in range(g)], False, "cpu")
    items, blocks, jobs, slots, written = build_plan(layout)
    assert written == ((p + g * l, p + g * l) if causal else (g * l, p))
    per_tile = {}
    for k_abs, k_len, _, begin, end, slot, _, _ in items.tolist():
        assert 0 < end - begin <= MAX_BLOCKS_PER_ITEM
        per_tile.setdefault((k_abs, k_len), []).append((slot, begin, end))
    covered = sorted((b, e) for pieces in per_tile.values() for _, b, e in pieces)
    assert covered[0][0] == 0 and covered[-1][1] == len(blocks)
    assert all(a[1] == b[0] for a, b in zip(covered, covered[1:]))
    used = sorted(s for pieces in per_tile.values() for s, _, _ in pieces if s >= 0)
    assert used == list(range(slots))
    reduced = {(k, n): (a, b) for k, n, a, b in jobs.tolist()}
    for tile, pieces in per_tile.items():
        if len(pieces) == 1:
            assert pieces[0][0] == -1 and tile not in reduced
        else:
            order = sorted(pieces)
            assert reduced[tile] == (order[0][0], order[-1][0] + 1)
            assert [b for _, b, _ in order] == sorted(b for _, b, _ in order)


def test_lists_are_cut_after_64_blocks_whatever_the_grid():
    """The cuts decide the order of a gradient's 32-bit sums: they follow from the list alone."""
    for p, g, l in ((333, 8, 211), (1024, 16, 512)):
        layout = grpo_group_layout(p, g, l, "cpu")
        items, _, jobs, _, _ = build_plan(layout)
        split = {k for k, *_ in jobs.tolist()}
        for k_abs, _, _, begin, end, slot, _, _ in items.tolist():
            assert (slot >= 0) == (k_abs in split)
        lengths = {}
        for k_abs, _, _, begin, end, _, _, _ in items.tolist():
            lengths.setdefault(k_abs, []).append((begin, end - begin))
        for pieces in lengths.values():
            sizes = [n for _, n in sorted(pieces)]
            assert all(n == 64 for n in sizes[:-1]) and 1 <= sizes[-1] <= 64
