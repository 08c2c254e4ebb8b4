"""The attention plan's list of decoded rows (no GPU needed)."""
import pytest
import torch

from nanoinfer_b200.parts.attention import SORTED_DECODE_ROWS, AttentionPlan


@pytest.mark.parametrize("n", [1, SORTED_DECODE_ROWS - 1, SORTED_DECODE_ROWS, 40])
@pytest.mark.parametrize("portion", [0, 5])
def test_many_decoded_rows_are_listed_longest_context_first(n, portion):
    pos0 = [(37 * e) % 101 for e in range(n)]
    starts = list(range(n + 1))
    if portion:                       # a prompt portion in the middle of the entries
        at = n // 2
        starts = starts[:at + 1] + [s + portion for s in starts[at:]]
        pos0 = pos0[:at] + [3] + pos0[at:]
    plan = AttentionPlan(starts, pos0, device=torch.device("cpu"))
    rows = {starts[e]: pos0[e] for e in range(len(pos0)) if starts[e + 1] - starts[e] == 1}
    listed = plan.words[:plan.n_decode]
    assert plan.n_decode == n and sorted(listed) == sorted(rows)
    contexts = [rows[r] for r in listed]
    if n >= SORTED_DECODE_ROWS:
        assert contexts == sorted(contexts, reverse=True) and plan.decode_rows.tolist() == listed
    else:
        assert listed == sorted(rows) and (plan.decode_rows is None) == (portion == 0)


@pytest.mark.parametrize("n", [1, SORTED_DECODE_ROWS - 1, SORTED_DECODE_ROWS, 40])
@pytest.mark.parametrize("portion", [0, 130])
def test_decoded_rows_are_listed_in_order_beside_the_longest_first(n, portion):
    pos0 = [(37 * e) % 101 for e in range(n)]
    starts = list(range(n + 1))
    if portion:
        at = n // 2
        starts = starts[:at + 1] + [s + portion for s in starts[at:]]
        pos0 = pos0[:at] + [3] + pos0[at:]
    plan = AttentionPlan(starts, pos0, device=torch.device("cpu"))
    rows = [starts[e] for e in range(len(pos0)) if starts[e + 1] - starts[e] == 1]
    assert (plan.rows_in_order.tolist() == rows) if portion else (plan.rows_in_order is None and rows == list(range(n)))
    assert (plan.longest_first is None) == (n < SORTED_DECODE_ROWS)
    if plan.longest_first is not None:
        assert sorted(plan.longest_first.tolist()) == rows
    if portion:
        assert plan.prefill_rows.tolist() == [r for r in range(n + portion) if r not in rows]
        assert plan.tiles.numel() == 2 * plan.n_tiles == 6 and plan.wide_tiles.tolist() == [n // 2, 128, n // 2, 0]


def test_rows_are_launched_longest_first_where_the_device_does_not_hold_them_at_once():
    from nanoinfer_b200.kernels.ops import DECODE_RESIDENT_BLOCKS, decode_longest_first

    assert not decode_longest_first(48 * 16, DECODE_RESIDENT_BLOCKS) and not decode_longest_first(74 * 12, DECODE_RESIDENT_BLOCKS)
    assert decode_longest_first(56 * 16, DECODE_RESIDENT_BLOCKS) and decode_longest_first(75 * 12, DECODE_RESIDENT_BLOCKS)
    assert decode_longest_first(56 * 8, DECODE_RESIDENT_BLOCKS // 2)     # (head sizes beyond 64: three blocks an SM)


@pytest.mark.parametrize("window", [0, 1, 100, 128, 500])
def test_work_of_the_wide_tiles_counts_the_key_tiles_that_are_walked(window):
    lens, pos0 = [1, 300, 128, 129, 1, 2], [40, 0, 1000, 127, 0, 255]
    starts = [sum(lens[:e]) for e in range(len(lens) + 1)]
    walks = []
    for n, p in zip(lens, pos0):
        for off in range(0, n, 128) if n > 1 else ():
            rows = range(p + off, p + min(off + 128, n))
            walks.append(len(range(max(0, rows[0] - window + 1) // 128 if window else 0, rows[-1] // 128 + 1)))
    plan = AttentionPlan(starts, pos0)
    assert plan.n_wide_tiles == len(walks) and plan.wide_work(window) == (sum(walks), max(walks))
    assert AttentionPlan([0, 1], [5]).wide_work(window) == (0, 0)


def test_blocks_of_the_prefill_attention_are_left_alone_while_the_device_holds_them_and_where_one_is_long():
    from nanoinfer_b200.kernels.ops import prefill_blocks_alone

    assert prefill_blocks_alone(12, 12, 12, 1) and prefill_blocks_alone(1, 148, 5000, 60)   # 144 and 148 blocks
    assert prefill_blocks_alone(12, 16, 136, 16)                                            # a triangle of 2,048 rows
    assert not prefill_blocks_alone(12, 24, 108, 8) and not prefill_blocks_alone(12, 32, 528, 32)
    assert not prefill_blocks_alone(25, 64, 288, 8)
