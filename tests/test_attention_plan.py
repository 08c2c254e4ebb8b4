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
