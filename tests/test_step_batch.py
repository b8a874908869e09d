"""The packed arrays of a step, on the CPU: what the rows of short portions beside long ones are."""
import pytest
import torch

from hipinfer_b200.engine import StepEntry, build_step_batch
from hipinfer_b200.engine.batch import SHORT_ROWS


def step(portions):
    """portions: (tokens before, new tokens) of each request; one cache group with pages of four tokens."""
    entries = [StepEntry(r, list(range(100 * r, 100 * r + n)), [n - 1]) for r, (_, n) in enumerate(portions)]
    tables = [[list(range(-(-(c + n) // 4)))] for c, n in portions]
    return build_step_batch(entries, [c for c, _ in portions], list(range(len(portions))), tables, [[list(range(c, c + n))] for c, n in portions], 1, "cpu")


@pytest.mark.parametrize("portions,rows,last", [
    ([(7, 1), (0, 40), (300, 15), (9, 16), (2, 3)], [0] + list(range(41, 56)) + list(range(72, 75)), 314),
    ([(0, 40), (5, 16)], [], 0),                       # all long
    ([(500, 1), (3, 64)], [0], 500),
    ([(3, 64), (500, 2)], [64, 65], 501)])
def test_rows_of_short_portions(portions, rows, last):
    b = step(portions)
    got, most = b.short_rows(SHORT_ROWS)
    assert got.dtype == torch.int32 and got.tolist() == rows and most == last
    assert b.short_rows(SHORT_ROWS)[0] is got                              # made once a step
    assert (b.short_list is None) == (not rows)                            # packed with the step where there are any
    assert b.positions[rows].tolist() == [c + i for c, n in portions if n < SHORT_ROWS for i in range(n)]
    assert b.tokens.tolist() == [100 * r + i for r, (_, n) in enumerate(portions) for i in range(n)]      # nothing else has moved
    assert b.slot_maps[0].tolist() == [c + i for c, n in portions for i in range(n)]


def test_rows_of_short_portions_by_another_limit():
    b = step([(7, 1), (0, 40), (300, 15), (2, 3)])
    assert b.short_rows(4)[0].tolist() == [0, 56, 57, 58] and b.short_rows(4)[1] == 7
    assert b.short_rows(SHORT_ROWS)[0].tolist() == [0] + list(range(41, 59))
    assert b.short_rows(64)[0].tolist() == list(range(59)) and b.short_rows(64)[1] == 314


def test_a_step_of_short_portions_alone_packs_no_list():
    """No kernel asks for one: the row kernels run over all rows."""
    b = step([(7, 1), (30, 5)])
    assert b.short_list is None and b.short_rows(SHORT_ROWS)[0].tolist() == list(range(6))
