"""The step's integer arrays, built on the host."""
import numpy as np
import pytest
import torch

from torchinferno_b200.engine.batch import EntryPlacement, build_batch


def _placements(lens, starts):
    rows = np.cumsum([0] + list(lens))
    return [EntryPlacement(i, 7 - i, int(rows[i]), n, s) for i, (n, s) in enumerate(zip(lens, starts))]


@pytest.mark.parametrize("lens", [(1, 1), (0, 2), (1,), (2, 0), (3, 1, 0, 4), (0, 1, 1, 2)])
def test_arrays_of_a_step_with_empty_portions(lens):
    starts = [5 * i for i in range(len(lens))]
    tokens = [[10 * i + j for j in range(n)] for i, n in enumerate(lens)]
    batch, _ = build_batch(_placements(lens, starts), tokens, [() for _ in lens], [], torch.device("cpu"))
    assert batch.token_ids.tolist() == sum(tokens, [])
    assert batch.positions.tolist() == [s + j for s, n in zip(starts, lens) for j in range(n)]
    assert batch.token_slot.tolist() == [7 - i for i, n in enumerate(lens) for _ in range(n)]
    assert batch.q_start.tolist() == [sum(lens[:i]) for i in range(len(lens) + 1)]


@pytest.mark.parametrize("convert", [list, tuple, np.array, torch.tensor, lambda t: [torch.tensor([v]) for v in t],
                                     lambda t: [np.int64(v) for v in t], lambda t: [str(v) for v in t]])
def test_tokens_in_any_form_that_int_takes(convert):
    lens, tokens = (3, 1, 2), [[4, 5, 6], [7], [8, 9]]
    batch, _ = build_batch(_placements(lens, (0, 3, 1)), [convert(t) for t in tokens], [() for _ in lens], [], torch.device("cpu"))
    assert batch.token_ids.tolist() == [4, 5, 6, 7, 8, 9]
