"""The states of newly opened slots are zeroed, by runs of neighbours or by an index, and no others."""
from types import SimpleNamespace

import pytest
import torch

from rustinfer_b200.engine.runner import ModelRunner
from rustinfer_b200.parts.base import FixedState, PagedKV


@pytest.mark.parametrize("slots", [[0], [3, 2, 2], [7, 0, 4], [0, 2, 4, 6], [0, 2, 4, 6, 9], [11, 9, 7, 5, 3, 1, 1], list(range(12))])
def test_only_the_new_slots_are_zeroed(slots):
    storage = [torch.ones(2, 12, 3, 4), torch.ones(5), torch.ones(1, 12, 2)]
    groups = [SimpleNamespace(need=n) for n in (FixedState((3, 4)), PagedKV(1, 4, None), FixedState((2,)))]
    runner = SimpleNamespace(cache=SimpleNamespace(newly_opened_slots=list(slots)), layout=SimpleNamespace(groups=groups), group_storage=storage)
    ModelRunner._zero_new_state(runner)
    for i in (0, 2):
        for s in range(12):
            assert (storage[i][:, s] == (0 if s in slots else 1)).all()
    assert (storage[1] == 1).all() and runner.cache.newly_opened_slots == []
