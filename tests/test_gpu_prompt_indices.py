"""A step of many tokens takes its ids as one array: what was refused and what was taken one by one stays so."""
import numpy as np
import pytest
import torch

from rustinfer_b200.cache.pages import OutOfPages, PagePool
from rustinfer_b200.engine.runner import StepEntry, _flat_ids


def test_every_kind_of_list_is_the_same_array():
    ids = [int(t) for t in np.random.RandomState(1).randint(0, 50, 20)]
    for tokens in (ids, tuple(ids), np.array(ids), np.array(ids, dtype=np.int32), [np.int64(t) for t in ids]):
        flat = _flat_ids([StepEntry(0, tokens, ()), StepEntry(1, [49], ())], 50)
        assert flat.dtype == np.int64 and flat.tolist() == [*ids, 49]
    for other in ([*ids, 50], [*ids, -1], [*ids, 1 << 70], [*ids, 50.0], np.array([*ids, 50])):
        assert _flat_ids([StepEntry(0, other, ())], 50) is None          # looked at one by one, and refused there
    assert _flat_ids([StepEntry(0, [float(t) for t in ids], ())], 50) is None


def test_pages_at_once_are_the_smallest_and_come_back():
    pool, held = PagePool(64), []
    rng = np.random.RandomState(3)
    for _ in range(300):
        if held and rng.rand() < 0.5:
            pool.free(held.pop(rng.randint(len(held))))
        else:
            n, free = int(rng.randint(1, 20)), sorted(pool.free_set())
            if n > len(free):
                with pytest.raises(OutOfPages):
                    pool.alloc(n)
                continue
            held.append(pool.alloc(n))
            assert held[-1] == free[:n]
    assert pool.free_set() | {p for t in held for p in t} == set(range(64)) and pool.free_count + sum(map(len, held)) == 64


@pytest.mark.gpu
def test_ids_are_looked_at_in_long_steps_too(tmp_path):
    # the 32-bit engine: its logits are the same bits every time (a bfloat16 step of 20 tokens adds its products' slices in the order they arrive)
    from helpers import make_sharp_model
    from rustinfer_b200.engine.runner import ModelRunner, StepEntry, StepError
    folder = make_sharp_model(str(tmp_path / "model"), "D")
    runner = ModelRunner(folder, dtype="float32", max_model_len=64, max_batch_seqs=2, max_batch_tokens=64, num_pages=8, capture_sizes=[])
    vocab = runner.spec.vocab_size
    ids = [int(t) for t in np.random.RandomState(1).randint(0, vocab, 20)]
    want = None
    for tokens in (ids, tuple(ids), np.array(ids), np.array(ids, dtype=np.int32), [float(t) for t in ids], [np.int64(t) for t in ids]):
        runner.open(0)
        got = runner.step([StepEntry(0, tokens, (19,))])
        runner.close(0)
        want = got.clone() if want is None else want
        assert torch.equal(got, want)
    runner.open(0)
    for bad in ([*ids, vocab], [*ids, -1], [*ids, 1 << 70], [*ids, float(vocab)]):
        with pytest.raises(StepError, match="outside"):
            runner.step([StepEntry(0, bad, ())])
    assert runner.cache.length(0) == 0 and torch.equal(runner.step([StepEntry(0, ids, (19,))]), want)
