"""What a decode batch begins with, as the host describes it, without a device."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from cpmcu_b200.engine.decode import DecodeRunner, _Bucket, bucket_size
from cpmcu_b200.memory import Staging
from cpmcu_b200.sampling import SamplingParams


def _runner(lengths):
    cpu = torch.device("cpu")
    r = object.__new__(DecodeRunner)
    r.ops = SimpleNamespace(device=cpu)
    r.cache = SimpleNamespace(length=lambda s: lengths[s], staging=Staging(cpu))
    r.pad_slot, r.buckets = 9, {}
    for n in (1, 2, 4):
        r.buckets[n] = _Bucket(n, cpu)
        r.buckets[n].warm = True
    return r


SP = [SamplingParams(0.5, 0.25), SamplingParams(), SamplingParams(1.5, 0.75)]


@pytest.mark.parametrize("form", [list, tuple, iter, lambda v: (x for x in v), lambda v: np.asarray(v, dtype=np.int64), lambda v: torch.tensor(v),
                                  lambda v: torch.tensor(v, dtype=torch.int32), lambda v: [np.int64(x) for x in v]])
def test_a_batch_is_described_from_any_sequence_of_numbers(form):
    r = _runner({3: 70, 0: 1, 5: 200})
    r.start([3, 0, 5], form([11, 12, 2**31 - 1]), form([1, 2, 3]), form([4, 5, 6]), SP)
    b = r.current
    assert b.size == bucket_size(3) and r.slots == [3, 0, 5]
    assert b.ids.tolist() == [11, 12, 2**31 - 1, 0] and b.positions.tolist() == [70, 1, 200, 0] and b.kv_len.tolist() == [71, 2, 201, 1]
    assert b.slot.tolist() == [3, 0, 5, 9] and b.live.tolist() == [1, 1, 1, 0]
    assert b.seq_key.tolist() == [1, 2, 3, 0] and b.step_key.tolist() == [4, 5, 6, 0]
    assert b.temperature.tolist() == [p.temperature for p in SP] + [0.0] and b.top_p.tolist() == [p.top_p for p in SP] + [1.0]


@pytest.mark.parametrize("form", [list, lambda v: np.asarray(v, dtype=np.int64), lambda v: torch.tensor(v)])
@pytest.mark.parametrize("which", range(3))
def test_numbers_beyond_32_bits_are_refused(form, which):
    r = _runner({3: 70, 0: 1, 5: 200})
    given = [[11, 12, 13], [1, 2, 3], [4, 5, 6]]
    given[which][1] += 2**32
    with pytest.raises((RuntimeError, OverflowError)):
        r.start([3, 0, 5], *(form(v) for v in given), SP)


@pytest.mark.parametrize("which", range(4))
def test_lists_of_another_length_than_the_batch_are_refused(which):
    for change in (lambda v: v[:-1], lambda v: v + v[:1]):
        r = _runner({3: 70, 0: 1, 5: 200})
        given = [[11, 12, 13], [1, 2, 3], [4, 5, 6], SP]
        given[which] = change(given[which])
        with pytest.raises((RuntimeError, ValueError)):
            r.start([3, 0, 5], *given)
