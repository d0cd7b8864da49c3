"""How the decode attention's pages are shared out: decisions made on the host, on the CPU."""
from types import SimpleNamespace

import pytest
import torch

from cpmcu_b200.ops.ops import Ops


@pytest.mark.parametrize("d", [32, 64, 96, 128])
def test_counters_are_given_only_for_shares_that_the_last_block_can_add_up(d):
    """At head size 32 a sequence has as many shares as the caller asks for, and the block that adds them up has room for 32."""
    ops = SimpleNamespace(workspace=object(), arrivals=torch.zeros(16384, dtype=torch.int32))
    for n_splits in (2, 16, 32, 33, 64, 1000):
        got = Ops._arrivals(ops, 2, 16, 2, d, n_splits)
        assert (got is not None) == (d == 64 or (d == 32 and n_splits <= 32)), n_splits
