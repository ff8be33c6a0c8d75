"""CPU: how a decode step is laid out on the 148 SMs, over all step sizes of one to three waves."""
import ctypes

import pytest


def _plan(lib, batch, heads_k):
    plan = (ctypes.c_int32 * 2)()
    assert lib.ifv2_decode_plan(batch, heads_k, plan) == 0
    return plan[0], plan[1]


@pytest.mark.parametrize("heads_k", [1, 2, 8])
def test_decode_step_needs_no_more_waves_than_it_has_to(lib, heads_k):
    for batch in range(1, 1400 // heads_k):
        pairs = batch * heads_k
        splits, resident = _plan(lib, batch, heads_k)
        # the split decides how the weights are rounded: it is a function of the number of pairs alone
        assert splits == min(max(148 * 3 // pairs, 1), 16)
        waves = [-(-pairs * splits // (148 * n)) for n in (2, 3)]
        assert resident == (2 if waves[0] == waves[1] else 3), (pairs, splits, resident)


@pytest.mark.parametrize("batch,heads_k", [(0, 2), (2, 0), (-1, 1)])
def test_decode_plan_refuses_empty_steps(lib, batch, heads_k):
    assert lib.ifv2_decode_plan(batch, heads_k, (ctypes.c_int32 * 2)()) == -1
