"""How a batch hands its work out: each block's own turns of a step, then the counter's, and
the layout a call's length picks -- against the members stepped one by one."""
import pytest

from spacetime_gb300 import capi
from spacetime_gb300.batch import Batch
from test_batch import _close, _compare, _member

pytestmark = pytest.mark.gpu

SPECS = [("bcc", 3, (9, 30, 31)), ("c15", 1, (3, 20, 21)), ("fcc", 3, (7, 29, 17)), ("bcc", 1, (5, 23, 19))]


# one row per item at 1 block per SM is some 15 turns of a block on 152 SMs; larger items leave
# two turns (one of its own), one and none
@pytest.mark.parametrize("item_nodes", [1, 900, 2500, 1 << 20])
@pytest.mark.parametrize("steps", [1, 10, 11])
def test_turns_and_call_lengths(gpu, item_nodes, steps):
    mem = [_member(s, capi.FP32, i) for i, s in enumerate(SPECS)]
    ref = [_member(s, capi.FP32, i) for i, s in enumerate(SPECS)]
    try:
        with Batch(mem) as b:
            b.set_tuning(capi.BATCH_BLOCKS_PER_SM, 1)
            b.set_tuning(capi.BATCH_ITEM_NODES, item_nodes)
            b.step(steps)
            n_il = 2 if steps >= 11 else 0  # the spin-1 members on BCC and FCC
            assert b.launches == 1 + 4 * n_il
        for r in ref:
            r.step(steps)
        _compare(mem, ref, capi.FP32)
    finally:
        _close(mem + ref)


def test_layout_once_set_holds_for_short_calls(gpu):
    mem = [_member(s, capi.FP32, i) for i, s in enumerate(SPECS)]
    try:
        with Batch(mem) as b:
            assert b.get_tuning(capi.BATCH_LAYOUT) == 1
            b.step(2)
            assert b.launches == 1
            b.set_tuning(capi.BATCH_LAYOUT, 1)
            b.step(2)
            assert b.launches == 2 + 4 * 2
    finally:
        _close(mem)
