"""Batches whose item lists are more rounds of the grid than blocks have turns of their own: every
item by the counter -- against the members stepped one by one."""
import pytest

from spacetime_gb300 import capi
from spacetime_gb300.batch import Batch
from test_batch import _close, _compare, _member
from test_batch_turns import SPECS

pytestmark = pytest.mark.gpu


# one row per item at 1 block per SM on 152 SMs: 2280 rows are 15 rounds, 2480 16, 2600 17, 3880 25
@pytest.mark.parametrize("more", [[], [("bcc", 1, (3, 20, 10))], [("bcc", 1, (3, 20, 16))], [("bcc", 1, (5, 40, 40))]])
@pytest.mark.parametrize("steps", [2, 11])
def test_long_lists(gpu, more, steps):
    mem = [_member(s, capi.FP32, i) for i, s in enumerate(SPECS + more)]
    ref = [_member(s, capi.FP32, i) for i, s in enumerate(SPECS + more)]
    try:
        with Batch(mem) as b:
            b.set_tuning(capi.BATCH_BLOCKS_PER_SM, 1)
            b.set_tuning(capi.BATCH_ITEM_NODES, 1)
            b.step(steps)
        for r in ref:
            r.step(steps)
        _compare(mem, ref, capi.FP32)
    finally:
        _close(mem + ref)
