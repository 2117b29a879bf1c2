"""A destroyed batch plan gives its device memory back."""
import numpy as np
import pytest

import slcs

pytestmark = pytest.mark.gpu


def _plan(pairs, m, n, **cfg):
    d = np.zeros(pairs, slcs.PAIR_DTYPE)
    d["m"], d["n"] = m, n
    d["out_offset"] = np.arange(pairs, dtype=np.int64) * (m + n)
    return slcs.BatchPlan(d, slcs.Config.make(**cfg))


@pytest.mark.parametrize("pairs,m,n,cfg", [(4000, 200, 20000, dict(strand_bits=16)),  # staged couples: 320 MB
                                           (600, 9000, 100000, {})])                  # hand-down rows: 480 MB
def test_destroyed_plan_gives_memory_back(cuda, pairs, m, n, cfg):
    import torch
    _plan(64, 300, 300).close()  # one-time set-up
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    plan = _plan(pairs, m, n, **cfg)
    held = before - torch.cuda.mem_get_info()[0]
    assert held > 200 << 20
    plan.close()
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept <= 64 << 20, f"{kept >> 20} MB of {held >> 20} kept"
