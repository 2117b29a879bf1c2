"""Making a batch plan takes time in proportion to its pairs, also where no two
couples fit into one warp."""
import time

import numpy as np
import pytest

import slcs

pytestmark = pytest.mark.gpu


def _seconds(pairs):
    rng = np.random.default_rng(pairs)
    d = np.zeros(pairs, slcs.PAIR_DTYPE)
    d["m"], d["n"] = rng.integers(290, 310, pairs), rng.integers(300, 376, pairs)
    d["m"][0] = 200  # some pair short enough for the packed plan
    d["out_offset"] = np.concatenate([[0], np.cumsum(d["m"].astype(np.int64) + d["n"])[:-1]])
    times = []
    for _ in range(3):
        t0 = time.perf_counter()
        plan = slcs.BatchPlan(d)
        times.append(time.perf_counter() - t0)
        assert plan.info["packed_pairs"] == pairs
        plan.close()
    return min(times)


def test_time_follows_the_pairs(cuda):
    _seconds(100)
    assert _seconds(120000) < 15 * _seconds(15000)  # 8 times as many pairs
