"""int16 host runs of batches that mix what the plan treats apart: couples
(which write int16 themselves), tall pairs and 32-bit ones (narrowed one by
one), and empty sides."""
import numpy as np
import pytest

import oracle as O
import slcs
from slcs import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs", [41, 8200])  # one launch, and chunks on streams of their own
@pytest.mark.parametrize("couples", [True, False])
def test_mixed_pairs(cuda, pairs, couples):
    rng = np.random.default_rng(pairs + couples)
    ms, ns = rng.integers(1, 200, pairs), rng.integers(1, 250, pairs)
    ms[5::40], ns[5::40] = 513, 90            # too tall for couples
    ms[7::41], ns[7::41] = 1400, 700
    ms[3::37] = 0                             # empty sides
    ns[4::39] = 0
    ms[6], ns[6] = 0, 0
    ms, ns = ms.astype(np.int32), ns.astype(np.int32)
    a_off = np.concatenate([[0], np.cumsum(ms.astype(np.int64) + 1)])[:-1]  # any byte
    b_off = np.concatenate([[0], np.cumsum(ns.astype(np.int64) + 3)])[:-1]
    a = rng.integers(0, 4, int(a_off[-1]) + 2000, dtype=np.uint8)
    b = rng.integers(0, 4, int(b_off[-1]) + 2000, dtype=np.uint8)
    batch = W.Batch(a, b, a_off, b_off, ms, ns)
    off, total = batch.strand_offsets()
    cfg = slcs.Config.make(strand_bits=16 if couples else 32)
    plan = slcs.BatchPlan(slcs.pair_descs(batch), cfg)
    info = plan.info
    assert (info["packed_pairs"] > 0) == couples and info["relay_groups"] > 0 and not info["relay_all"]
    out = np.full(total, -7, np.int16)
    plan.run_host16(a, b, out)
    plan.close()
    want = O.comb_batch(a, b, a_off, b_off, ms, ns, off, total)
    np.testing.assert_array_equal(out, want)
