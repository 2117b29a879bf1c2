"""The relay kernel with two pairs per register (batches whose ids fit 15 bits):
every shape, against the same batch with 32-bit strands, and its smallest
pairs against the CPU oracle.  Pairs of unequal sizes share registers, the
last one of an odd count has its own, strings start at any byte."""
import numpy as np
import pytest

import oracle as O
import slcs
from slcs import workloads as W

pytestmark = pytest.mark.gpu


def _batch(count, m, n, jitter, seed, align):
    rng = np.random.default_rng(seed)
    ms = m - rng.integers(0, jitter + 1, count)
    ns = n - rng.integers(0, jitter + 1, count)
    pairs = [(rng.integers(0, 4, x, dtype=np.uint8), rng.integers(0, 4, y, dtype=np.uint8)) for x, y in zip(ms, ns)]
    if align:
        return pairs, W.pack(pairs)
    ao = np.concatenate([[1], 1 + np.cumsum(ms + 1)[:-1]])
    bo = np.concatenate([[3], 3 + np.cumsum(ns + 2)[:-1]])
    a = np.zeros(int(ao[-1] + ms[-1] + 16), np.uint8)
    b = np.zeros(int(bo[-1] + ns[-1] + 16), np.uint8)
    for (x, y), i, j in zip(pairs, ao, bo):
        a[i:i + len(x)] = x
        b[j:j + len(y)] = y
    return pairs, W.Batch(a, b, ao.astype(np.int64), bo.astype(np.int64), ms.astype(np.int32), ns.astype(np.int32))


def _run(batch, cfg=None):
    import torch
    off, total = batch.strand_offsets()
    plan = slcs.BatchPlan(slcs.pair_descs(batch), cfg)
    out = torch.full((total,), -7, dtype=torch.int32, device="cuda")
    plan.run(torch.from_numpy(batch.a_blob).cuda(), torch.from_numpy(batch.b_blob).cuda(), out)
    torch.cuda.synchronize()
    slcs.device_status(0)
    return out.cpu().numpy(), off, plan.info


# (count, rows, columns, jitter): 2 x 4, 4 x 4, 8 x 2 and 8 x 4 rows by columns
# a lane and step; the longest ids that fit; pairs of a few rows.
@pytest.mark.parametrize("count,m,n,jitter", [(65, 400, 5000, 30), (255, 600, 500, 90), (99, 3000, 3000, 700),
                                              (31, 9000, 4000, 500), (41, 2000, 30767, 0), (501, 300, 2000, 290)])
@pytest.mark.parametrize("align", [True, False])
def test_duos(cuda, count, m, n, jitter, align):
    pairs, batch = _batch(count, m, n, jitter, count, align)
    got, off, info = _run(batch)
    want, _, wide = _run(batch, slcs.Config.make(strand_bits=32))
    assert info["relay_all"] and info["relay_duos"] == (count + 1) // 2 and wide["relay_duos"] == 0
    np.testing.assert_array_equal(got, want)
    p = int(np.argmin([len(x) * len(y) for x, y in pairs]))
    one = W.pack([pairs[p]])
    first, total = one.strand_offsets()
    strands = O.comb_batch(one.a_blob, one.b_blob, one.a_off, one.b_off, one.ms, one.ns, first, total)
    np.testing.assert_array_equal(got[off[p]:off[p] + total], strands[first[0]:first[0] + total])


def test_one_id_too_many_keeps_32_bits(cuda):
    pairs, batch = _batch(41, 2000, 30768, 0, 5, True)
    got, off, info = _run(batch)
    assert info["relay_groups"] >= 41 and info["relay_duos"] == 0
    np.testing.assert_array_equal(got, _run(batch, slcs.Config.make(strand_bits=32))[0])
