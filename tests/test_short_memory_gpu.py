"""Calls that need little themselves still run where the memory for their
faster form is not to be had."""
import gc

import numpy as np
import pytest

import oracle as O
import slcs

pytestmark = pytest.mark.gpu


@pytest.fixture
def little(cuda):
    """All device memory but about a gigabyte is taken."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    taken = [torch.empty(free - (1 << 30), dtype=torch.uint8, device=cuda)]
    yield
    taken.clear()
    gc.collect()
    torch.cuda.empty_cache()


def test_batch_without_room_for_staged_couples(cuda, little):
    """40,000 times one pair whose couples would take 3.2 GB of staging."""
    import torch
    rng = np.random.default_rng(1)
    m, n = 200, 20000
    a, b = rng.integers(0, 4, m, dtype=np.uint8), rng.integers(0, 4, n, dtype=np.uint8)
    d = np.zeros(40000, slcs.PAIR_DTYPE)
    d["m"], d["n"] = m, n
    d["out_offset"] = np.arange(len(d)) % 3 * (m + n)
    plan = slcs.BatchPlan(d, slcs.Config.make(strand_bits=16))
    out = torch.empty(3 * (m + n), dtype=torch.int32, device=cuda)
    plan.run(torch.from_numpy(a).to(cuda), torch.from_numpy(b).to(cuda), out)
    torch.cuda.synchronize()
    slcs.device_status(0)
    plan.close()
    want = np.concatenate(O.comb(a, b))
    for x in out.cpu().numpy().reshape(3, -1):
        np.testing.assert_array_equal(x, want)


def test_queries_without_room_for_the_table(cuda, little):
    import torch
    m, n = 5, 200_000_000
    v = torch.zeros(n, dtype=torch.int32, device=cuda)  # 0.8 GB of h strands
    v[1000::1000] = torch.arange(m, m + len(range(1000, n, 1000)), dtype=torch.int32, device=cuda)
    q = np.array([[0, 3_000_000], [999, 1000], [500, 2_500_001], [7, n - 190_000_000]], np.int64)
    got = slcs.substring_llcs(v, m, *(torch.from_numpy(q[:, x].astype(np.int32)).to(cuda) for x in (0, 1)))
    torch.cuda.synchronize()
    slcs.device_status(0)
    at = np.arange(1000, n, 1000)
    ids = m + np.arange(len(at))
    want = [j - i - np.count_nonzero((at >= i) & (at < j) & (ids >= m + i)) for i, j in q]
    np.testing.assert_array_equal(got.cpu().numpy(), want)
