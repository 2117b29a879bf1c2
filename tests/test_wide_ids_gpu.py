"""Pairs whose strand ids pass the cell rule's fast form (m + n above
0x3F800000): the plan takes the wavefront kernel's compare-and-select form."""
import numpy as np
import pytest

import oracle as O
import slcs

pytestmark = pytest.mark.gpu


def test_plan_with_wide_ids(cuda):
    """One row against 0x3F800000 + 5 columns, beside a small pair.  With one
    row the strands have a closed form: the row's strand (id 0) is swapped at
    every match and nowhere else, so column j leaves with the id of the column
    of the match before it."""
    import torch
    n = 0x3F800000 + 5
    rng = np.random.default_rng(5)
    a2, b2 = rng.integers(0, 4, 300, dtype=np.uint8), rng.integers(0, 4, 411, dtype=np.uint8)
    a = torch.from_numpy(np.concatenate([[1], a2]).astype(np.uint8)).to(cuda)
    b = torch.randint(0, 4, (n + 411,), dtype=torch.uint8, device=cuda)
    b[n:] = torch.from_numpy(b2).to(cuda)
    descs = np.zeros(2, slcs.PAIR_DTYPE)
    descs[0] = (0, 0, 0, 1, n)
    descs[1] = (1, n, n + 1, 300, 411)
    out = torch.empty(n + 1 + 711, dtype=torch.int32, device=cuda)
    plan = slcs.BatchPlan(descs)
    assert plan.info["stream_pairs"] == 0 and plan.info["wavefront_tasks"] == 3
    plan.run(a, b, out)
    torch.cuda.synchronize()
    slcs.device_status(0)
    plan.close()
    eh, ev = O.comb(a2, b2)
    np.testing.assert_array_equal(out[n + 1:].cpu().numpy(), np.concatenate([eh, ev]))
    h = 0  # the id travelling along the row
    v = out[1:n + 1]
    for c0 in range(0, n, 1 << 26):
        c1 = min(n, c0 + (1 << 26))
        want = torch.arange(c0 + 1, c1 + 1, dtype=torch.int32, device=cuda)
        at = torch.nonzero(b[c0:c1] == 1).flatten()
        if at.numel():
            ids = want[at]
            want[at[1:]] = ids[:-1]
            want[at[0]] = h
            h = int(ids[-1])
        assert torch.equal(v[c0:c1], want), c0
    assert int(out[0]) == h
