"""Steady-ant nodes one block finishes: node sizes on either side of each warp
count (320 entries one warp; 300, 600, 900, 1200 the warps of 30 lanes) and
one entry over the largest, random permutations and the extremes (no crossing,
every crossing), exactly against the reference multiplication.
"""
import numpy as np
import pytest

import oracle as O
import slcs

pytestmark = pytest.mark.gpu


def _check(P, Q, k, cutoff):
    import torch
    want, _ = O.staggered_multiply(P, Q, k, False)
    dev = lambda x: torch.from_numpy(np.ascontiguousarray(x, np.int32)).cuda()
    cfg = slcs.Config.make(braid_cutoff=cutoff) if cutoff else None
    got = slcs.braid_multiply(dev(P), dev(Q), k, False, cfg=cfg)
    torch.cuda.synchronize()
    slcs.device_status(0)
    np.testing.assert_array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("k", [1, 2, 3, 9, 10, 11, 319, 320, 321, 599, 600, 601, 900, 901, 1199, 1200, 1201, 2400])
def test_node_sizes(cuda, k):
    rng = np.random.default_rng(k)
    ident, rev = np.arange(k), np.arange(k)[::-1]
    for P, Q in [(rng.permutation(k), rng.permutation(k)), (rev, rng.permutation(k)), (rng.permutation(k), rev),
                 (ident, rng.permutation(k)), (rev, rev)]:
        _check(P, Q, k, None)


@pytest.mark.parametrize("cutoff", [1, 3, 320, 330, 1200, 1 << 20])
def test_cutoffs(cuda, cutoff):
    rng = np.random.default_rng(cutoff)
    _check(rng.permutation(5003), rng.permutation(4999), 4801, cutoff)


@pytest.mark.parametrize("k,cutoff", [(1023, 8), (1024, 8), (1025, 9), (1025, 8), (2049, 1024), (4801, 38), (4801, 37),
                                      (153600, 1200), (153601, 1200), (4801, 19), (4801, 18),
                                      (307200, 1200), (307201, 1200)])
def test_partitions(cuda, k, cutoff):
    """Every level in one pass up to 256 nodes (one entry more: level by level), around its tiles of 1024."""
    rng = np.random.default_rng(k)
    _check(rng.permutation(k + 3), rng.permutation(k + 2500), k, cutoff)


def test_many_slice_blocks(cuda):
    """More blocks of the slices than add their predecessors' counts themselves."""
    rng = np.random.default_rng(3)
    _check(rng.permutation(2200000), rng.permutation(300), 57, None)
    _check(rng.permutation(300), rng.permutation(2200000), 57, None)
