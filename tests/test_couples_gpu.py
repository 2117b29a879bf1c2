"""Batch plans through the couple kernels (two pairs per register, bundles of
couples in a warp) and through the relay kernel, against the CPU oracle."""
import numpy as np
import pytest

import oracle as O
import slcs
from slcs import workloads as W

pytestmark = pytest.mark.gpu


def _pack(pairs, seed):
    """Strings at odd byte offsets (seed >= 0) or 16-byte aligned."""
    if seed < 0:
        return W.pack(pairs)
    rng = np.random.default_rng(seed)

    def blob(strings):
        off = np.zeros(len(strings), np.int64)
        pos = 0
        for i, s in enumerate(strings):
            pos += int(rng.integers(0, 4))
            off[i] = pos
            pos += len(s)
        buf = np.zeros(pos + 16, np.uint8)
        for o, s in zip(off, strings):
            buf[o:o + len(s)] = s
        return buf, off

    a, ao = blob([p[0] for p in pairs])
    b, bo = blob([p[1] for p in pairs])
    return W.Batch(a, b, ao, bo, np.array([len(p[0]) for p in pairs], np.int32),
                   np.array([len(p[1]) for p in pairs], np.int32))


def _run(batch, cfg, cuda):
    import torch
    off, total = batch.strand_offsets()
    plan = slcs.BatchPlan(slcs.pair_descs(batch), cfg)
    out = torch.full((total,), -7, dtype=torch.int32, device=cuda)
    a, b = torch.from_numpy(batch.a_blob).to(cuda), torch.from_numpy(batch.b_blob).to(cuda)
    for _ in range(2):
        out.fill_(-7)
        plan.run(a, b, out)
        torch.cuda.synchronize()
        slcs.device_status(0)
    info = plan.info
    plan.close()
    want = O.comb_batch(batch.a_blob, batch.b_blob, batch.a_off, batch.b_off, batch.ms, batch.ns, off, total)
    np.testing.assert_array_equal(out.cpu().numpy(), want)
    return info


def _pairs(seed, count, mmax, nmax):
    rng = np.random.default_rng(seed)
    pairs = []
    for i in range(count):
        m, n = int(rng.integers(1, mmax + 1)), int(rng.integers(1, nmax + 1))
        if i % 50 == 7:
            m, n = mmax, 1
        elif i % 50 == 8:
            m, n = 1, nmax
        sigma = int(rng.choice([2, 4, 256]))
        pairs.append((rng.integers(0, sigma, m, dtype=np.uint8), rng.integers(0, sigma, n, dtype=np.uint8)))
    return pairs


@pytest.mark.parametrize("count,mmax,nmax", [(1, 5, 3), (2, 512, 700), (3, 16, 16), (333, 512, 300), (500, 40, 17), (150, 30, 900),
                                             (401, 600, 90)])
@pytest.mark.parametrize("seed", [-1, 3])
def test_couples(cuda, seed, count, mmax, nmax):
    """Rows of 1 to 32 lanes, one column to several hundred, odd counts; pairs
    over 512 rows go to the relay kernel beside the couples."""
    pairs = _pairs(count, count, mmax, nmax)
    info = _run(_pack(pairs, seed), slcs.Config.make(tile_n=4), cuda)
    tall = sum(len(a) > 512 for a, _ in pairs)
    assert info["packed_pairs"] == count - tall and not info["relay_all"]
    assert (info["relay_groups"] > 0) == (tall > 0)


def test_couples_id_limit(cuda):
    """m + n = 32767 is combed in a couple, 32768 with 32-bit strands."""
    rng = np.random.default_rng(9)
    pairs = [(rng.integers(0, 4, m, dtype=np.uint8), rng.integers(0, 4, n, dtype=np.uint8))
             for m, n in [(512, 32255), (512, 32256), (1, 32766), (100, 40), (33, 32734)]]
    info = _run(_pack(pairs, 1), slcs.Config.make(tile_n=4), cuda)
    assert info["packed_pairs"] == 4 and info["stream_classes"] == 2


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("count,mmax,nmax", [(1, 300, 3000), (5, 2500, 1200), (40, 1500, 300)])
def test_relay_takes_the_plan(cuda, graph, count, mmax, nmax):
    """Few pairs without a configuration: the relay kernel combs all of them."""
    pairs = _pairs(count + 100, count, mmax, nmax)
    pairs.insert(0, (np.zeros(0, np.uint8), np.zeros(9, np.uint8)))
    info = _run(_pack(pairs, 2), slcs.Config.make(use_graph=graph), cuda)
    assert info["relay_all"] == 1 and info["relay_groups"] >= count
