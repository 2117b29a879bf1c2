"""Substring queries of every mixture of lengths: the device chooses between
the table and a warp per query, and either gives the formula's answers."""
import numpy as np
import pytest

import slcs

pytestmark = pytest.mark.gpu


def _answers(cuda, v, m, q):
    import torch
    qi, qj = (torch.from_numpy(np.ascontiguousarray(q[:, x], np.int32)).to(cuda) for x in (0, 1))
    got = slcs.substring_llcs(v if torch.is_tensor(v) else torch.from_numpy(v).to(cuda), m, qi, qj)
    torch.cuda.synchronize()
    slcs.device_status(0)
    return got.cpu().numpy()


def _formula(v, m, q):
    return np.array([j - i - np.count_nonzero(v[i:j] >= m + i) for i, j in q])


@pytest.mark.parametrize("n", [32768, 50001, 300007])
@pytest.mark.parametrize("nq,long_one_in", [(1, 0), (64, 0), (65, 64), (3000, 0), (3000, 1500), (3000, 100), (3000, 1)])
def test_mixed_lengths(cuda, n, nq, long_one_in):
    rng = np.random.default_rng(n + nq + long_one_in)
    m = 700
    v = rng.permutation(m + n)[:n].astype(np.int32)
    i = rng.integers(0, n - 100, nq)
    q = np.stack([i, i + rng.integers(0, 101, nq)], axis=1)
    if long_one_in:
        some = rng.integers(0, nq, max(1, nq // long_one_in))
        q[some] = np.sort(rng.integers(0, n + 1, (len(some), 2)), axis=1)
    np.testing.assert_array_equal(_answers(cuda, v, m, q), _formula(v, m, q))


def test_ids_far_below_m(cuda):
    """Ids so small that their distance from m passes 32 bits count as any id below m."""
    rng = np.random.default_rng(5)
    m, n = 1000, 40000
    v = rng.permutation(m + n)[:n].astype(np.int32)
    v[rng.integers(0, n, 9000)] = -2 ** 31
    q = np.sort(rng.integers(0, n + 1, (300, 2)), axis=1)
    np.testing.assert_array_equal(_answers(cuda, v, m, q), _formula(v, m, q))


def test_answers_over_the_queries(cuda):
    """The answers may take the place of the begins or of the ends."""
    import torch
    rng = np.random.default_rng(6)
    m, n, nq = 1000, 50001, 5000
    v = rng.permutation(m + n)[:n].astype(np.int32)
    q = np.sort(rng.integers(0, n + 1, (nq, 2)), axis=1).astype(np.int32)
    want = _formula(v, m, q)
    dv = torch.from_numpy(v).to(cuda)
    for over in (0, 1):
        cols = [torch.from_numpy(np.ascontiguousarray(q[:, x])).to(cuda) for x in (0, 1)]
        slcs.check(slcs.lib().slcs_substring_llcs(dv.data_ptr(), m, n, cols[0].data_ptr(), cols[1].data_ptr(), nq,
                                                  cols[over].data_ptr(), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        np.testing.assert_array_equal(cols[over].cpu().numpy(), want)


def test_short_windows_cost_no_pass_over_the_columns(cuda):
    """64 windows of 100 columns take about as long in 2^25 columns as in 2^15."""
    import torch

    def once(n):
        v = torch.arange(1000, 1000 + n, dtype=torch.int32, device=cuda)
        i = torch.arange(64, dtype=torch.int32, device=cuda) * (n // 64 - 100) // 2
        j = i + 100
        times = []
        for _ in range(7):
            torch.cuda.synchronize()
            t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            t0.record()
            for _ in range(10):
                slcs.substring_llcs(v, 1000, i, j)
            t1.record()
            t1.synchronize()
            times.append(t0.elapsed_time(t1))
        return sorted(times)[3]

    assert once(1 << 25) < 5 * once(1 << 15)


def test_most_columns(cuda):
    """More columns than 2^31 - 2^21: sizes of blocks and places of columns pass 31 bits on the way."""
    import torch
    m, n = 5, 2_147_400_001
    rng = np.random.default_rng(7)
    at = np.unique(rng.integers(0, n, 4000))
    at = np.unique(np.concatenate([at, [0, n - 1]]))
    ids = (m + np.unique(rng.integers(0, n, 2 * len(at)))[:len(at)]).astype(np.int32)
    ids = rng.permutation(ids)
    v = torch.zeros(n, dtype=torch.int32, device=cuda)  # h strands, but for these
    v[torch.from_numpy(at).to(cuda)] = torch.from_numpy(ids).to(cuda)
    long = np.sort(rng.integers(0, n + 1, (60, 2)), axis=1)
    long[0] = (0, n)
    short = np.stack([at[:50], np.minimum(at[:50] + 1000, n)], axis=1)
    short[-1] = (n - 40, n)
    for q in (long, short):
        want = [j - i - np.count_nonzero((at >= i) & (at < j) & (ids >= m + i)) for i, j in q]
        np.testing.assert_array_equal(_answers(cuda, v, m, q), want)
