"""Substring queries answered from the table of counts (long v strands, many
queries) against the formula, at the edges of its blocks."""
import numpy as np
import pytest

import oracle as O
import slcs

pytestmark = pytest.mark.gpu


def _answers(cuda, v, m, qi, qj):
    import torch
    got = slcs.substring_llcs(*(torch.from_numpy(v).to(cuda), m), torch.from_numpy(qi).to(cuda),
                              torch.from_numpy(qj).to(cuda))
    torch.cuda.synchronize()
    slcs.device_status(0)
    return got.cpu().numpy()


@pytest.mark.parametrize("m,n,nq", [(1, 32768, 300), (5000, 32769, 300), (70000, 33023, 40), (17, 16385, 20000),
                                    (3, 262144, 200), (900, 262145, 200), (40000, 300007, 100)])
def test_table_queries(cuda, m, n, nq):
    """Strands as a comb leaves them: distinct ids below m + n in any order."""
    rng = np.random.default_rng(n)
    v = rng.permutation(m + n)[:n].astype(np.int32)
    q = np.sort(rng.integers(0, n + 1, (nq, 2)), axis=1).astype(np.int32)
    near = rng.integers(0, n // 256, nq // 4) * 256  # block edges, and one column beside them
    q[:len(near), 0] = np.minimum(near + rng.integers(-1, 2, len(near)).clip(0), n)
    q[:len(near), 1] = np.minimum(q[:len(near), 0] + 256 * rng.integers(0, 9, len(near)), n)
    q[-1] = (0, n)
    q[-2] = (n, n)
    qi, qj = np.ascontiguousarray(q[:, 0]), np.ascontiguousarray(q[:, 1])
    np.testing.assert_array_equal(_answers(cuda, v, m, qi, qj), O.substring_llcs(v, m, qi, qj))


def test_table_not_strands(cuda):
    """Arrays that no comb leaves (equal ids, ids past m + n) are counted as they are."""
    rng = np.random.default_rng(3)
    m, n = 100, 40000
    v = rng.integers(0, m + n + 5000, n).astype(np.int32)
    q = np.sort(rng.integers(0, n + 1, (50, 2)), axis=1).astype(np.int32)
    want = [int(j - i - np.sum(v[i:j] >= m + i)) for i, j in q]
    got = _answers(cuda, v, m, np.ascontiguousarray(q[:, 0]), np.ascontiguousarray(q[:, 1]))
    np.testing.assert_array_equal(got, want)
