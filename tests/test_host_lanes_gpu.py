"""Host-pointer calls on their kept streams and page-locked buffers: several
threads at once, sizes on both sides of the buffer, and refusals in between."""
import threading

import numpy as np
import pytest

import oracle as O
import slcs

pytestmark = pytest.mark.gpu


def _call(seed, m, n, words, errors):
    try:
        rng = np.random.default_rng(seed)
        a, b = rng.integers(0, 200, m, dtype=np.uint8), rng.integers(0, 200, n, dtype=np.uint8)
        if words:
            h, v = slcs.comb_pair_words_host(a.astype(np.int32) * 1000 - 7, b.astype(np.int32) * 1000 - 7)
        else:
            h, v = slcs.comb_pair_host(a, b)
        eh, ev = O.comb(a, b) if m and n else (np.arange(m), np.arange(m, m + n))
        np.testing.assert_array_equal(h, eh)
        np.testing.assert_array_equal(v, ev)
    except Exception as e:  # reported by the test's thread
        errors.append((seed, m, n, words, e))


@pytest.mark.parametrize("words", [False, True])
def test_threads_and_sizes(cuda, words):
    errors = []
    sizes = [(1, 1), (0, 9), (9, 0), (300, 500), (1000, 3), (20, 300000), (3, 600000), (700, 800)]
    for _ in range(2):
        threads = [threading.Thread(target=_call, args=(i, m, n, words, errors)) for i, (m, n) in enumerate(sizes)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        too_many = np.arange(300, dtype=np.int32)
        with pytest.raises(slcs.SlcsError) as err:
            slcs.comb_pair_words_host(too_many, too_many[:5])
        assert err.value.status == 6
    assert not errors, errors[0]
