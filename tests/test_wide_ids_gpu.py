"""The wavefront kernel's cell rule for strand ids of any size (taken by pairs
whose ids pass the fast rule, and by strand_bits = 32 at any size)."""
import numpy as np
import pytest

import oracle as O
import slcs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tm", [2, 4, 8, 12, 14, 16])
def test_wide_rule(cuda, tm):
    """Ragged shapes of one stripe and of several, alone and as tiles."""
    import torch
    rng = np.random.default_rng(tm)
    for m, n, tiles in [(1, 1, {}), (32 * tm - 1, 67, {}), (32 * tm + 1, 5, {}), (70 * tm + 3, 1030, {}),
                        (900, 1111, dict(algo=slcs.ALGO_STRIPS, strips=3, bands=2))]:
        sigma = int(rng.choice([2, 4, 256]))
        a, b = rng.integers(0, sigma, m, dtype=np.uint8), rng.integers(0, sigma, n, dtype=np.uint8)
        cfg = slcs.Config.make(tile_m=tm, strand_bits=32, **tiles)
        h, v = slcs.comb_pair(torch.from_numpy(a).to(cuda), torch.from_numpy(b).to(cuda), cfg=cfg)
        torch.cuda.synchronize()
        slcs.device_status(0)
        eh, ev = O.comb(a, b)
        np.testing.assert_array_equal(h.cpu().numpy(), eh)
        np.testing.assert_array_equal(v.cpu().numpy(), ev)
