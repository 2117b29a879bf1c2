"""The wavefront kernel's cell rule for strand ids of any size (strand_bits = 64
asks for it at any size) in every form of launch: each number of warps per
block, 4 and 8 columns per step, all stripes resident and more than that."""
import numpy as np
import pytest

import oracle as O
import slcs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tm,warps", [(2, 2), (4, 4), (8, 8), (12, 2), (14, 8), (16, 4)])
def test_forms(cuda, tm, warps):
    import torch
    rng = np.random.default_rng(tm * 10 + warps)
    shapes = [(32 * tm + 3, 4101),          # two stripes and many columns: 8 per step where a lane has 14 or 16 rows
              (40 * 32 * tm - 5, 131)]
    if tm == 2:
        shapes.append((2500 * 64 + 1, 37))  # more stripes than 16 warps of 148 SMs take at once
    for m, n in shapes:
        a, b = rng.integers(0, 3, m, dtype=np.uint8), rng.integers(0, 3, n, dtype=np.uint8)
        cfg = slcs.Config.make(algo=slcs.ALGO_WAVEFRONT, tile_m=tm, warps=warps, strand_bits=64)
        h, v = slcs.comb_pair(torch.from_numpy(a).to(cuda), torch.from_numpy(b).to(cuda), cfg=cfg)
        torch.cuda.synchronize()
        slcs.device_status(0)
        eh, ev = O.comb(a, b)
        np.testing.assert_array_equal(h.cpu().numpy(), eh)
        np.testing.assert_array_equal(v.cpu().numpy(), ev)
