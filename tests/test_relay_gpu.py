"""The relay kernel (slcs_comb_pair's default below its size limits) against
the CPU oracle: every shape, group and interval edges, ragged ends, bands and
strips."""
import numpy as np
import pytest

import oracle as O
import slcs

pytestmark = pytest.mark.gpu

# Sides at the edges of lanes, warps (32 * rows per lane) and groups (3 warps),
# of blocks (2 or 4 columns), intervals (16 or 32) and symbol words (128); the
# last ones reach the taller shapes and the tilings.
SHAPES = [(1, 1), (1, 131), (131, 1), (32, 32), (33, 31), (64, 127), (96, 128), (97, 129), (128, 255), (129, 16),
          (192, 257), (193, 4), (384, 1000), (385, 1001), (769, 3), (1153, 515), (300, 20001), (20001, 300),
          (9000, 2047), (116003, 2001), (120001, 33), (260001, 17), (600001, 13),
          (70001, 300), (90, 70003)]


@pytest.fixture(scope="module")
def seen():
    return set()


@pytest.mark.parametrize("m,n", SHAPES)
def test_relay_shapes(cuda, seen, m, n):
    import torch
    info = slcs.pair_plan_info(m, n)
    assert info["relay_tile_m"] > 0
    seen.add((info["relay_tile_m"], info["relay_cols"], info["relay_warps"], info["relay_strips"] > 1,
              info["relay_bands"] > 1))
    rng = np.random.default_rng(m * 7 + n)
    sigma = int(rng.choice([2, 4, 256]))
    a, b = rng.integers(0, sigma, m, dtype=np.uint8), rng.integers(0, sigma, n, dtype=np.uint8)
    eh, ev = O.comb(a, b)
    for off in (0, 3):  # b at a word and at an odd byte
        bd = torch.from_numpy(np.concatenate([np.zeros(off, np.uint8), b])).to(cuda)[off:]
        h, v = slcs.comb_pair(torch.from_numpy(a).to(cuda), bd)
        torch.cuda.synchronize()
        slcs.device_status(0)
        np.testing.assert_array_equal(h.cpu().numpy(), eh)
        np.testing.assert_array_equal(v.cpu().numpy(), ev)


def test_relay_shapes_reached(seen):
    """The sizes above reach every shape, strips and bands."""
    assert {x[:3] for x in seen} == {(1, 4, 3), (2, 4, 3), (4, 2, 3), (8, 2, 3), (8, 4, 4), (14, 4, 4), (14, 4, 8),
                                     (14, 4, 16)}
    assert any(x[3] for x in seen) and any(x[4] for x in seen)
