"""A pair's comb recorded into a CUDA graph: replays comb what the input
buffers hold then, and need nothing of the call that was recorded."""
import numpy as np
import pytest

import oracle as O
import slcs

pytestmark = pytest.mark.gpu

TILES = dict(algo=slcs.ALGO_STRIPS, strips=3, bands=2, tile_m=4)


@pytest.mark.parametrize("m,n,conf", [(152, 187, {}), (3000, 2000, {}), (20000, 1000, {}), (500, 60000, {}),
                                      (3000, 3001, TILES)])
def test_pair_replays(cuda, m, n, conf):
    import torch
    cfg = slcs.Config.make(**conf) if conf else None
    rng = np.random.default_rng(m + n)

    def strings():
        return rng.integers(0, 4, m, dtype=np.uint8), rng.integers(0, 4, n, dtype=np.uint8)

    a, b = (torch.from_numpy(x).to(cuda) for x in strings())
    out = torch.empty(m + n, dtype=torch.int32, device=cuda)
    slcs.comb_pair(a, b, cfg=cfg, out=out)  # one-time set-up before the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        slcs.comb_pair(a, b, cfg=cfg, out=out)
    junk = [np.full(k, 0x77, np.uint8) for k in range(64, 1 << 16, 64)]  # over whatever host memory the call gave back
    for _ in range(2):
        x, y = strings()
        a.copy_(torch.from_numpy(x))
        b.copy_(torch.from_numpy(y))
        out.fill_(-1)
        graph.replay()
        torch.cuda.synchronize()
        slcs.device_status(0)
        eh, ev = O.comb(x, y)
        got = out.cpu().numpy()
        np.testing.assert_array_equal(got[:m], eh)
        np.testing.assert_array_equal(got[m:], ev)
    assert len(junk) > 0


def test_tiled_plans_are_reached(cuda):
    assert slcs.pair_plan_info(20000, 1000)["relay_bands"] > 1
    assert slcs.pair_plan_info(500, 60000)["relay_strips"] > 1
