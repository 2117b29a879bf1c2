"""strand_bits = 16 or 32 is a batch setting: it leaves the plan of a single
pair as it is (64 asks for the wide cell rule, which the relay kernel lacks)."""
import pytest

import slcs


@pytest.mark.parametrize("m,n", [(152, 187), (4096, 4096), (20011, 9973), (1003, 250007), (131072, 131072)])
def test_single_pairs_ignore_the_batch_setting(m, n):
    want = slcs.pair_plan_info(m, n, sms=148)
    assert want["relay_tile_m"] > 0
    for bits in (16, 32):
        assert slcs.pair_plan_info(m, n, slcs.Config.make(strand_bits=bits), sms=148) == want
    assert slcs.pair_plan_info(m, n, slcs.Config.make(strand_bits=64), sms=148)["relay_tile_m"] == 0
