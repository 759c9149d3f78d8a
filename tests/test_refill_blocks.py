"""How many blocks per SM the lane-refill kernels get: the tuning's, its default where it is 0, and half of
either in groups of three and more rounds."""
import pytest

from phosphor_b200 import _capi as A


@pytest.mark.parametrize("setting", [0, 1, 2, 5, 8, 64])
@pytest.mark.parametrize("rounds", [1, 2, 3, 4, 8])
def test_blocks_per_sm(setting, rounds):
    full = setting or 8
    want = full if rounds < 3 else (full + 1) // 2
    assert A.load().phx_selftest_refill_blocks(setting, rounds) == want
