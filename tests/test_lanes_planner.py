"""Which launches run in the lane engine (cmc_plan_describe, no device): those
whose estimated time there is shorter, as measured on B200."""
import pytest


@pytest.mark.parametrize("shape,count,lanes", [
    # t = 64, N = 2^16: 18.9 against 34.1 ms at 2^20 trials, 0.9 against 0.25 at 4,000
    (("bgh25", 64, 16, 3, 96, 100, "affine"), 1 << 20, True),
    (("bgh25", 64, 16, 3, 96, 100, "affine"), 1 << 16, True),
    (("bgh25", 64, 16, 3, 96, 100, "affine"), 4000, False),
    # 64-bit domain: 0.83 against 3.3 ms
    (("bgh25", 16, 32, 3), 1 << 17, True),
    # t = 16384, N = 2^28: 338 against 402 ms
    (("bgh25", 16384, 28, 3, 24576, 1000, "affine"), 1 << 16, True),
    (("bgh25", 16384, 28, 3, 24576, 1000, "affine"), 1 << 10, False),
    # many candidates over a small PRP: the round cache is cheaper
    (("bgh25", 4096, 16, 3), 1 << 15, False),
    # tables beyond an eighth of the device's memory
    (("bgh25", 50000, 20, 3, 70000, 50, "affine"), 1 << 20, False),
])
def test_lane_engine_choice(cmc, shape, count, lanes):
    assert ("engine=lanes" in cmc.plan_describe(cmc.parameters(*shape), count)) == lanes
