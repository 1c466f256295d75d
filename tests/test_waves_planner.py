"""Which launches run in the wave engine (cmc_plan_describe, no device): those
whose estimated time there is shorter, as measured on B200."""
import pytest


@pytest.mark.parametrize("shape,count,waves", [
    # t = 1024, N = 2^20: 245 against 299 ms at 2^20 trials
    (("bgh25", 1024, 20, 3, 1536, 500, "affine"), 1 << 20, True),
    # t = 4096, N = 2^16: long walks over a small PRP, 17 against 32 ms
    (("bgh25", 4096, 16, 3), 1 << 15, True),
    # round caches in global memory (h = 14): 47 against 54 ms
    (("drrt18", 1500, 24, 4, 1875, 500, "affine"), 20011, True),
    # 64-bit domains have no round cache; direct evaluation is cheaper at t = 64
    (("bgh25", 16, 32, 3), 1 << 17, False),
    (("bgh25", 64, 16, 3, 96, 100, "affine"), 1 << 20, False),
    # a few trials
    (("bgh25", 1024, 20, 3, 1536, 500, "affine"), 200, False),
])
def test_wave_engine_choice(cmc, shape, count, waves):
    assert ("engine=waves" in cmc.plan_describe(cmc.parameters(*shape), count)) == waves
