"""Planner at table sizes whose byte counts pass 32 bits (cmc_plan_describe, no
device): such a table is refused, or planned with its whole size, never with a
wrapped one."""
import pytest


@pytest.mark.parametrize("buckets", [
    (1 << 28) - 1, 1 << 28, (1 << 28) + 4096,                   # 16-byte entries pass 2^32
    (1 << 30) - 80000, 1 << 30, (1 << 30) + 1, (1 << 32) - 1,   # 4-byte ones
])
@pytest.mark.parametrize("t,ell", [(3000, 20), (30000, 20), (65534, 28)])
@pytest.mark.parametrize("sms", [148, 2])
def test_table_bytes_do_not_wrap(cmc, t, ell, buckets, sms):
    p = cmc.parameters("bgh25", t, ell, 3, buckets, 50, "affine")
    try:
        text = cmc.plan_describe(p, 1 << 10, sms=sms)
    except cmc.CmcError as e:
        assert e.code == cmc.CMC_EINVAL and (buckets + 3 * t) * 4 > (1 << 32) - 256
        return
    assert (buckets + 3 * t) * 4 <= (1 << 32) - 256
    assert "slots_in=global" in text
    if "region=" in text:
        assert int(text.split("region=")[1].split()[0]) >= buckets * 16
