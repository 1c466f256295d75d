"""Throughput floors of the group engine where the automatic choice is another
engine now: half of the rates measured on B200 with lanes and waves off.  Its
walks over global slots (items with their buckets, SlotWalk in cmc_engine.cu, and
plain 32-bit slots) serve every resident server launch and every call short of
memory, and have turned 4-5x slower before after changes of the kernel's register
allocation that passed every correctness test."""
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    # name, shape, trials, measured trials/s
    ("t16384_n28", ("bgh25", 16384, 28, 3, 24576, 1000, "affine"), 1 << 15, 1.57e5),
    ("t8000_n24", ("bgh25", 8000, 24, 3, 11200, 500, "affine"), 1 << 15, 4.75e5),
    ("drrt18_t9700_n20", ("drrt18", 9700, 20, 3, 14550, 500, "affine"), 1 << 15, 6.11e5),
    ("drrt18_t20000_n24", ("drrt18", 20000, 24, 3, 30000, 500, "affine"), 1 << 13, 9.06e4),
    ("t2000_n32", ("bgh25", 2000, 32, 3, 2700, 500, "affine"), 1 << 14, 1.56e5),
]


@pytest.fixture(autouse=True)
def _group_engine(ctx):
    ctx.set_option("lanes", 0)
    ctx.set_option("waves", 0)
    yield
    ctx.set_option("lanes", -1)
    ctx.set_option("waves", -1)


@pytest.mark.parametrize("name,shape,n,measured", SHAPES, ids=[s[0] for s in SHAPES])
def test_group_engine_floor(ctx, cmc, name, shape, n, measured):
    p = cmc.parameters(*shape)
    ctx.launch(p, cmc.batch_key(5, 0), 0, n)          # warm
    ctx.launch(p, cmc.batch_key(5, 1), 0, n)
    assert "slots_in=global" in ctx.last_plan and "->" not in ctx.last_plan
    rate = n / (ctx.last_engine_ms() / 1e3)
    assert rate >= 0.5 * measured, (name, rate, ctx.last_plan)
