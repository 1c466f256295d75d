"""Wave engine (cmc_waves.cu: groups of warps build a wave's bucket maps from
round caches, then walk one trial per thread) against the oracle and the group
engine.  Outcomes are integer decisions, so the bar is equality of the failure
lists and of the probe counts."""
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [
    # mode, input, t, ell_i, k, B, kick, trials
    ("bgh25", "sequential", 16, 8, 3, 0, 0, 2000),        # golden shape, h = 5
    ("drrt18", "sequential", 16, 8, 3, 0, 0, 2000),
    ("bgh25", "affine", 3, 8, 3, 0, 0, 500),              # smallest t
    ("bgh25", "affine", 64, 16, 3, 70, 20, 3000),         # most trials fail, h = 9
    ("drrt18", "affine", 64, 16, 3, 80, 20, 3000),
    ("bgh25", "sequential", 27, 12, 2, 30, 5, 3000),      # k = 2 above its threshold, h = 7
    ("drrt18", "sequential", 5, 8, 3, 6, 5, 3000),        # fewer candidates than lanes
    ("drrt18", "affine", 200, 20, 2, 400, 30, 1000),      # h = 11
    ("bgh25", "affine", 300, 20, 4, 330, 50, 1500),       # h = 12, k = 4: copy 3 in the entry
    ("drrt18", "affine", 1500, 24, 4, 1650, 60, 200),     # h = 14, global cache
    ("bgh25", "affine", 200, 28, 4, 230, 100, 300),       # h = 16, all of the half width
    ("bgh25", "affine", 50000, 20, 3, 70000, 50, 8),      # 32-bit entries
    ("bgh25", "affine", 16384, 20, 4, 20000, 50, 8),      # t = 2^14 with k = 4
]


@pytest.fixture(autouse=True)
def _reset(ctx):
    yield
    ctx.set_option("waves", -1)
    ctx.set_option("lanes", -1)


@pytest.mark.parametrize("groups", [1, 2, 4, 8])
@pytest.mark.parametrize("shape", SHAPES)
def test_waves_vs_oracle(ctx, cmc, oracle, shape, groups):
    mode, im, t, ell, k, buckets, kick, n = shape
    p = cmc.parameters(mode, t, ell, k, buckets, kick, im)
    want = oracle.batch(oracle.params(mode, t, ell, k, buckets, kick, im), 11, 2, 5, n)
    ctx.set_option("waves", groups)
    assert ctx.launch(p, cmc.batch_key(11, 2), 5, n) == want
    assert "engine=waves" in ctx.last_plan
    probes, walks = (ctx.last_stats()[x] for x in ("probes", "walks"))
    ctx.set_option("waves", 0)
    ctx.set_option("lanes", 0)
    assert ctx.launch(p, cmc.batch_key(11, 2), 5, n) == want
    assert "engine=waves" not in ctx.last_plan
    assert walks == n and probes == ctx.last_stats()["probes"]


@pytest.mark.parametrize("shape,groups", [
    (("bgh25", "affine", 200, 16, 2, 500, 100, 100003), 8),    # several waves per group
    (("drrt18", "affine", 100, 12, 3, 120, 60, 150001), 2),
])
def test_several_waves(ctx, cmc, shape, groups):
    mode, im, t, ell, k, buckets, kick, n = shape
    p = cmc.parameters(mode, t, ell, k, buckets, kick, im)
    ctx.set_option("waves", groups)
    got = ctx.launch(p, cmc.batch_key(3, 1), 0, n)
    assert "engine=waves" in ctx.last_plan
    probes = ctx.last_stats()["probes"]
    ctx.set_option("waves", 0)
    ctx.set_option("lanes", 0)
    assert got == ctx.launch(p, cmc.batch_key(3, 1), 0, n)
    assert probes == ctx.last_stats()["probes"]


def test_waves_job_table(ctx, cmc):
    # jobs of both modes and several PRP widths in one wave
    jobs = [(cmc.parameters("bgh25", 64, 16, 3, 72, 50, "affine"), 3, 0, 7, 2000),
            (cmc.parameters("drrt18", 300, 20, 4, 330, 40, "sequential"), 4, 1, 0, 700),
            (cmc.parameters("bgh25", 1000, 12, 2, 2100, 30, "affine"), 5, 2, 3, 333),
            (cmc.parameters("drrt18", 20, 12, 2, 45, 9, "affine"), 6, 0, 0, 1)]
    ctx.set_option("lanes", 0)
    ctx.set_option("waves", 0)
    want = ctx.run_jobs(jobs)
    ctx.set_option("waves", 2)
    assert ctx.run_jobs(jobs) == want
    assert "engine=waves" in ctx.last_plan


@pytest.mark.parametrize("groups", [1, 2, 8])
@pytest.mark.parametrize("shape", [
    # round 7 filled in part: buckets that end with a high half (no cuts), and
    # not; domains of 3/4, 3/8 and nearly all of 4^h; each end of the widths
    ("bgh25", "affine", 64, 20, 3, 96, 20, 1500),          # h = 11, 512 of 2048 entries
    ("bgh25", "sequential", 64, 20, 3, 75, 30, 1500),      # h = 11, 74 cuts
    ("drrt18", "affine", 93, 18, 3, 110, 30, 1500),        # h = 10, two rows of four
    ("bgh25", "affine", 300, 19, 3, 330, 50, 600),         # h = 11, 3/8, most fail
    ("bgh25", "affine", 50, 21, 2, 113, 10, 1500),         # h = 11, one entry above 4^h / 2
    ("drrt18", "sequential", 40, 22, 4, 4096, 3, 500),     # h = 12, the whole of 4^h
    ("bgh25", "affine", 1000, 24, 3, 1100, 60, 200),       # h = 13, global cache
    ("drrt18", "affine", 150, 30, 3, 170, 60, 100),        # h = 16
])
def test_part_of_last_round(ctx, cmc, oracle, shape, groups):
    mode, im, t, ell, k, buckets, kick, n = shape
    p = cmc.parameters(mode, t, ell, k, buckets, kick, im)
    want = oracle.batch(oracle.params(mode, t, ell, k, buckets, kick, im), 5, 1, 3, n)
    ctx.set_option("waves", groups)
    assert ctx.launch(p, cmc.batch_key(5, 1), 3, n) == want
    assert "engine=waves" in ctx.last_plan
    probes = ctx.last_stats()["probes"]
    ctx.set_option("waves", 0)
    ctx.set_option("lanes", 0)
    assert ctx.launch(p, cmc.batch_key(5, 1), 3, n) == want
    assert probes == ctx.last_stats()["probes"]


@pytest.mark.parametrize("shape,groups", [
    # a round cache of h = 13 in the shared memory of a single group
    (("bgh25", "affine", 1000, 24, 3, 1100, 60, 200), 1),
    (("drrt18", "sequential", 333, 24, 2, 800, 40, 300), 1),
    (("bgh25", "affine", 2000, 22, 4, 2300, 60, 150), 1),    # h = 13, every pair cycle-walks
    (("drrt18", "affine", 17500, 24, 3, 66000, 60, 16), 1),  # with 32-bit entries
    # the same width with more groups, and the next width, in global memory
    (("bgh25", "affine", 1000, 24, 3, 1100, 60, 200), 2),
    (("bgh25", "affine", 1366, 26, 3, 1500, 60, 100), 1),
    # global caches with two and with four lookup chains per lane
    (("drrt18", "affine", 900, 26, 3, 1000, 60, 100), 2),    # h = 14
    (("bgh25", "affine", 900, 28, 3, 1000, 60, 100), 2),     # h = 15
    (("bgh25", "affine", 37, 30, 3, 43, 30, 60), 4),         # h = 16, fewer pairs than lanes
])
def test_round_cache_places(ctx, cmc, oracle, shape, groups):
    mode, im, t, ell, k, buckets, kick, n = shape
    p = cmc.parameters(mode, t, ell, k, buckets, kick, im)
    want = oracle.batch(oracle.params(mode, t, ell, k, buckets, kick, im), 7, 1, 9, n)
    ctx.set_option("waves", groups)
    assert ctx.launch(p, cmc.batch_key(7, 1), 9, n) == want
    assert "cache=" + ("smem" if p.half_bits == 13 and groups == 1 else "global") in ctx.last_plan.split("->")[-1]
    probes = ctx.last_stats()["probes"]
    ctx.set_option("waves", 0)
    ctx.set_option("lanes", 0)
    assert ctx.launch(p, cmc.batch_key(7, 1), 9, n) == want
    assert probes == ctx.last_stats()["probes"]
