"""cmc_autotune never makes the calls it tunes slower: its candidates are group
engine plans, timed on a sample of the trials, and a mix whose full calls run in
the lane or wave engine keeps those."""
import pytest

pytestmark = pytest.mark.gpu


def best_ms(ctx, jobs, calls=4):
    times = []
    for _ in range(calls):
        result = ctx.run_jobs(jobs)
        times.append(ctx.last_engine_ms())
    return min(times), result


@pytest.mark.parametrize("shapes,count", [
    ([("bgh25", 64, 16, 3, 90, 40, "affine")], 1 << 18),                       # lanes
    ([("bgh25", 1024, 20, 3, 1400, 100, "affine")], 1 << 15),                  # waves
    ([("bgh25", t, 24, k, t + t // 3 + 1, 100, "affine")                       # a sweep: several classes
      for t, k in ((20, 2), (64, 3), (200, 4), (404, 2), (700, 3), (1500, 3), (2500, 2))], 1 << 15),
    ([("bgh25", 30, 12, 3, 40, 30, "affine"), ("drrt18", 90, 12, 3, 110, 30, "affine")], 3000),  # a short call
])
def test_tuned_calls_are_not_slower(cmc, shapes, count):
    jobs = [(cmc.parameters(*s), 31 + i, 0, 0, count) for i, s in enumerate(shapes)]
    with cmc.Context(0) as ctx:
        plain, want = best_ms(ctx, jobs)
        choice = ctx.autotune(jobs, sample_div=16)
        tuned, got = best_ms(ctx, jobs)
        plan = ctx.last_plan
        assert got == want
        # run-to-run spread is about 1 %
        assert tuned <= 1.1 * plain, (plain, tuned, choice, plan)
        # the same sets with far more trials: what was tuned is not applied there
        more = [(p, s, b, f, min(1 << 19, 64 * n)) for p, s, b, f, n in jobs[:1]]
        again = ctx.autotune([(p, s, b, f, n // 64 + 1) for p, s, b, f, n in more], sample_div=4)
        tuned_more, _ = best_ms(ctx, more, 3)
        plan_more = ctx.last_plan
    with cmc.Context(0) as ctx:
        plain_more, _ = best_ms(ctx, more, 3)
        assert tuned_more <= 1.1 * plain_more, (plain_more, tuned_more, again, plan_more)
