"""The server's device-memory budget: what a job is counted as decides its
admission, what runs stays within the budget (with fewer walk slots, or shared
ones, where it has to), and results do not depend on it."""
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20
# beside the budget: job ring and failure bits of resident launches, 2 MB steps
# of cudaMalloc for about 20 buffers
BESIDE = 48 * MB


def free_bytes():
    import torch
    return torch.cuda.mem_get_info(0)[0]


def flat(ctx, cmc, p, seed, budget, bits):
    per = 1 << bits
    return [x for b in range(budget // per) for x in ctx.launch(p, cmc.batch_key(seed, b), 0, per)]


def serve(ctx, cmc, jobs, budget, resident, work=1 << 24):
    """Runs the jobs; returns (failures per job, most device memory used)."""
    before = free_bytes()
    srv = cmc.Server(ctx, max_jobs=16, mem_budget=budget, batch_bits=12, max_iteration_trials=1 << 14)
    srv.set_option("resident", resident)
    try:
        ids = [srv.submit(p, seed, n) for p, seed, n in jobs]
        used, steps = 0, 0
        while srv.pending():
            srv.step(work)
            used = max(used, before - free_bytes())
            steps += 1
            assert steps < 200000
        return [srv.status(i)[1] for i in ids], used
    finally:
        srv.close()


@pytest.mark.parametrize("resident", [0, 1])
def test_a_table_that_exceeds_the_budget_is_refused(ctx, cmc, resident):
    # t = 2000, N = 2^32: 673 MB of walk slots, counted for two launches in flight
    p = cmc.parameters("bgh25", 2000, 32, 3, 3000, 0, "affine")
    srv = cmc.Server(ctx, max_jobs=16, mem_budget=1 << 30, batch_bits=12, max_iteration_trials=1 << 14)
    srv.set_option("resident", resident)
    try:
        srv.submit(p, 3, 4096)
        before = free_bytes()
        with pytest.raises(cmc.CmcError) as e:
            srv.step(1 << 20)
        assert e.value.code == cmc.CMC_ENOMEM
        assert before - free_bytes() < BESIDE
    finally:
        srv.close()


@pytest.mark.parametrize("resident", [0, 1])
@pytest.mark.parametrize("budget", [1600 * MB, 24 * MB, 2 * MB])
def test_what_runs_is_within_the_budget(ctx, cmc, resident, budget):
    # tables that walk in shared memory when alone: a resident launch walks all
    # sizes in global slots, or in shared ones where not one per SM is in budget
    jobs = [(cmc.parameters("bgh25", 64, 16, 3, 72, 40, "affine"), 5, 4096),
            (cmc.parameters("drrt18", 600, 20, 3, 690, 40, "affine"), 6, 4096),
            (cmc.parameters("bgh25", 1000, 20, 2, 2200, 40, "sequential"), 7, 4096),
            (cmc.parameters("bgh25", 100, 32, 3, 115, 40, "affine"), 8, 4096)]
    if budget > 1 << 30:
        jobs.append((cmc.parameters("bgh25", 2000, 32, 3, 2300, 40, "affine"), 9, 4096))
    got, used = serve(ctx, cmc, jobs, budget, resident)
    assert used <= budget + BESIDE, (used, budget)
    for (p, seed, n), failed in zip(jobs, got):
        assert failed == len(flat(ctx, cmc, p, seed, n, 12)), (p.pnum, budget)


@pytest.mark.parametrize("resident", [0, 1])
@pytest.mark.parametrize("budget", [4 * MB, 2 * MB])
def test_small_budgets_of_one_kind(ctx, cmc, resident, budget):
    # 16-bit tables alone: fewer item slots, fewer groups, then shared slots;
    # t = 1500 walks in global slots when alone and is refused by its count
    jobs = [(cmc.parameters("bgh25", t, 16, 3, t + t // 7, 40, "affine"), t, 4096) for t in (40, 300, 900, 1500)]
    got, used = serve(ctx, cmc, jobs[:3], budget, resident)
    assert used <= budget + BESIDE
    for (p, seed, n), failed in zip(jobs, got):
        assert failed == len(flat(ctx, cmc, p, seed, n, 12)), (p.pnum, budget)
    with pytest.raises(cmc.CmcError) as e:
        serve(ctx, cmc, jobs[3:], budget, resident)
    assert e.value.code == cmc.CMC_ENOMEM
