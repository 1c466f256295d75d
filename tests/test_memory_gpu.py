"""Calls short of device memory: with "pool_bytes" a context plans within a
limit, as it does when cudaMalloc fails -- the group engine, then fewer walk
slots -- and every result stays that of the unlimited call."""
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


@pytest.fixture(autouse=True)
def _reset(ctx):
    yield
    ctx.set_option("pool_bytes", 0)


@pytest.mark.parametrize("shape,n,limits", [
    (("bgh25", 64, 16, 3, 96, 100, "affine"), 1 << 17, [8 * MB, MB]),               # lanes, else no pool
    (("bgh25", 1024, 20, 3, 1250, 60, "affine"), 1 << 15, [200 * MB, 8 * MB]),      # waves
    (("bgh25", 3000, 24, 3, 3450, 60, "affine"), 4000, [1200 * MB, 100 * MB, 60 * MB, 48 * MB]),  # items, h = 13
    (("drrt18", 16384, 16, 3, 19000, 40, "affine"), 300, [400 * MB, 60 * MB]),
    (("bgh25", 16384, 28, 3, 19000, 40, "affine"), 300, [700 * MB, 200 * MB]),      # round caches of h = 16
    (("bgh25", 50000, 20, 3, 57000, 40, "affine"), 40, [900 * MB, 200 * MB]),       # 32-bit slots
    (("bgh25", 2000, 32, 3, 2300, 40, "affine"), 600, [300 * MB, 20 * MB]),         # 64-bit domain
])
def test_launch_within_a_limit(ctx, cmc, shape, n, limits):
    p = cmc.parameters(*shape)
    want = ctx.launch(p, cmc.batch_key(3, 1), 7, n)
    probes = ctx.last_stats()["probes"]
    assert want
    for limit in limits:
        ctx.set_option("pool_bytes", limit)
        for _ in range(2):
            assert ctx.launch(p, cmc.batch_key(3, 1), 7, n) == want, (limit, ctx.last_plan)
            assert ctx.last_stats()["probes"] == probes
    ctx.set_option("pool_bytes", 0)
    assert ctx.launch(p, cmc.batch_key(3, 1), 7, n) == want


def test_equal_batched_calls_within_a_limit(ctx, cmc):
    # the second call is captured, which allows no allocation, the third replays
    jobs = [(cmc.parameters("bgh25", 64, 16, 3, 70, 20, "affine"), 3, 0, 7, 50000),
            (cmc.parameters("drrt18", 700, 20, 3, 800, 40, "affine"), 4, 1, 0, 20000),
            (cmc.parameters("bgh25", 3000, 24, 3, 3450, 60, "affine"), 5, 2, 3, 3000)]
    want = ctx.run_jobs(jobs)
    assert "-> engine" in ctx.last_plan
    ctx.set_option("pool_bytes", 100 * MB)
    states = []
    for _ in range(4):
        assert ctx.run_jobs(jobs) == want
        assert "-> engine" not in ctx.last_plan
        states.append(ctx.last_plan.rsplit("graph=", 1)[-1])
    assert states == ["eager", "captured", "replayed", "replayed"], states
    ctx.set_option("pool_bytes", 0)
    assert ctx.run_jobs(jobs) == want
    assert "-> engine" in ctx.last_plan


def test_a_limit_that_fits_nothing_is_refused(ctx, cmc):
    p = cmc.parameters("bgh25", 16384, 28, 3, 19000, 40, "affine")
    want = ctx.launch(p, cmc.batch_key(3, 1), 0, 200)
    ctx.set_option("pool_bytes", MB)
    with pytest.raises(cmc.CmcError) as e:
        ctx.launch(p, cmc.batch_key(3, 1), 0, 200)
    assert e.value.code == cmc.CMC_ENOMEM
    ctx.set_option("pool_bytes", 0)
    assert ctx.launch(p, cmc.batch_key(3, 1), 0, 200) == want


@pytest.mark.parametrize("pool", ["none yet", "allocated"])
def test_capture_of_a_device_launch_ends_well(cmc, pool):
    # on a stream that the caller captures nothing is allocated, and the launch
    # takes no tables that a later call could replace (the graph is not replayed)
    import torch
    p = cmc.parameters("bgh25", 64, 16, 3, 90, 40, "affine")
    n = 1 << 17
    key = torch.tensor(cmc.batch_key(3, 1), dtype=torch.int64).to(torch.int32).cuda()
    offsets = torch.zeros(n, dtype=torch.int32, device="cuda")
    nfailed = torch.zeros(1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    with cmc.Context(0) as ctx:
        def launch():
            ctx.launch_device(p, key.data_ptr(), 0, n, offsets.data_ptr(), nfailed.data_ptr(), stream.cuda_stream)

        if pool == "none yet":  # the other buffers are sized by a call in the group engine
            ctx.set_option("lanes", 0)
            ctx.set_option("waves", 0)
        launch()
        stream.synchronize()
        ctx.check()
        want = nfailed.item(), offsets[:nfailed.item()].tolist()
        ctx.set_option("lanes", -1)
        ctx.set_option("waves", -1)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            launch()
        assert "-> engine" not in ctx.last_plan
        del graph
        launch()
        stream.synchronize()
        ctx.check()
        assert "-> engine" in ctx.last_plan
        assert (nfailed.item(), offsets[:nfailed.item()].tolist()) == want
