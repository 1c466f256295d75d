"""Performance cases of the cuckoo-hashing Monte Carlo estimator.

Each case is work that a program does with this library through its public
entry points: the Launch seam with host buffers (Context.launch), its
device-pointer forms (Context.launch_device, launch_static), the batched call
(Context.run_jobs) and the serving loop (Server).  Shapes are those of the
benchmark workloads, of the tests and of the command line's defaults.

A launch evaluates `count` trials of one batch: a trial places t items, k
copies each, into B buckets; the output is the list of failing trials.  The
`launch` cases also return the walks' probe count (Context.last_stats), a whole
number that depends on every trial of the launch.
"""
import importlib.util
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
PACKAGE = ROOT / "pbc-based-dmpf-monte-carlo-test_b200"


def package():
    """This repository's package (its folder's name is not an identifier)."""
    if "cmc_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("cmc_b200", PACKAGE / "__init__.py")
        mod = importlib.util.module_from_spec(spec)
        sys.modules["cmc_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["cmc_b200"]


_context = None


def context():
    """One context per process and device, as a user's program keeps it."""
    global _context
    if _context is None:
        _context = package().Context(0)
    return _context


def shape(mode, inputs, t, ell, k, buckets=0, kick=0):
    """buckets or kick 0: derived from t as the command line derives them."""
    return dict(mode=mode, inputs=inputs, t=t, ell=ell, k=k, buckets=buckets, kick=kick)


def listed():
    return [
        # The smallest call in use: one micro-launch of the golden run, t = 16
        # items, 2^8 keys, 256 trials.  Launch latency decides.
        dict(name="golden_micro_t16", call="launch", count=256, **shape("bgh25", "sequential", 16, 8, 3)),
        # The benchmark's first workload: one batch of 2^16 trials, t = 64.
        dict(name="batch_t64", call="launch", count=1 << 16, **shape("bgh25", "affine", 64, 16, 3, 96, 100)),
        # The command line's defaults (t = 16, N = 2^32 keys: a PRP domain above
        # 2^32) at its default micro-launch of 2^17 trials.
        dict(name="cli_default_n32", call="launch", count=1 << 17, **shape("bgh25", "sequential", 16, 32, 3)),
        # The other eviction rule, with the B it derives; odd sizes throughout.
        dict(name="drrt18_t93", call="launch", count=100003, **shape("drrt18", "sequential", 93, 20, 3)),
        # A small device-resident micro-launch of an odd size: a host that keeps
        # keys and results on the device and queues launches on its own stream.
        dict(name="device_t300_k4", call="device", count=3001, **shape("bgh25", "affine", 300, 20, 4, 330, 50)),
        # The form without device allocation, in the middle of its range.
        dict(name="static_t200_k2", call="static", count=20000, **shape("bgh25", "affine", 200, 16, 2, 500, 100)),
        # The benchmark's default workload: one batch of 2^20 trials, t = 1024.
        dict(name="batch_t1024", call="launch", count=1 << 20, **shape("bgh25", "affine", 1024, 20, 3, 1536, 500)),
        # The size of the reference's published CPU figure: t = 4096, N = 2^16.
        # Few keys for many items: long walks over a small PRP.
        dict(name="published_t4096_n16", call="launch", count=1 << 15, **shape("bgh25", "sequential", 4096, 16, 3)),
        # A mid-size table with many keys, four copies, DRRT18 and tight load.
        dict(name="drrt18_t1500_n24_k4", call="launch", count=20011,
             **shape("drrt18", "affine", 1500, 24, 4, 1875, 500)),
        # The benchmark's large-table workload: t = 16384, N = 2^28, one step of
        # 2^16 trials.  The largest case.
        dict(name="table_t16384_n28", call="launch", count=1 << 16,
             **shape("bgh25", "affine", 16384, 28, 3, 24576, 1000)),
        # The benchmark's sweep of parameter sets (t = 16..4096, k = 2, 3, 4,
        # N = 2^24) in one batched call, fewer sets and trials.
        dict(name="sweep_24_sets", call="jobs", sets=24, draw=3, count=4096),
        # The benchmark's served stream (t = 2^4..2^14, k = 2, 3, N = 2^24),
        # jobs submitted together and stepped until all have finished.
        dict(name="serve_16_jobs", call="serve", sets=16, draw=5, low=9, high=13),
    ]


def geometry(c):
    """(half width h, cycle-walking factor, domain above 2^32) of a shape."""
    keys = c["k"] << c["ell"]
    buckets = c["buckets"] or math.ceil(1.5 * c["t"])
    domain = buckets * -(-keys // buckets)
    h = max(1, -(-(domain - 1).bit_length() // 2))
    return h, 2.0 ** (2 * h) / domain, domain > 0xffffffff


def blocks(c):
    """AES blocks one trial cannot do without: two for its seeds and either
    every round value of its PRP or one evaluation per item, whichever is less."""
    h, walk, _ = geometry(c)
    return 2 + 8 * min(2.0 ** h, walk * c["t"])


def expense(c):
    """Cost of one trial in AES blocks of the narrow path, walk included, for
    bounding the drawn sizes."""
    h, walk, wide = geometry(c)
    passes = 8 * walk * c["t"] * c["k"]
    return (6 * passes if wide else min(8 * 2.0 ** h if h <= 16 else passes, passes)) + 12 * c["t"] + 20


def sets_of(c):
    """The parameter sets of a batched or served case, from its own draw."""
    rng = random.Random(c["draw"])
    out = []
    for _ in range(c["sets"]):
        if c["call"] == "jobs":
            t = round(math.exp(rng.uniform(math.log(16), math.log(4096))))
            s = shape("bgh25", "affine", t, 24, rng.choice([2, 3, 4]),
                      math.ceil(rng.choice([1.25, 1.35, 1.5]) * t), rng.choice([100, 500]))
            out.append((s, c["count"]))
        else:
            t = round(2 ** rng.uniform(4, 14))
            s = shape("bgh25", "affine", t, 24, rng.choice([2, 3]),
                      math.ceil(rng.choice([1.2, 1.3, 1.4, 1.5]) * t), 500)
            out.append((s, round(2 ** rng.uniform(c["low"], c["high"]))))
    return out


def served_trials(budget):
    """Trials a served budget runs as: whole batches of 2^ceil(log2 budget)."""
    return 1 << max(1, (budget - 1).bit_length())


def draw(rng):
    call = rng.choices(["launch", "device", "static", "jobs", "serve"], [10, 3, 2, 2, 1])[0]
    if call == "jobs":
        return dict(call=call, sets=rng.randint(3, 24), draw=rng.randrange(1 << 20),
                    count=round(2 ** rng.uniform(5, 12)))
    if call == "serve":
        return dict(call=call, sets=rng.randint(2, 16), draw=rng.randrange(1 << 20),
                    low=7, high=rng.randint(9, 13))
    t = round(2 ** rng.uniform(math.log2(3), 9 if call == "static" else 14))
    ell = rng.choice([e for e in (8, 12, 16, 20, 24, 28, 32) if e >= 16 or (1 << e) >= t])
    k = rng.choice([2, 3, 3, 3, 4])
    if rng.random() < 0.25 and k == 3:
        buckets, kick = 0, 0
    else:
        load = rng.choice([2.2, 2.5]) if k == 2 else rng.choice([1.2, 1.25, 1.35, 1.5])
        kick = rng.choice([100, 500, 1000])
        if call != "launch":  # failing trials are all that these return: stressed shapes, as in the tests
            load, kick = (2.2 if k == 2 else 1.15), rng.choice([5, 20])
        buckets = math.ceil(load * t)
    s = shape(rng.choice(["bgh25", "bgh25", "drrt18"]), rng.choice(["sequential", "affine"]), t, ell, k,
              buckets, kick)
    top = min(1 << 20, 1.5e10 / expense(s))
    return dict(call=call, count=max(1, round(2 ** rng.uniform(4, math.log2(top)))), **s)


def parameters(s):
    return package().parameters(s["mode"], s["t"], s["ell"], s["k"], s["buckets"], s["kick"], s["inputs"])


def prepare(case, seed):
    cmc = package()
    ctx = context()
    if case["call"] == "jobs":
        jobs = [(parameters(s), seed * 1000 + i, 0, 0, n) for i, (s, n) in enumerate(sets_of(case))]
        return dict(case=case, ctx=ctx, jobs=jobs)
    if case["call"] == "serve":
        srv = cmc.Server(ctx, max_jobs=1024, mem_budget=8 << 30, batch_bits=20, max_iteration_trials=1 << 22)
        return dict(case=case, server=srv,
                    jobs=[(parameters(s), seed * 1000 + i, n) for i, (s, n) in enumerate(sets_of(case))])
    state = dict(case=case, ctx=ctx, params=parameters(case), key=cmc.batch_key(seed, 1))
    if case["call"] != "launch":
        state["d_key"] = torch.tensor(state["key"], dtype=torch.int64).to(torch.int32).cuda()
        state["offsets"] = torch.zeros(case["count"], dtype=torch.int32, device="cuda")
        state["failed"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    return state


def mask(count, failed):
    """Which of `count` trials failed, from the list of failing offsets."""
    m = np.zeros(count, dtype=bool)
    m[failed] = True
    return m


def run(state):
    case = state["case"]
    if case["call"] == "launch":
        failed = state["ctx"].launch(state["params"], state["key"], 0, case["count"])
        return dict(failed=mask(case["count"], failed), probes=state["ctx"].last_stats()["probes"])
    if case["call"] == "jobs":
        counts, per_job = state["ctx"].run_jobs(state["jobs"])
        return dict(counts=np.array(counts, dtype=np.int64),
                    failed=[mask(n, per_job[i]) for i, (_, _, _, _, n) in enumerate(state["jobs"])])
    if case["call"] == "serve":
        srv = state["server"]
        ids = [srv.submit(p, seed, budget) for p, seed, budget in state["jobs"]]
        while srv.pending():
            srv.step(400_000_000)
        return dict(status=np.array([srv.status(i) for i in ids], dtype=np.int64))
    stream = torch.cuda.current_stream().cuda_stream
    where = (state["d_key"].data_ptr(), 0, case["count"], state["offsets"].data_ptr(),
             state["failed"].data_ptr(), stream)
    if case["call"] == "device":
        state["ctx"].launch_device(state["params"], *where)
    else:
        package().launch_static(state["params"], *where)
    return dict(offsets=state["offsets"], failed=state["failed"])


def work(case):
    """Bytes: keys in, failing offsets out.  Operations: the table lookups of the
    AES blocks no method can do without (160 per block), and one step of the walk
    per item."""
    if case["call"] in ("jobs", "serve"):
        sets = [(s, n if case["call"] == "jobs" else served_trials(n)) for s, n in sets_of(case)]
    else:
        sets = [(case, case["count"])]
    ops = sum(n * (160 * blocks(s) + s["t"]) for s, n in sets)
    return {"bytes": sum(176 + n / 8 for _, n in sets), "flops": ops}
