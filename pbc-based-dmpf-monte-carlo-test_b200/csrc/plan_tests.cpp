// plan_tests -- tests of the context's host side (buffers, graph keys, plans of
// launches) without a GPU: device-memory calls go to a fake, nothing is launched.
#include <functional>
#include <iostream>
#include <stdexcept>

#include "cmc_capi_internal.hpp"

using namespace cmc;

namespace {

int g_checks = 0;

void require(bool ok, const char* what) {
    ++g_checks;
    if (!ok) throw std::runtime_error(what);
}

// A device whose free memory is one run of bytes from kBase on: an allocation
// takes the lowest address where it fits.
struct FakeDevice {
    static constexpr uintptr_t kBase = 1 << 20;
    size_t size = 0;
    std::map<uintptr_t, size_t> live;
    uint32_t allocs = 0, releases = 0;
} g_device;

cudaError_t fake_alloc(void** out, size_t n) {
    ++g_device.allocs;
    uintptr_t at = FakeDevice::kBase;
    for (auto& [p, m] : g_device.live) {
        if (p - at >= n) break;
        at = p + m;
    }
    if (at + n > FakeDevice::kBase + g_device.size) return cudaErrorMemoryAllocation;
    g_device.live[at] = n;
    *out = reinterpret_cast<void*>(at);
    return cudaSuccess;
}

cudaError_t fake_release(void* p) {
    ++g_device.releases;
    return g_device.live.erase(reinterpret_cast<uintptr_t>(p)) ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t fake_available(size_t* n) {
    *n = g_device.size;
    for (auto& [p, m] : g_device.live) *n -= m;
    return cudaSuccess;
}

void use_fake(Ctx& c, size_t bytes) {
    g_device = FakeDevice{};
    g_device.size = bytes;
    c.memory = DeviceMemory{fake_alloc, fake_release, fake_available};
    c.sms = 148;
    c.smem_optin = 232448;
}

int grow_pool(Ctx& c, size_t bytes) {
    void* p = c.d_slots;
    const int rc = c.grow_bytes(p, c.slots_cap, bytes, 1, "pool");
    c.d_slots = static_cast<char*>(p);
    return rc;
}

// A buffer that cannot grow stays as it is, unless giving it up makes the room.
void check_grow() {
    Ctx c;
    use_fake(c, 1000);
    require(grow_pool(c, 400) == CMC_OK && c.slots_cap == 400, "first allocation");
    char* const first = c.d_slots;
    require(grow_pool(c, 300) == CMC_OK && g_device.allocs == 1, "a smaller need allocates nothing");
    require(grow_pool(c, 5000) == CMC_ENOMEM, "more than the device has");
    require(c.d_slots == first && c.slots_cap == 400 && g_device.live.size() == 1 && g_device.releases == 0,
            "a failed allocation leaves the buffer");
    require(grow_pool(c, 800) == CMC_OK && c.slots_cap == 800 && g_device.live.size() == 1,
            "the old buffer makes room for the new one");
    c.fixed_memory = true;  // a stream capture
    const uint32_t calls = g_device.allocs + g_device.releases;
    char* const kept = c.d_slots;
    require(grow_pool(c, 900) == CMC_ENOMEM && g_device.allocs + g_device.releases == calls && c.d_slots == kept &&
                c.slots_cap == 800,
            "no allocation or release during a capture");
    c.fixed_memory = false;
}

// A graph is replayed only with the buffers, and the sizes, it was captured with.
void check_graphs() {
    Ctx c;
    use_fake(c, 1000);
    std::vector<Job> jobs(1);
    cmc_params p;
    require(cmc_derive_params(CMC_MODE_BGH25, 64, 16, 3, 96, 100, 1, &p) == CMC_OK &&
                c.make_job(p, 0, 1000, 0, jobs[0]) == CMC_OK,
            "a job");
    const std::vector<uint32_t> bounds{0, 1};
    auto replays = [&]() {
        for (const Ctx::GraphEntry& g : c.graphs)
            if (g.key == c.graph_key(jobs, bounds, 1000, 1000)) return true;
        return false;
    };
    require(grow_pool(c, 800) == CMC_OK, "pool");
    const uintptr_t large = reinterpret_cast<uintptr_t>(c.d_slots);
    c.graphs.push_back(Ctx::GraphEntry{c.graph_key(jobs, bounds, 1000, 1000)});
    require(replays(), "the same call");
    // a call whose pool does not fit, then the smaller one it falls back to: at
    // no point may the graph of the larger pool match a smaller one at its address
    require(grow_pool(c, 2000) == CMC_ENOMEM, "too large a pool");
    require(!replays() || c.slots_cap >= 800, "a graph replays in its own pool");
    require(grow_pool(c, 100) == CMC_OK, "the pool of the fallback");
    require(!replays() || (reinterpret_cast<uintptr_t>(c.d_slots) == large && c.slots_cap >= 800),
            "a graph replays in its own pool, also after a fallback");
    require(grow_pool(c, 900) == CMC_OK && c.graphs.empty(), "graphs go with the buffer they name");

    // every pointer counts in full
    for (void** at : {(void**)&c.d_jobs, (void**)&c.d_bits, (void**)&c.d_out, (void**)&c.d_slots,
                      (void**)&c.d_job_failed, (void**)&c.h_failed}) {
        void* const was = *at;
        *at = reinterpret_cast<void*>(0x7ffffffffff0);
        const std::string a = c.graph_key(jobs, bounds, 0xfffffffe, 0xfffffffe);
        *at = reinterpret_cast<void*>(0x7ffffffffff1);
        require(a != c.graph_key(jobs, bounds, 0xfffffffe, 0xfffffffe), "a pointer is part of the key");
        *at = was;
    }
}

cmc_params params(uint32_t mode, uint32_t t, uint32_t ell, uint32_t k, uint32_t buckets, uint32_t kick) {
    cmc_params p;
    require(cmc_derive_params(mode, t, ell, k, buckets, kick, CMC_INPUT_AFFINE, &p) == CMC_OK, "parameters");
    return p;
}

// The kernels of a call run one after another: they take the pool in turn, and
// only classes side by side in one kernel have regions of their own.
void check_regions() {
    Ctx c;
    use_fake(c, 0);
    std::vector<cmc_job> in;
    for (uint32_t t : {64u, 200u, 300u, 700u, 1024u, 1500u, 2500u, 4000u, 8000u})
        for (uint32_t k : {2u, 3u, 4u})
            for (uint32_t count : {40u, 65536u})
                in.push_back({params(CMC_MODE_BGH25, t, 24, k, t + t / 2, 500), 1, 0, 0, count});
    uint32_t engines = 0, fused = 0;
    for (int use_fused : {1, 0}) {
        c.use_fused = use_fused;
        std::vector<Job> jobs;
        std::vector<uint32_t> order, bounds;
        uint64_t total = 0;
        LaunchPlan lp;
        require(c.prepare_jobs(in.data(), uint32_t(in.size()), 0, jobs, order, total, bounds) == CMC_OK &&
                    c.plan_launch(jobs, bounds, lp) == CMC_OK,
                "a mix");
        std::vector<uint32_t> runs(lp.plans.size(), 0);
        uint64_t largest = 0;
        for (const auto& members : lp.kernels) {
            uint64_t sum = 0;
            for (uint32_t m : members) {
                ++runs[m];
                const bool own = lp.lanes[m].warps || lp.waves[m].ng;
                engines += own;
                require(!own || members.size() == 1, "lanes and waves have kernels of their own");
                require(lp.region[m] == sum, "regions of one kernel lie side by side");
                sum += lp.pool_bytes(m);
                require(!own || lp.pool_bytes(m) <= c.memory_bytes / 8 + 1024, "an eighth of the device");
            }
            fused += members.size() > 1;
            largest = std::max(largest, sum);
        }
        for (uint32_t n : runs) require(n == 1, "every class runs once");
        require(lp.pool == largest, "the pool holds the largest kernel's regions, not all of them");
    }
    require(engines >= 4 && fused >= 1, "the mix has lanes or waves and a fused kernel");
}

// One call of the jobs as Ctx::run plans it; the text of its plan.
std::string fitted(Ctx& c, const std::vector<cmc_job>& in, LaunchPlan& lp) {
    std::vector<Job> jobs;
    std::vector<uint32_t> order, bounds;
    uint64_t total = 0;
    require(c.prepare_jobs(in.data(), uint32_t(in.size()), 0, jobs, order, total, bounds) == CMC_OK, "jobs");
    const int rc = c.fit_launch(jobs, bounds, lp);
    if (rc) return std::to_string(rc);
    require(lp.pool <= c.slots_cap, "the pool holds the plan");
    return lp.text;
}

// A call whose pool does not fit takes the group engine with fewer walk slots,
// and an equal call after it allocates nothing.
void check_short_memory() {
    const auto has = [](const std::string& text, const char* what) { return text.find(what) != std::string::npos; };
    const uint64_t gb = 1000000000;
    // 13 GB of lane tables; the walk slots of a launch of 200 trials
    const std::vector<cmc_job> lanes{{params(CMC_MODE_BGH25, 16384, 28, 3, 24576, 1000), 4, 0, 0, 65536}};
    const std::vector<cmc_job> waves{{params(CMC_MODE_BGH25, 16384, 20, 3, 65535, 500), 4, 0, 0, 200}};
    const std::vector<cmc_job> wide{{params(CMC_MODE_DRRT18, 50000, 20, 3, 70000, 500), 4, 0, 0, 300}};
    for (const auto* in : {&lanes, &waves, &wide})
        for (uint64_t size : {180 * gb, 5 * gb, 2 * gb, gb / 2, gb / 4}) {
            Ctx c;
            use_fake(c, size);
            std::string first;
            for (int call = 0; call < 3; ++call) {
                LaunchPlan lp;
                const uint32_t calls = g_device.allocs + g_device.releases;
                const std::string text = fitted(c, *in, lp);
                require(has(text, "engine="), "a call that fits in some form succeeds");
                require(size < 180 * gb || in == &wide || has(text, "->"), "the engine of choice where there is room");
                require(call == 0 || (text == first && g_device.allocs + g_device.releases == calls),
                        "an equal call takes the same plan and allocates nothing");
                require(g_device.live.size() == 1, "one pool");
                for (const Plan& pl : lp.plans)
                    require(pl.ng >= 1 && pl.ns >= pl.ng && pl.ns % pl.ng == 0, "slots for every group");
                first = text;
            }
            // under the call's own capture the same plan, and under the caller's
            // the group engine; neither makes a call
            LaunchPlan lp;
            const uint32_t calls = g_device.allocs + g_device.releases;
            c.fixed_memory = c.capturing = true;
            require(fitted(c, *in, lp) == first, "the plan of a capture");
            c.capturing = false;
            require(!has(fitted(c, *in, lp), "->"), "no lanes or waves in the caller's graph");
            c.fixed_memory = false;
            require(g_device.allocs + g_device.releases == calls, "no allocation during a capture");
            // more room: the engine of choice again
            g_device.size = 180 * gb;
            if (in != &wide) require(has(fitted(c, *in, lp), "->"), "memory that was short is not short for good");
        }
    // nothing fits
    Ctx c;
    use_fake(c, 1000000);
    LaunchPlan lp;
    require(fitted(c, lanes, lp) == std::to_string(CMC_ENOMEM) && !c.group_engine && c.slot_budget == ~0ull,
            "too little memory for any form");
    // the caller's limit
    use_fake(c, 180 * gb);
    c.pool_limit = gb;
    require(!has(fitted(c, lanes, lp), "->") && lp.pool <= gb, "a plan within the limit");
}

// A small generator of shapes: t = 3..60000, N = 2^8..2^36, loads and k in use.
struct Draw {
    uint64_t s;
    uint64_t operator()(uint64_t n) {
        s = s * 6364136223846793005ULL + 1442695040888963407ULL;
        return (s >> 33) % n;
    }
};

cmc_params drawn(Draw& d) {
    for (;;) {
        const uint32_t t = uint32_t(3 + (d(64) << d(11)) % 60000), k = uint32_t(2 + d(3)), ell = uint32_t(8 + 4 * d(8));
        const uint32_t load[] = {110, 125, 150, 220};
        cmc_params p;
        if (cmc_derive_params(uint32_t(1 + d(2)), t, ell, k, uint32_t(uint64_t(t) * load[d(4)] / 100) + 1, 100, 1, &p) == CMC_OK)
            return p;
    }
}

// A server plans its jobs at admission, for their size class and for each launch
// with different counts: where the walk slots are and how many bytes are counted
// must not depend on them, and what is admitted runs within the budget.
void check_served_plans() {
    Ctx c;
    use_fake(c, 0);
    Draw d{7};
    const auto jobs_of = [&](const std::vector<cmc_params>& ps, uint32_t count) {
        std::vector<Job> jobs(ps.size());
        for (size_t i = 0; i < ps.size(); ++i)
            require(c.make_job(ps[i], 0, count, 0, jobs[i]) == CMC_OK, "job");
        return jobs;
    };
    for (int i = 0; i < 20000; ++i) {
        const std::vector<cmc_params> one{drawn(d)};
        Plan a, b;
        uint64_t pa = 0, pb = 0;
        require(c.plan_served(jobs_of(one, 1), ~0ull, false, a, pa) == CMC_OK &&
                    c.plan_served(jobs_of(one, 200000), ~0ull, false, b, pb) == CMC_OK,
                "plans");
        require(a.slots_smem == b.slots_smem && pa == pb && a.claim_bytes == b.claim_bytes && a.ng == b.ng &&
                    a.wg == b.wg && a.ns == b.ns,
                "a served plan does not depend on the counts");
        require(a.variant == 0 || a.claim_bytes == pa, "plain slots are counted as they are");
        require(!a.reduced && a.claim_bytes <= pa, "item slots take no less than is counted");
    }
    const std::vector<cmc_params> wide{params(CMC_MODE_BGH25, 2000, 32, 3, 3000, 0)};
    Plan pl;
    uint64_t pool = 0;
    require(c.plan_served(jobs_of(wide, 1), ~0ull, false, pl, pool) == CMC_OK && !pl.slots_smem &&
                pl.claim_bytes > 600000000,
            "t = 2000, N = 2^32 walks global slots and is counted so");

    uint32_t shared = 0, fewer = 0;
    for (int i = 0; i < 20000; ++i) {
        std::vector<cmc_params> set;
        for (uint64_t n = 1 + d(4); n; --n) set.push_back(drawn(d));
        const uint64_t budget = (1 + d(1000)) << d(22);  // bytes for one of two iterations
        require(c.plan_served(jobs_of(set, 1), budget, false, pl, pool) == CMC_OK, "plan");
        if (pl.claim_bytes > budget) continue;  // not admitted
        require(pool <= budget, "an admitted set's iteration is within the budget");
        Plan rp;
        uint64_t rpool = 0;
        require(c.plan_served(jobs_of(set, 1), 2 * budget, true, rp, rpool) == CMC_OK && rpool <= 2 * budget,
                "and so is its resident launch");
        require(!rp.pool_stage, "resident launches have plain producers");
        shared += rp.slots_smem;
        fewer += rp.reduced;
        for (const Plan* q : {&pl, &rp})
            require(q->ng >= 1 && q->ns >= q->ng && q->ns % q->ng == 0 && q->smem_bytes <= 232448 && q->threads <= 512,
                    "a plan that can be launched");
        // each part of the set, in any proportion
        std::vector<cmc_params> part{set[d(set.size())]};
        if (set.size() > 2) part.push_back(set[0]);
        require(c.plan_served(jobs_of(part, uint32_t(1 + d(1 << 20))), budget, false, pl, pool) == CMC_OK && pool <= budget,
                "so is every part of an admitted set");
    }
    require(shared > 100 && fewer > 100, "budgets that bind");
}

}  // namespace

int main() {
    const std::pair<const char*, void (*)()> tests[] = {{"buffers", check_grow}, {"graphs", check_graphs},
                                                        {"regions", check_regions},
                                                        {"short memory", check_short_memory},
                                                        {"served plans", check_served_plans}};
    int bad = 0;
    for (auto& [name, test] : tests) {
        try {
            test();
        } catch (const std::exception& e) {
            std::cerr << "FAILED " << name << ": " << e.what() << '\n';
            ++bad;
        }
    }
    if (!bad) std::cout << "ALL PLAN TESTS PASSED (" << g_checks << " checks)\n";
    return bad != 0;
}
