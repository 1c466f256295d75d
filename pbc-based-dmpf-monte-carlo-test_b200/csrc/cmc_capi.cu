// cmc_capi.cu -- C ABI over the engine: per-device context, launch planning
// and the Launch seam (cuckoo_bench.cu:980-1031).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "cmc.h"
#include "cmc_capi_internal.hpp"
#include "cmc_engine.cuh"
#include "cmc_hostcore.hpp"
#include "cmc_lanes.cuh"
#include "cmc_trial.cuh"
#include "cmc_waves.cuh"

namespace cmc {

template <typename MapT, typename BinT, bool WIDE, bool SMEMSLOTS>
__global__ void cmc_engine(const EngineArgs a);
template <typename MapT, typename BinT, bool WIDE>
__global__ void cmc_engine_split(const EngineArgs a);
template <typename MapT, typename BinT>
__global__ void cmc_engine_pooled(const EngineArgs a);
template <typename MapT, typename BinT, bool WIDE, bool SMEMSLOTS>
__global__ void cmc_engine_fused(const __grid_constant__ FusedArgs f);
template <bool NARROW, bool WIDE>
__global__ void cmc_lanes(const LaneArgs a);
template <bool NARROW, bool GC>
__global__ void cmc_waves(const WaveArgs a);
__global__ void cmc_compact_failures(const uint32_t* bits, uint64_t nbits, uint32_t value_base,
                                     uint32_t* out, uint32_t* count, uint64_t cap,
                                     const unsigned long long* nbits_dev,
                                     CallResult* result, const Ctrl* ctrl, uint32_t nctrl);
__global__ void cmc_selftest(const uint32_t* t0, const uint32_t* fips_rk, uint32_t* out,
                             uint32_t r256);

namespace {

thread_local std::string g_thread_error;


uint32_t round_up(uint32_t x, uint32_t a) { return (x + a - 1) / a * a; }

// What a launch that runs in the lane engine adds to its plan's text.
std::string lanes_text(const LanePlan& lp) {
    if (!lp.warps) return "";
    char buf[96];
    snprintf(buf, sizeof buf, " -> engine=lanes warps=%u lanes_per_warp=%u region=%llu", lp.warps, lp.share,
             (unsigned long long)lp.region_bytes);
    return buf;
}

std::string waves_text(const WavePlan& wp) {
    if (!wp.ng) return "";
    char buf[112];
    snprintf(buf, sizeof buf, " -> engine=waves groups=%u warps_per_group=%u wave=%u region=%llu cache=%s", wp.ng,
             wp.wg, wp.wave, (unsigned long long)wp.region_bytes, wp.global_cache ? "global" : "smem");
    return buf;
}

}  // namespace

void set_thread_error(const std::string& message) { g_thread_error = message; }

int Ctx::fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    err = buf;
    return code;
}

int Ctx::cuda(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return CMC_OK;
    return fail(CMC_ECUDA, "%s: %s", what, cudaGetErrorString(e));
}

// Room for `need` elements of `size` bytes in a device buffer.  A buffer is
// replaced only by a larger one: the new one is allocated first, and only where
// both do not fit the old one is given up for it.  During a stream capture
// (fixed_memory) nothing is allocated or freed: both calls would end the capture.
int Ctx::grow_bytes(void*& ptr, size_t& cap, size_t need, size_t size, const char* what) {
    if (need <= cap && ptr) return CMC_OK;
    const size_t n = std::max<size_t>(need, 1);
    if (fixed_memory)
        return fail(CMC_ENOMEM, "%zu bytes for %s are not allocated during a stream capture", n * size, what);
    void* fresh = nullptr;
    bool ok = memory.alloc(&fresh, n * size) == cudaSuccess;
    size_t left = 0;
    if (!ok && ptr && memory.available(&left) == cudaSuccess && left + cap * size >= n * size) {
        memory.release(ptr);  // waits for the work that uses it
        ptr = nullptr;
        cap = 0;
        forget_graphs();
        ok = memory.alloc(&fresh, n * size) == cudaSuccess;
    }
    if (!ok) {
        cudaGetLastError();
        return fail(CMC_ENOMEM, "cudaMalloc of %zu bytes for %s failed", n * size, what);
    }
    if (ptr) {
        memory.release(ptr);
        forget_graphs();
    }
    ptr = fresh;
    cap = n;
    return CMC_OK;
}

// Captured graphs name the buffers they were captured with.
void Ctx::forget_graphs() {
    for (GraphEntry& g : graphs)
        if (g.exec) cudaGraphExecDestroy(g.exec);
    graphs.clear();
}

template <typename T>
int Ctx::grow(T*& ptr, size_t& cap, size_t need, const char* what) {
    void* p = ptr;
    const int rc = grow_bytes(p, cap, need, sizeof(T), what);
    ptr = static_cast<T*>(p);
    return rc;
}

void Ctx::look_for_capture(cudaStream_t st) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &status) != cudaSuccess) cudaGetLastError();
    fixed_memory = status != cudaStreamCaptureStatusNone;
}

// Map method of a parameter set.  Direct passes cost 8 AES blocks per Feistel
// evaluation, k*t*c evaluations per trial (c = 2^2h / D for cycle-walking).  A
// round cache costs 8 * 2^h blocks per trial and then 8 lookups per
// evaluation: from shared memory (h <= 12, a lookup ~1/64 block) or from an
// L2-resident global buffer (h <= 16; ~0.3 block: the 8 lookups of an
// evaluation are dependent L2 round trips, two chains in flight per lane).
uint32_t choose_method(uint32_t h, uint64_t domain, double candidates, int force, bool may_allocate) {
    const double c = std::ldexp(1.0, 2 * int(h)) / double(domain);
    const double direct = candidates * 8.0 * c;
    const double build = 8.0 * std::ldexp(1.0, int(h));
    const bool gcache_ok = may_allocate && domain <= 0xffffffffULL && h <= 16;
    if (force == 0) return kMethodDirect;
    if (force == 1) return h <= 12 ? kMethodCache : gcache_ok ? kMethodGCache : kMethodDirect;
    if (force == 2) return gcache_ok ? kMethodGCache : kMethodDirect;
    if (h <= 12 && build + direct / 64.0 < direct) return kMethodCache;
    if (gcache_ok && build + direct * 0.3 < direct) return kMethodGCache;
    return kMethodDirect;
}

// Job::last_rows and last_cuts.  L's above the domain lead to another pass and
// need their round; of the others a bucket no narrower than 2^h cuts at most
// one per bucket, at 119 shared-memory wavefronts per 32 entries against 106 in
// rows.  Rows are dropped in pairs (the fill loops' step), and only where a
// sixteenth of the fill goes with them (3 % at t = 1500, k = 4, N = 2^24 lost as
// much in the lookups).  t = 1024, k = 3, N = 2^20 needs 512 of 2048 entries.
static void last_round(Job& j) {
    const uint32_t h = j.half_bits;
    if (j.domain > 0xffffffffULL || h < 9 || h > 16 || j.width < (1ULL << h)) return;
    const uint32_t rows = uint32_t(j.domain >> h >> 8) & ~1u;
    const uint64_t cuts = j.width & j.mask ? (j.domain - 1) / j.width : 0;
    if (256.0 * rows - 1.15 * cuts < j.mask / 2) return;
    j.last_rows = rows;
    j.last_cuts = uint32_t(cuts);
}

// AES blocks of a round cache.
static double cache_blocks(const Job& j) {
    return 8.0 * std::ldexp(1.0, int(j.half_bits)) - 256.0 * j.last_rows + 1.15 * j.last_cuts;
}

// Fill a device job descriptor from derived parameters.
int Ctx::make_job(const cmc_params& p, uint32_t first, uint32_t count, uint64_t base, Job& j) {
    std::memset(&j, 0, sizeof j);
    if (p.mode != CMC_MODE_BGH25 && p.mode != CMC_MODE_DRRT18)
        return fail(CMC_EINVAL, "invalid mode %u", p.mode);
    if (p.k < 2 || p.k > 4) return fail(CMC_EINVAL, "k must be 2..4 (got %u)", p.k);
    if (p.pnum < 3 || p.pnum > 65534) return fail(CMC_EINVAL, "PNUM out of range");
    if (p.buckets < 1 || p.bucket_size < 1 || p.domain == 0)
        return fail(CMC_EINVAL, "invalid bucket parameters");
    if (p.domain > 0xffffffffULL) {
        if (p.half_bits > 32) return fail(CMC_EINVAL, "PRP half width above 32 bits");
    } else if (p.half_bits > 16) {
        return fail(CMC_EINVAL, "PRP half width inconsistent with domain");
    }
    if (uint64_t(p.pnum) * p.k > 0xffffffffULL) return fail(CMC_EINVAL, "too many candidates");
    j.pnum = p.pnum;
    j.k = p.k;
    j.buckets = p.buckets;
    j.kick = p.kick;
    j.mode = p.mode;
    j.input_mode = p.input_mode;
    j.half_bits = p.half_bits;
    j.domain = p.domain;
    j.mask = p.mask;
    j.range_mask = p.range_mask;
    j.width = p.bucket_size;
    j.width_magic = p.domain <= 0xffffffffULL ? uint32_t(0xffffffffULL / p.bucket_size) : 0;
    j.first = first;
    j.count = count;
    j.trial_base = base;
    j.method = choose_method(p.half_bits, p.domain, double(p.pnum) * p.k, force_method, may_allocate);
    last_round(j);
    return CMC_OK;
}

// Choose groups, warps per group and slot placement for a set of jobs.
int Ctx::plan(const std::vector<Job>& jobs, Plan& pl) {
    uint32_t max_b = 0, max_t = 0, max_cand = 0, max_cache_h = 0, any_cache = 0, wide = 0, wide_domain = 0;
    uint32_t max_gcache_h = 0, any_gcache = 0, max_h = 0, dfold_h = 0, any_dfold = 0;
    double work = 0, cand_work = 0;
    for (const Job& j : jobs) {
        max_h = std::max(max_h, j.half_bits);
        if (!plan_no_dfold && j.method == kMethodDirect && j.domain <= 0xffffffffULL && j.half_bits <= 13) {
            any_dfold = 1;  // direct passes with a word-split round-2 fold table
            dfold_h = std::max(dfold_h, j.half_bits);
        }
        max_b = std::max(max_b, j.buckets);
        max_t = std::max(max_t, j.pnum);
        max_cand = std::max(max_cand, j.pnum * j.k);
        if (j.method == kMethodCache) {
            any_cache = 1;
            max_cache_h = std::max(max_cache_h, j.half_bits);
        }
        if (j.method == kMethodGCache) {
            any_gcache = 1;
            max_gcache_h = std::max(max_gcache_h, j.half_bits);
        }
        if (j.domain > 0xffffffffULL) wide_domain = 1;
        // 16-bit entries: 14-bit ordinal + 2-bit choice, never equal to 0xffff
        const bool narrow_ok = j.buckets <= 0xffff && j.pnum <= 16384 && !(j.k == 4 && j.pnum > 16383);
        if (!narrow_ok) wide = 1;
        work += double(j.count);
        cand_work += double(j.count) * j.pnum * j.k;
    }
    if (wide_domain) wide = 1;
    pl.variant = wide_domain ? 2 : (wide ? 1 : 0);
    const uint32_t entry = wide ? 4 : 2;
    // slots are addressed by 32-bit offsets
    if ((uint64_t(max_b) + max_cand) * entry > 0xffffff00ULL)
        return fail(CMC_EINVAL, "a table of %u buckets exceeds the 4 GiB of a walk slot", max_b);
    pl.bins_bytes = round_up(max_b * entry, 16);
    const uint32_t map_bytes = round_up(max_cand * entry, 16);
    pl.slot_stride = round_up(pl.bins_bytes + map_bytes, 128);
    // a round-cache job keeps its fold table (and a shared-memory cache) in
    // its group's shared region
    const uint32_t cache_bytes = any_cache ? fold_table_bytes(max_cache_h) + (16u << max_cache_h) : 0;
    const uint32_t gfold_bytes = any_gcache ? fold_table_bytes(max_gcache_h) : 0;
    const uint32_t dfold_bytes = any_dfold ? fold_table_bytes(dfold_h) : 0;
    pl.group_bytes = kGroupHeaderBytes + std::max({cache_bytes, gfold_bytes, dfold_bytes});
    const double avg_cand = work > 0 ? cand_work / work : 0;
    // one-warp groups for direct passes up to 1,536 candidates per trial (with
    // pooled passes, measured: t=300 k=3 6.75 M trials/s against 5.14 M in
    // 4-warp groups; t=1000: 1.57 M against 1.61 M)
    pl.wg = (any_cache || any_gcache || avg_cand >= 1536.0) ? 4 : 1;
    if (force_wg) pl.wg = force_wg;
    pl.walker_ctas = force_walker_ctas > 0 ? uint32_t(force_walker_ctas) : 0;
    if (pl.walker_ctas >= uint32_t(sms)) return fail(CMC_EINVAL, "walker_ctas must be below the SM count");
    // Isolated walkers (sub-partition 3 only) pay off when walks are long
    // enough to hold producers back; short walks keep all 16 warps busy.
    double avg_probe_work = 0;
    for (const Job& j : jobs) avg_probe_work += double(j.count) * j.pnum;
    avg_probe_work = work > 0 ? avg_probe_work / work : 0;
    pl.isolate = pl.walker_ctas ? 0 : (force_isolate >= 0 ? uint32_t(force_isolate)
                                                          : (avg_probe_work >= 512 ? 1u : 0u));
    pl.nw = pl.walker_ctas ? 0 : (force_walkers ? force_walkers : 1);
    // measured best with isolated walkers: 2 groups of 6 producer warps on
    // sub-partitions 0..2 (2 x 7, adding two beside the walker, is within 3%)
    if (pl.isolate && !force_wg) pl.wg = (any_cache || any_gcache) ? 6 : 4;
    if (pl.isolate && pl.nw > 4) pl.nw = 4;
    const uint32_t budget = uint32_t(smem_optin) - kEngineTableBytes - kCtaSharedBytes;
    uint32_t cap_ng = force_ng;
    // Short launches (longer ones of these shapes run in the lane or wave engine)
    // and calls without allocation, but not a server's, whose plans must not
    // depend on the counts: split all 15 warps beside the
    // walker into as many groups as shared memory holds with enough walk slots
    // -- 4 per group up to 28 -- and as there are trials for.  More, smaller
    // groups overlap their serial set-ups and barriers.  Measured on B200
    // against three 4-warp groups: t=30, N=2^8 0.121 against 0.211 ms (14 x 1),
    // t=200, N=2^16 0.654 against 0.777 (7 x 2), t=600, N=2^24 1.46 against 1.75
    // (5 x 3), t=1300 3.01 against 3.47 (3 x 5),
    // t=2092, k=2 5.43 against 6.43 (2 x 7), t=300, k=4 (h=12) 1.68 against
    // 1.92 (2 x 7).  Direct passes in pooled one-warp groups only where 13 or 14
    // fit (t=280: 12 pooled groups 0.98 ms, 7 x 2 0.75).  Shared caches with long
    // walks keep the walker isolated and take the split with most slots (t=700,
    // N=2^16: 21 slots 1.22 ms, 16 slots 1.40).  64-bit domains, whose set-up is
    // longest, keep their one-warp groups (t=391, k=4: 1.96 against 2.13 ms).
    const double per_sm = work / sms;
    const bool short_launch = !served && (!may_allocate || per_sm <= 200);
    if (short_launch && !force_wg && !force_ng && !force_walkers && force_isolate < 0 &&
        !pl.walker_ctas && !any_gcache && !wide_domain) {
        const bool direct_pool = force_pool != 0 && !any_cache;
        auto slots_at = [&](uint32_t ng, uint32_t bytes) {
            return ng * bytes > budget
                       ? 0u
                       : ng * std::min<uint32_t>({(budget - ng * bytes) / pl.slot_stride / ng, 32 / ng,
                                                  max_slots_per_group});
        };
        if (any_cache && avg_probe_work >= 512) {
            uint32_t most = 0;
            for (uint32_t ng : {1u, 2u, 3u, 4u, 6u}) {
                const uint32_t s = slots_at(ng, pl.group_bytes);
                if (s > most && ng <= std::max(1.0, std::ceil(per_sm))) {
                    most = s;
                    cap_ng = ng;
                    pl.wg = 12 / ng;
                }
            }
        } else {
            for (uint32_t wg : {1u, 2u, 3u, 5u, 7u, 15u}) {
                const uint32_t ng = std::min<uint32_t>(kMaxGroups, 15 / wg);
                if (ng == 1 && avg_probe_work >= 1500) break;  // long walks: isolated walkers, global slots
                const uint32_t pool = pool_group_bytes(round_up(max_cand * entry, 16),
                                                       max_h <= 10 ? fold_table_bytes(max_h) : 0);
                // a group per trial, where there are no more (of tables below a
                // warp's width, whose set-up is most of the work, two)
                if (ng > 1 && ng > (max_cand < 64 ? 2 * per_sm + 1 : per_sm + 0.5)) continue;
                const uint32_t enough = std::min({4 * ng, 28u, std::max(2 * ng, uint32_t(per_sm) + 1)});
                if (wg == 1 && direct_pool && slots_at(ng, pool) < 28 && slots_at(13, pool) < 26) continue;
                if (!(wg == 1 && direct_pool) && slots_at(ng, pl.group_bytes) < enough) continue;
                pl.wg = wg;
                pl.isolate = 0;
                cap_ng = ng;
                break;
            }
        }
    }
    // Pooled direct passes (producer_pooled): one-warp groups whose jobs all
    // use direct passes with 16-bit halves; each group then holds three trials'
    // headers and staged maps.  Dropped below if the walk slots go global.
    // Measured on B200 (same failure lists): t=64, B=96 24.4 -> 29.1 M
    // trials/s; t=27 42.3 -> 58.1 M; t=93 sequential 18.3 -> 20.7 M.
    // With h <= 10 the passes also take the round-2 fold (a trial's fold table
    // has at most 4 entries per round, so a warp's fold loads touch few
    // addresses): 111 table lookups per AES block instead of 124.
    pl.pool_stage = pl.pool_fold = 0;
    if (force_pool != 0 && !any_cache && !any_gcache && !wide_domain && pl.wg == 1 && !pl.walker_ctas) {
        pl.pool_stage = round_up(max_cand * entry, 16);
        pl.pool_fold = max_h <= 10 ? fold_table_bytes(max_h) : 0;
        pl.group_bytes = pool_group_bytes(pl.pool_stage, pl.pool_fold);  // its own fold, if any
    }
    auto groups_for = [&](uint32_t nw) {
        uint32_t ng = std::min<uint32_t>(kMaxGroups, (16 - nw) / pl.wg);
        if (cap_ng) ng = std::min(ng, cap_ng);
        while (ng > 1 && ng * pl.group_bytes > budget) --ng;
        return ng;
    };
    const uint32_t ng = groups_for(pl.nw);
    if (ng * pl.group_bytes > budget)
        return fail(CMC_EINVAL, "round cache of %u bytes does not fit shared memory", cache_bytes);
    // Slots.  A CTA walks about slots / (probes per trial x probe latency)
    // trials per cycle: ~2.4 t probes per trial, ~300 cycles per probe in
    // shared memory (~800 when the walker shares its sub-partition with
    // producers), ~3000 in global memory (two dependent DRAM round trips
    // once the slots outgrow L2).  Its producers build AES blocks at a
    // measured ~0.157 per cycle (direct passes, shared-memory cache) or ~0.2
    // (global round cache), over the job's blocks per trial.  Shared-memory
    // slots (2..8 per group, giving up at most half of the groups) are kept
    // when their walks outpace the producers by 1.4x -- a small pool with
    // uneven walk lengths queues below that -- or beat global slots; global
    // slots take 32 per walker warp, with 4 walker warps on sub-partition 3
    // when walkers are isolated.  The split engine keeps one global slot per
    // walker-CTA thread.
    double avg_cost = 0;
    for (const Job& j : jobs) avg_cost += double(j.count) * job_cost(j);
    avg_cost = work > 0 ? avg_cost / work : 1;
    const double probes = std::max(1.0, 2.4 * avg_probe_work);
    const double produce = (any_gcache ? 0.2 : 0.157) / std::max(1.0, avg_cost);
    const auto caches = [&](uint32_t groups) {  // round caches of all CTAs
        return any_gcache ? uint64_t(sms) * groups * (16u << max_gcache_h) : 0;
    };
    pl.slots_smem = false;
    for (uint32_t g = ng; !pl.walker_ctas && !force_global_slots &&
                          g >= std::max<uint32_t>(1, (ng + 1) / 2); --g) {
        const uint32_t left = budget - g * pl.group_bytes;
        const uint32_t s = std::min<uint32_t>({left / pl.slot_stride / g, 32 * pl.nw / g,
                                               max_slots_per_group});
        if (s >= 2) {
            pl.ng = g;
            pl.ns = g * s;
            pl.slots_smem = true;
            break;
        }
    }
    if (pl.walker_ctas) {
        pl.ng = ng;
        pl.ns = pl.walker_ctas * pl.ng * pl.wg * 32;
    } else {
        const uint32_t nw_g = (pl.isolate && !force_walkers) ? 4 : pl.nw;
        const uint32_t ng_g = groups_for(nw_g);
        const uint32_t ns_g = std::max<uint32_t>(1, std::min(kMaxSlots, 32 * nw_g) / ng_g) * ng_g;
        // a walker beside ALU-bound producers issues slower: ~800 cycles per
        // shared probe (measured at t=500, k=4), ~300 when isolated
        const double walk_smem = pl.slots_smem ? pl.ns / (probes * (pl.isolate ? 300.0 : 800.0)) : 0.0;
        // (short launches: ~4500, measured at t=1500, N=2^16, where 10 shared
        // slots give 3.74 ms and 128 global ones 5.17)
        const double walk_global = ns_g / (probes * (short_launch ? 4500.0 : 3000.0));
        const bool keep_smem = pl.slots_smem && (!may_allocate || walk_smem >= 1.4 * produce ||
                                                 walk_smem >= walk_global ||
                                                 (short_launch && !any_gcache && pl.ns > per_sm));  // a slot for every trial
        if (!keep_smem) {
            pl.slots_smem = false;
            pl.nw = nw_g;
            pl.ng = ng_g;
            pl.ns = ns_g;
        }
    }
    // (the split engine has one pool of slots, the others one per CTA)
    pl.claim_bytes = pl.slots_smem ? 0 : uint64_t(pl.walker_ctas ? 1 : sms) * pl.ns * pl.slot_stride;
    pl.claim_bytes = (pl.claim_bytes + 255) / 256 * 256 + caches(pl.ng);
    pl.reduced = false;
    if (!pl.slots_smem && !pl.walker_ctas && !force_global_slots &&
        uint64_t(sms) * (wide ? pl.slot_stride : 8ull * (max_b + max_t)) + caches(1) > slot_budget) {
        // not even one global slot per CTA is within the budget
        for (uint32_t g = groups_for(1); g >= 1 && !pl.slots_smem; --g) {
            const uint32_t left = budget - g * pl.group_bytes;
            const uint32_t s = std::min<uint32_t>({left / pl.slot_stride / g, 32 / g, max_slots_per_group});
            if (s < 1) continue;
            pl.slots_smem = true;
            pl.nw = 1;
            pl.ng = g;
            pl.ns = g * s;
        }
    }
    if (pl.slots_smem && caches(pl.ng) > slot_budget) {
        const uint32_t s = pl.ns / pl.ng;
        while (pl.ng > 1 && caches(pl.ng) > slot_budget) --pl.ng;
        pl.ns = pl.ng * s;
    }
    if (!pl.slots_smem) pl.pool_stage = pl.pool_fold = 0;
    if (!pl.slots_smem && !pl.walker_ctas) {
        if (!wide) {
            // global slots of items (item_slots in cmc_engine.cu): [B x 8 bytes]
            // [t x 8 bytes]
            pl.bins_bytes = round_up(max_b * 8, 16);
            pl.slot_stride = round_up(pl.bins_bytes + max_t * 8, 128);
        }
        // as many as the budget holds beside the round caches, down to one per
        // group and then one group
        auto fit = [&](uint32_t groups) {
            return (slot_budget - std::min(slot_budget, caches(groups))) / (uint64_t(sms) * pl.slot_stride);
        };
        pl.reduced = fit(pl.ng) < pl.ns;
        while (pl.ng > 1 && fit(pl.ng) < pl.ng) --pl.ng;
        if (pl.ns > fit(pl.ng)) pl.ns = std::max<uint32_t>(1, uint32_t(fit(pl.ng)) / pl.ng) * pl.ng;
        if (pl.ns % pl.ng) pl.ns -= pl.ns % pl.ng;
    }
    pl.group_off = kEngineTableBytes + kCtaSharedBytes;
    pl.slots_off = pl.group_off + pl.ng * pl.group_bytes;
    pl.smem_bytes = pl.slots_off + (pl.slots_smem ? pl.ns * pl.slot_stride : 0);
    if (pl.isolate) {
        pl.threads = 512;  // walker warps sit at ids 15, 11, ...; unused ids exit at once
    } else {
        pl.threads = (pl.ng * pl.wg + pl.nw) * 32;
    }
    pl.ctas = sms;
    pl.gslot_bytes = pl.walker_ctas  ? uint64_t(pl.ns) * pl.slot_stride
                     : pl.slots_smem ? 0
                                     : uint64_t(pl.ctas) * pl.ns * pl.slot_stride;
    pl.gcache_stride = any_gcache ? (8u << max_gcache_h) : 0;
    pl.gcache_bytes = uint64_t(pl.ctas) * pl.ng * pl.gcache_stride * 2;
    char buf[256];
    snprintf(buf, sizeof buf,
             "engine=%s variant=%s groups=%u warps_per_group=%u walkers=%u%s slots=%u slots_in=%s "
             "smem=%u threads=%u ctas=%u cache=%s%s",
             pl.walker_ctas ? "split" : "group", pl.variant == 0 ? "narrow" : pl.variant == 1 ? "wide" : "wide-domain", pl.ng, pl.wg,
             pl.walker_ctas ? pl.walker_ctas : pl.nw, pl.isolate ? "(isolated)" : "", pl.ns,
             pl.slots_smem ? "smem" : "global", pl.smem_bytes, pl.threads, pl.ctas,
             any_cache && any_gcache ? "smem+global" : any_cache ? "smem" : any_gcache ? "global" : "off",
             pl.pool_stage ? " pooled" : "");
    plan_text = buf;
    // The fold tables of direct passes (build_map_direct) come out of the walk
    // slots' shared memory; with fewer than 4 slots per group left, or none,
    // the walks lose more than the passes gain (measured at t=2000, h=13:
    // 9 -> 6 slots, 0.82 -> 0.72 M trials/s; t=1000: 18 -> 15 slots, 1.59 ->
    // 1.74 M), so plan again without them.
    if (any_dfold && !pl.pool_stage && (!pl.slots_smem || pl.ns < 4 * pl.ng)) {
        plan_no_dfold = true;
        const int rc2 = plan(jobs, pl);
        plan_no_dfold = false;
        return rc2;
    }
    return CMC_OK;
}

namespace {

// Expected number of (item, copy) buckets the lane engine evaluates in one
// trial: every probe of a random walk meets an empty bin with probability
// 1 - load, so filling B bins up to t takes -B ln(1 - t/B) distinct buckets
// (simulated at t = 1024: 1,688 of 1,688 at B = 1536, 2,136 at B = 1250).
// With k = 2 a walk fails soon after half of the bins are full.
double lane_evaluations(const Job& j) {
    const double b = j.buckets, cand = double(j.pnum) * j.k;
    const double t = j.k == 2 ? std::min<double>(j.pnum, 0.55 * b) : double(j.pnum);
    return t < 0.999 * b ? std::min(cand, -b * std::log(1.0 - t / b)) : cand;
}

// Feistel passes per evaluation (cycle-walking).
double walk_factor(const Job& j) { return std::ldexp(1.0, 2 * int(j.half_bits)) / double(j.domain); }

// Expected probes of one trial (measured at t/B = 2/3: 2.39 t and 1.75 t).
double expected_probes(const Job& j) {
    return (j.mode == CMC_MODE_BGH25 ? 2.4 : 1.75) * j.pnum * (j.k == 2 ? 0.8 : 1.0);
}

// Probes by which the longest walk of a launch of small tables exceeds the
// mean: one of its trials fails, at the eviction limit.
double straggler_probes(const Job& j) { return j.pnum < 256 ? std::min<double>(j.kick, 500) : 0.0; }

// The three engines' times for a launch, in SM cycles.  Constants fitted to 290
// launches drawn over t = 3..15,000, N = 2^8..2^32, k = 2..4, both modes and
// 2^2..2^20 trials (B200), standard errors 30 % (group), 30 % (lanes), 14 %
// (waves); the engine chosen is within 3 % of the best one on average.
//
// Group engine: AES blocks over the measured 0.19-0.21 blocks per cycle and SM
// (0.135 with 64-bit domains, 0.125-0.15 beside walks over global slots) and a
// trial's serial set-up in its group, or its walks over the slots, whichever
// takes longer, and one trial's latency.
double group_cycles(const std::vector<Job>& jobs, const Plan& g, int sms) {
    double trials = 0, produce = 0, walk = 0, latency = 0;
    const bool wide_domain = g.variant == 2;
    for (const Job& j : jobs) {
        const double n = j.count, cand = double(j.pnum) * j.k * walk_factor(j);
        const double build = j.method == kMethodDirect ? 8.0 * cand : 8.0 * std::ldexp(1.0, int(j.half_bits));
        const double rate = wide_domain ? 0.135 : g.pool_stage ? 0.21
                            : j.method == kMethodGCache ? (g.slots_smem ? 0.17 : 0.15)
                            : g.slots_smem || j.method == kMethodCache ? 0.19 : 0.125;
        const double lookups = j.method == kMethodCache ? cand : j.method == kMethodGCache ? 1.5 * cand : 0.0;
        trials += n;
        produce += n * ((2.0 + build) / rate + lookups +
                        (g.pool_stage ? 600.0 : (wide_domain ? 25000.0 : 17000.0) / g.ng));
        const double probe = g.slots_smem ? (g.isolate ? (j.mode == CMC_MODE_BGH25 ? 350.0 : 900.0) : 500.0) : 3500.0;
        walk += n * expected_probes(j) * probe / std::max(1u, g.ns);
        latency = std::max(latency, (expected_probes(j) + straggler_probes(j)) * (g.slots_smem ? 180.0 : 1600.0) +
                                        6.0 * build);
    }
    return std::max(produce, walk) / trials * (trials / sms + 0.5) + latency + 24000.0;
}

}  // namespace

// The lane engine's form of a launch (warps == 0: it does not fit).  A trial is
// a chain of P passes (evaluations x cycle-walking, +8 % for passes a BGH25 lane
// sits out, +2 % for DRRT18), and W warps make a pass in 8,000 + 740 W cycles
// (latency of 80 dependent AES rounds, then 960 shared-memory wavefronts per
// warp; 15 % more with 64-bit domains); W is chosen by the estimate.
LanePlan Ctx::plan_lanes(const std::vector<Job>& jobs, const Plan& group) const {
    LanePlan lp;
    const bool wide_domain = group.variant == 2;
    double trials = 0, max_b = 0, passes = 0, longest = 0;  // passes: of all trials
    double spread = 0, sits_out = 0;  // relative spread of a trial's passes; passes a straggler sits out
    for (const Job& j : jobs) {
        const double n = j.count, e = lane_evaluations(j);
        // a lane on known buckets sits out up to one pass per kLaneHops probes
        const double idle = j.pnum < 16 ? j.kick / double(kLaneHops) : 0.0;
        const double p = e * walk_factor(j) * (j.mode == CMC_MODE_BGH25 ? 1.08 : 1.02) + 0.02 * idle;
        trials += n;
        max_b = std::max<double>(max_b, j.buckets);
        spread += n * (jobs.size() > 1 ? 0.5 : (j.mode == CMC_MODE_BGH25 ? 2.0 : 1.1) / std::sqrt(std::max(1.0, e)));
        passes += n * p;
        longest = std::max(longest, p + 3.0 * std::sqrt(p) + 6.0 + idle);
        sits_out = std::max(sits_out, idle);
    }
    const double per_sm = trials / sms;
    uint32_t warps = 0;
    lp.cycles = 1e300;
    for (uint32_t w = 1; w <= kMaxLaneWarps; ++w) {
        if (force_lanes > 0 && w != uint32_t(force_lanes)) continue;
        const double lanes = w * std::min(32.0, std::ceil(per_sm / w));
        const double step = (8000.0 + 740.0 * w) * (wide_domain ? 1.15 : 1.0);
        // trials of even length run in whole waves; the more their lengths
        // differ, the less the last wave waits for
        const double waves = per_sm / lanes;
        const double even = std::max(0.0, 1.0 - 3.0 * spread / trials * std::sqrt(waves));
        const double tail = even * (std::ceil(waves) - waves) + (1.0 - even) * 0.5 + 0.1;
        const double cycles = (waves <= 1.0 ? longest * step : passes / trials * step * (waves + tail) + 0.3 * sits_out * step) +
                              4000.0 * waves + 30000.0;
        if (cycles < lp.cycles) {
            lp.cycles = cycles;
            warps = w;
        }
    }
    lp.variant = group.variant;
    lp.ctas = sms;
    lp.share = uint32_t(std::min(32.0, std::max(1.0, std::ceil(per_sm / warps))));
    lp.region_bytes = (uint64_t(max_b) * (group.variant == 0 ? 8 : 16) + 127) / 128 * 128;
    if (lp.region_bytes > 0xffffffffULL) return lp;  // a table is filled by 32-bit counts
    lp.smem_bytes = kLaneTableBytes + warps * kLaneFoldBytes;
    lp.regions_bytes = lp.region_bytes * sms * warps * lp.share;
    lp.stock_bytes = uint64_t(sms) * warps * kRecordBlockBytes;
    // tables of all lanes: 13.0 GB at B = 24576; never more than an eighth of the device
    if (lp.regions_bytes + lp.stock_bytes > memory_bytes / 8 || lp.smem_bytes > smem_optin) return lp;
    lp.warps = warps;
    return lp;
}

// The wave engine's form of a launch (ng == 0: it does not fit).  A map costs
// the fill (8 * 2^h blocks or less at 106 wavefronts per 32 and 98 % of the shared-memory
// pipe: 3.4 cycles a block), its lookups and 3 cycles per probe; a walk step
// takes 900 cycles and 145 more per lane of the warp.  Fewer groups lose overlap
// of fill, map and walk; more than two spill global caches out of L2, and at
// h = 16 two do out of L1 (t=12000, k=4, N=2^28: 28.0 ms with one, 34.5 with two;
// t=4139 48.6 and 51.3).  With one
// group at h = 13, 1.15 is where its lookups begin to pay (about 8,000 passes).
WavePlan Ctx::plan_waves(const std::vector<Job>& jobs, const Plan& group) const {
    WavePlan wp;
    wp.cycles = 1e300;
    if (group.variant == 2) return wp;
    double trials = 0, build = 0, probes = 0, stragglers = 0;
    uint64_t max_b = 0, max_t = 0;
    uint32_t max_h = 0;
    for (const Job& j : jobs) max_h = std::max(max_h, j.half_bits);
    double lookups = 0;
    for (const Job& j : jobs) {
        lookups += j.count * double(j.pnum) * j.k * walk_factor(j);
        build += j.count * (3.4 * cache_blocks(j) + 3.0 * expected_probes(j) + 1200.0);
        probes = std::max(probes, expected_probes(j));
        stragglers = std::max(stragglers, straggler_probes(j));
        trials += j.count;
        max_b = std::max<uint64_t>(max_b, j.buckets);
        max_t = std::max<uint64_t>(max_t, j.pnum);
    }
    const uint64_t entry = group.variant == 0 ? 8 : 16;
    WavePlan q;
    q.variant = group.variant;
    q.ctas = sms;
    q.cache_off = kWaveHeaderBytes + fold_table_bytes(max_h);
    const uint64_t map_off = (max_b * entry + 15) / 16 * 16;
    if (map_off > 0xffffffffULL) return wp;  // WavePlan::map_off
    q.map_off = uint32_t(map_off);
    q.region_bytes = (map_off + max_t * entry + 127) / 128 * 128;
    for (uint32_t ng : {1u, 2u, 4u, 8u}) {
        if (force_waves > 0 && ng > uint32_t(force_waves)) break;
        // A round cache of h = 13 (128 KiB) fits in shared memory beside the
        // T-table for one group.  Its fill and map then no longer overlap, but
        // the map's gathers from L2 go: one group against two with global
        // caches 7.2 against 7.4 ms (t=2570, k=3), 40.6 against 43.9 (t=4599,
        // k=2, 30,000 trials), 23.4 against 26.5 (DRRT18 t=15580).  Parts of
        // larger caches there measured slower (h=14, 2 of 8 rounds: 47.2 ->
        // 56.3 ms): L1 holds as much of them and loses that room.
        const bool gc = max_h > (ng == 1 ? 13 : 12);
        const double map = (build + (gc ? 6.0 : 1.8) * lookups) / trials;
        q.global_cache = gc;
        q.gcache_stride = gc ? 8u << max_h : 0;
        q.group_bytes = q.cache_off + (gc ? 0 : 16u << max_h);
        q.smem_bytes = kEngineTableBytes + ng * q.group_bytes;
        if (q.smem_bytes > smem_optin) continue;
        q.ng = ng;
        q.wg = 16 / ng;
        q.gcache_bytes = uint64_t(sms) * ng * q.gcache_stride * 2;
        const double lost = gc ? (ng == 1 ? (max_h == 16 ? 0.95 : 1.02) : ng == 2 ? 1.0 : ng == 4 ? 1.03 : 1.2) *
                                     (q.gcache_bytes > 140000000 ? 1.08 : 1.0)
                               : (ng == 1 ? (max_h == 13 ? 1.15 : 1.3) : ng == 2 ? 1.12 : ng == 4 ? 1.0 : 0.97);
        // One wave where a group's share of the launch fits its threads: the
        // walks of all groups then run once, after all maps.  Longer launches
        // run in waves of equal size; towards the end they shrink to the trials
        // whose maps take as long to build as a walk does.
        const double share = std::ceil(trials / (double(sms) * ng)), nt = q.wg * 32, waves = std::ceil(share / nt);
        q.wave = uint32_t(std::ceil(share / waves));
        const double walk = probes * (900.0 + 145.0 * q.wave / q.wg) + 1000.0 * stragglers;
        q.min_wave = waves > 1 ? uint32_t(std::min(double(q.wave), std::max(1.0, walk / (map * ng)))) : q.wave;
        const double maps = share * ng * map * lost;
        q.cycles = (waves > 1 ? std::max(maps, waves * walk) : maps) + walk + 60000.0;
        q.regions_bytes = q.region_bytes * sms * ng * q.wave;
        q.stock_bytes = uint64_t(sms) * ng * q.wg * kRecordBlockBytes;
        if (q.regions_bytes + q.stock_bytes + q.gcache_bytes > memory_bytes / 8) continue;
        if (q.cycles < wp.cycles || force_waves > 0) wp = q;
    }
    return wp;
}

// Which engine runs a launch whose group-engine plan is `group`: lanes and
// waves are left empty where it is the group engine.  The others have to be
// estimated 10 and 16 % shorter, about the estimates' error.
void Ctx::choose_engine(const std::vector<Job>& jobs, const Plan& group, LanePlan& lanes, WavePlan& waves) const {
    lanes = LanePlan{};
    waves = WavePlan{};
    if (group_engine) return;
    const bool group_options = force_wg || force_ng || force_global_slots || force_walkers ||
                               force_walker_ctas >= 0 || force_isolate >= 0 || force_method >= 0 ||
                               force_pool >= 0 || max_slots_per_group != 8 || map_chains || fill_blocks;
    if (force_waves > 0) {
        waves = plan_waves(jobs, group);
        if (waves.ng) return;
    }
    if (force_lanes > 0) {
        lanes = plan_lanes(jobs, group);
        return;
    }
    uint64_t count = 0, items = 0;
    for (const Job& j : jobs) {
        count += j.count;
        items = std::max<uint64_t>(items, j.pnum);
    }
    // the smallest launches gain nothing: not worth the estimates
    if (group_options || force_waves > 0 || (count < 4ull * sms && items < 128)) return;
    const double limit = group_cycles(jobs, group, sms);
    if (force_waves < 0) waves = plan_waves(jobs, group);
    if (force_lanes < 0 && count >= 16ull * sms) lanes = plan_lanes(jobs, group);
    if (!lanes.warps || lanes.cycles >= 0.9 * limit) lanes = LanePlan{};
    if (!waves.ng || waves.cycles >= 0.84 * limit || (lanes.warps && lanes.cycles < waves.cycles)) waves = WavePlan{};
    if (waves.ng) lanes = LanePlan{};
}

// Plans of a call, one per plan class: class c covers the job-table range
// [bounds[c], bounds[c + 1]) and so a contiguous range of global trial indices.
// Several classes of the group engine run as ONE persistent kernel per entry
// width and walk-slot placement that two or more of them share (both are
// template parameters), in the order of each kind's heaviest class, unless
// "fused" is off or a class uses the split engine.  Pooled direct passes, lanes
// and waves have kernels of their own, as a class alone in its kind.
//
// The kernels of a call run one after another in one stream and take the pool in
// turn; only classes side by side in a fused kernel have regions of their own
// (64 sets of t = 16..4096 with 65,536 trials each: 2.6 GB, 6.6 with a region
// for every class).
int Ctx::plan_launch(const std::vector<Job>& jobs, const std::vector<uint32_t>& bounds, LaunchPlan& lp) {
    const uint32_t nclass = uint32_t(bounds.size()) - 1;
    if (nclass < 1 || nclass > kMaxClasses) return fail(CMC_EINVAL, "bad plan classes");
    lp.plans.assign(nclass, Plan{});
    lp.lanes.assign(nclass, LanePlan{});
    lp.waves.assign(nclass, WavePlan{});
    lp.work.assign(nclass, 0.0);
    lp.trials.assign(nclass, 0.0);
    lp.region.assign(nclass, 0);
    lp.kernels.clear();
    lp.pool = 0;
    lp.heaviest = 0;
    lp.text.clear();
    bool any_split = false;
    std::vector<Job> some;
    for (uint32_t c = 0; c < nclass; ++c) {
        if (nclass > 1) some.assign(jobs.begin() + bounds[c], jobs.begin() + bounds[c + 1]);
        const std::vector<Job>& part = nclass > 1 ? some : jobs;
        const int rc = plan(part, lp.plans[c]);
        if (rc) return rc;
        any_split = any_split || lp.plans[c].walker_ctas;
        for (const Job& j : part) {
            lp.trials[c] += double(j.count);
            lp.work[c] += job_cost(j) * j.count;
        }
        if (lp.trials[c] > lp.trials[lp.heaviest]) lp.heaviest = c;
        choose_engine(part, lp.plans[c], lp.lanes[c], lp.waves[c]);
        if (c) lp.text += " | ";
        lp.text += plan_text;
        if (lp.lanes[c].warps) lp.text += lanes_text(lp.lanes[c]);
        if (lp.waves[c].ng) lp.text += waves_text(lp.waves[c]);
    }
    const bool fuse = use_fused && nclass > 1 && nclass <= kMaxFusedClasses && !any_split;
    if (fuse) lp.text = "fused(" + std::to_string(nclass) + ") " + lp.text;
    std::vector<bool> placed(nclass, false);
    for (uint32_t lead = 0; lead < nclass && fuse; ++lead) {
        auto alone = [&](uint32_t c) { return placed[c] || lp.plans[c].pool_stage || lp.lanes[c].warps || lp.waves[c].ng; };
        if (alone(lead)) continue;
        std::vector<uint32_t> members;
        for (uint32_t c = lead; c < nclass; ++c)
            if (!alone(c) && lp.plans[c].variant == lp.plans[lead].variant &&
                lp.plans[c].slots_smem == lp.plans[lead].slots_smem)
                members.push_back(c);
        if (members.size() < 2) continue;
        for (uint32_t c : members) placed[c] = true;
        lp.kernels.push_back(members);
    }
    for (uint32_t c = 0; c < nclass; ++c)
        if (!placed[c]) lp.kernels.push_back({c});
    for (const std::vector<uint32_t>& members : lp.kernels) {
        uint64_t at = 0;
        for (uint32_t c : members) {
            lp.region[c] = at;
            at += lp.pool_bytes(c);
        }
        lp.pool = std::max(lp.pool, at);
    }
    return CMC_OK;
}

// Room for n bytes of tables, walk slots and round caches.  A size that the
// device did not have is asked for again only when there is more room than there
// was then, so that a context short of memory does not try on every call.
int Ctx::reserve_pool(uint64_t n) {
    if (n == 0 || (n <= slots_cap && d_slots)) return CMC_OK;
    if (n > pool_limit)
        return fail(CMC_ENOMEM, "%llu bytes of walk tables exceed the option pool_bytes", (unsigned long long)n);
    auto room = [&]() {
        size_t left = 0;
        return memory.available(&left) == cudaSuccess ? uint64_t(left) + slots_cap : 0;
    };
    if (refused && n >= refused && !fixed_memory && room() <= refused_room)
        return fail(CMC_ENOMEM, "%llu bytes of walk tables do not fit the device", (unsigned long long)n);
    const int rc = grow(d_slots, slots_cap, size_t(n), "slot and cache pool");
    if (rc == CMC_ENOMEM && !fixed_memory) {
        if (!refused || n < refused) refused = n;
        refused_room = room();
    } else if (rc == CMC_OK && n >= refused) {
        refused = 0;
    }
    return rc;
}

// The plan of a call and the pool it needs.  Where the device, or the caller's
// limit, has no room for it: the group engine alone, and then with half as many
// walk slots each time (t = 16384, B = 65535, 200 trials: 0.35 GB of waves, else
// 12.4 GB of walk slots at most and 0.1 at least).
int Ctx::fit_launch(const std::vector<Job>& jobs, const std::vector<uint32_t>& bounds, LaunchPlan& lp) {
    // A graph that the caller captures names the pool for as long as it lives, and
    // a later call may replace that: the group engine, which mostly needs none.
    group_engine = fixed_memory && !capturing;
    int rc = plan_launch(jobs, bounds, lp);
    if (!rc) rc = reserve_pool(lp.pool);
    group_engine = false;
    if (rc != CMC_ENOMEM) return rc;
    const std::string why = err;
    const uint64_t budget = slot_budget;
    uint64_t smallest = lp.pool;  // that was refused
    group_engine = true;
    for (;;) {
        if ((rc = plan_launch(jobs, bounds, lp))) break;
        if (lp.pool < smallest) {
            if ((rc = reserve_pool(lp.pool)) != CMC_ENOMEM) break;
            smallest = lp.pool;
        } else if (slot_budget < (1u << 20)) {
            rc = fail(CMC_ENOMEM, "%s", why.c_str());
            break;
        }
        slot_budget = std::min(slot_budget, lp.pool) / 2;
    }
    group_engine = false;
    slot_budget = budget;
    return rc;
}

// Queue the engine kernels of a call over `jobs` (already on the device in
// d_jobs) and the compaction of their shared failure bitmap.
int Ctx::run(const std::vector<Job>& jobs, uint64_t total, cudaStream_t st, uint32_t value_base,
             uint32_t* d_out, uint32_t* d_count, uint64_t out_cap_now,
             unsigned long long* job_failed, unsigned long long* job_done,
             const std::vector<uint32_t>* bounds_in, bool read_back) {
    // launch checks below read cudaGetLastError: start from a clean slate (an
    // earlier non-fatal error, e.g. of a timing query, is not this launch's)
    cudaGetLastError();
    const std::vector<uint32_t> bounds = bounds_in ? *bounds_in : std::vector<uint32_t>{0, uint32_t(jobs.size())};
    const uint32_t nclass = uint32_t(bounds.size()) - 1;
    LaunchPlan& lp = call_plan;
    int rc = fit_launch(jobs, bounds, lp);
    if (rc) return rc;
    const std::vector<Plan>& plans = lp.plans;
    plan_text = lp.text;
    const size_t words = (total + 31) / 32;
    if ((rc = bitmap(words))) return rc;
    uint32_t* const bits = d_bits + kCtrlWords;
    if ((rc = cuda(cudaMemsetAsync(d_bits, 0, (kCtrlWords + words) * 4, st), "memset ctrl and bitmap"))) return rc;
    // timing events stay out of captured graphs: a replay records them
    // around the graph launch instead
    if (!capturing && (rc = cuda(cudaEventRecord(ev_start, st), "event"))) return rc;
    kernels = 0;
    auto class_args = [&](uint32_t c) {
        const Plan& pl = plans[c];
        char* base = d_slots + lp.region[c];
        const size_t cache_off = size_t((pl.gslot_bytes + 255) / 256 * 256);
        EngineArgs a{};
        a.jobs = d_jobs;
        a.njobs = uint32_t(jobs.size());
        a.gidx_begin = jobs[bounds[c]].trial_base;
        a.total = bounds[c + 1] < jobs.size() ? jobs[bounds[c + 1]].trial_base : total;
        a.ctrl = d_ctrl + c;
        a.fail_bits = bits;
        a.job_failed = job_failed;
        a.job_done = job_done;
        a.gslots = pl.slots_smem ? nullptr : base;
        a.gcache = pl.gcache_bytes ? reinterpret_cast<uint16_t*>(base + cache_off) : nullptr;
        a.gcache_stride = pl.gcache_stride;
        a.ghdr = pl.walker_ctas ? d_ghdr : nullptr;
        a.split = pl.walker_ctas ? 1 : 0;
        a.producer_ctas = pl.ctas - pl.walker_ctas;
        a.total_groups = a.producer_ctas * pl.ng;
        a.t0 = d_t0;
        a.slot_stride = pl.slot_stride;
        a.bins_bytes = pl.bins_bytes;
        a.ng = pl.ng;
        a.wg = pl.wg;
        a.ns = pl.ns;
        a.nw = pl.nw;
        a.isolate_walkers = pl.isolate;
        a.r256 = 256u;
        a.group_bytes = pl.group_bytes;
        a.group_off = pl.group_off;
        a.slots_off = pl.slots_off;
        a.spin_limit = spin_limit;
        a.idle_polls = spin_limit;
        a.map_chains = map_chains;
        a.fill_blocks = fill_blocks;
        a.pool_stage = pl.pool_stage;
        a.pool_fold = pl.pool_fold;
        return a;
    };
    for (const std::vector<uint32_t>& members : lp.kernels) {
        if (members.size() > 1) {
            FusedArgs fa{};
            fa.nclass = uint32_t(members.size());
            uint32_t smem = 0;
            double all = 0, cum = 0;
            for (uint32_t c : members) all += lp.work[c];
            for (uint32_t i = 0; i < members.size(); ++i) {
                const uint32_t c = members[i];
                fa.cls[i] = class_args(c);
                fa.cost[i] = float(lp.work[c] / std::max(1.0, lp.trials[c]));
                fa.first_cta[i] = uint16_t(std::lround(double(sms) * cum / std::max(all, 1e-30)));
                cum += lp.work[c];
                smem = std::max(smem, plans[c].smem_bytes);
            }
            fa.first_cta[members.size()] = uint16_t(sms);
            const Plan& lead = plans[members[0]];
            const void* fn = fused_engine_kernel(lead.variant, lead.slots_smem);
            void* args[] = {&fa};
            if ((rc = cuda(cudaLaunchKernel(fn, dim3(sms), dim3(512), args, smem, st), "fused engine launch")))
                return rc;
            ++kernels;
            continue;
        }
        const uint32_t c = members[0];
        const Plan& pl = plans[c];
        if (lp.waves[c].ng) {
            const WavePlan& wp = lp.waves[c];
            const EngineArgs e = class_args(c);
            WaveArgs a{};
            a.jobs = e.jobs;
            a.njobs = e.njobs;
            a.total = e.total;
            a.gidx_begin = e.gidx_begin;
            a.ctrl = e.ctrl;
            a.fail_bits = e.fail_bits;
            a.job_failed = e.job_failed;
            a.t0 = e.t0;
            a.regions = d_slots + lp.region[c];
            a.region_bytes = wp.region_bytes;
            a.map_off = wp.map_off;
            a.wave = wp.wave;
            a.min_wave = wp.min_wave;
            a.stock = reinterpret_cast<uint32_t*>(a.regions + wp.regions_bytes);
            a.gcache = wp.global_cache ? reinterpret_cast<uint16_t*>(a.regions + wp.regions_bytes + wp.stock_bytes)
                                       : nullptr;
            a.gcache_stride = wp.gcache_stride;
            a.ng = wp.ng;
            a.wg = wp.wg;
            a.group_bytes = wp.group_bytes;
            a.cache_off = wp.cache_off;
            void* args[] = {&a};
            if ((rc = cuda(cudaLaunchKernel(wave_kernel(wp.variant, wp.global_cache), dim3(wp.ctas),
                                            dim3(wp.ng * wp.wg * 32), args, wp.smem_bytes, st),
                           "wave engine launch")))
                return rc;
            ++kernels;
            continue;
        }
        if (lp.lanes[c].warps) {
            const LanePlan& ln = lp.lanes[c];
            const EngineArgs e = class_args(c);
            LaneArgs a{};
            a.jobs = e.jobs;
            a.njobs = e.njobs;
            a.total = e.total;
            a.gidx_begin = e.gidx_begin;
            a.ctrl = e.ctrl;
            a.fail_bits = e.fail_bits;
            a.job_failed = e.job_failed;
            a.t0 = e.t0;
            a.regions = d_slots + lp.region[c];
            a.region_bytes = ln.region_bytes;
            a.hops = kLaneHops;
            a.stock = reinterpret_cast<uint32_t*>(a.regions + ln.regions_bytes);
            a.share = ln.share;
            void* args[] = {&a};
            if ((rc = cuda(cudaLaunchKernel(lane_kernel(ln.variant), dim3(ln.ctas), dim3(ln.warps * 32), args,
                                            ln.smem_bytes, st),
                           "lane engine launch")))
                return rc;
            ++kernels;
            continue;
        }
        if (pl.walker_ctas) {
            if ((rc = grow(d_ghdr, ghdr_cap, pl.ns, "slot headers"))) return rc;
            if ((rc = cuda(cudaMemsetAsync(d_ghdr, 0, size_t(pl.ns) * sizeof(GSlotHeader), st), "memset slots")))
                return rc;
        }
        EngineArgs a = class_args(c);
        const void* fn =
            pl.walker_ctas
                ? (pl.variant == 0   ? (const void*)cmc_engine_split<uint16_t, uint16_t, false>
                   : pl.variant == 1 ? (const void*)cmc_engine_split<uint32_t, uint32_t, false>
                                     : (const void*)cmc_engine_split<uint32_t, uint32_t, true>)
                : engine_kernel(pl.variant, pl.slots_smem, pl.pool_stage != 0);
        void* args[] = {&a};
        // The split engine's producer and walker CTAs hand trials to each other, so
        // they must all be resident at once: a cooperative launch guarantees it.
        if ((rc = cuda(pl.walker_ctas ? cudaLaunchCooperativeKernel(fn, dim3(pl.ctas), dim3(pl.threads),
                                                                     args, pl.smem_bytes, st)
                                      : cudaLaunchKernel(fn, dim3(pl.ctas), dim3(pl.threads), args,
                                                         pl.smem_bytes, st),
                       "engine launch")))
            return rc;
        ++kernels;
    }
    if (!capturing && (rc = cuda(cudaEventRecord(ev_stop, st), "event"))) return rc;
    if (d_out) {
        cmc_compact_failures<<<1, 1024, 0, st>>>(bits, total, value_base, d_out, d_count, out_cap_now,
                                                 nullptr, read_back ? d_result : nullptr, d_ctrl, nclass);
        if ((rc = cuda(cudaGetLastError(), "compaction launch"))) return rc;
        ++kernels;
    }
    last_plan = plans[lp.heaviest];
    ctrl_count = nclass;
    return CMC_OK;
}

// Room for the control blocks and a failure bitmap of `words` words.
int Ctx::bitmap(size_t words) {
    const int rc = grow(d_bits, bits_cap, kCtrlWords + words, "failure bitmap");
    d_ctrl = reinterpret_cast<Ctrl*>(d_bits);
    return rc;
}

int Ctx::check_ctrl() {
    if (!d_ctrl) return CMC_OK;  // no launch since an allocation failed
    Ctrl c[kMaxClasses]{};
    const uint32_t n = std::max<uint32_t>(1, ctrl_count);
    int rc = cuda(cudaMemcpy(c, d_ctrl, n * sizeof(Ctrl), cudaMemcpyDeviceToHost), "read ctrl");
    return rc ? rc : check_ctrl(c);
}

int Ctx::check_ctrl(const Ctrl* c) {
    const uint32_t n = std::max<uint32_t>(1, ctrl_count);
    Ctrl sum{};
    for (uint32_t i = 0; i < n; ++i) {
        if (c[i].error && !sum.error) {
            sum.error = c[i].error;
            sum.where = c[i].where;
        }
        sum.next += c[i].next;
        sum.walks += c[i].walks;
        sum.probes += c[i].probes;
        sum.slot_wait_cycles += c[i].slot_wait_cycles;
        sum.walker_idle_cycles += c[i].walker_idle_cycles;
        sum.walker_cycles += c[i].walker_cycles;
    }
    last_ctrl = sum;
    if (sum.error)
        return fail(-int(sum.error), "%s (site %u): results discarded", ctrl_error_text(sum.error),
                    sum.where);
    return CMC_OK;
}

const void* engine_kernel(int variant, bool smem_slots, bool pooled) {
    if (pooled && smem_slots && variant != 2)
        return variant == 0 ? (const void*)cmc_engine_pooled<uint16_t, uint16_t>
                            : (const void*)cmc_engine_pooled<uint32_t, uint32_t>;
    if (smem_slots)
        return variant == 0   ? (const void*)cmc_engine<uint16_t, uint16_t, false, true>
               : variant == 1 ? (const void*)cmc_engine<uint32_t, uint32_t, false, true>
                              : (const void*)cmc_engine<uint32_t, uint32_t, true, true>;
    return variant == 0   ? (const void*)cmc_engine<uint16_t, uint16_t, false, false>
           : variant == 1 ? (const void*)cmc_engine<uint32_t, uint32_t, false, false>
                          : (const void*)cmc_engine<uint32_t, uint32_t, true, false>;
}

const void* fused_engine_kernel(int variant, bool smem_slots) {
    if (smem_slots)
        return variant == 0   ? (const void*)cmc_engine_fused<uint16_t, uint16_t, false, true>
               : variant == 1 ? (const void*)cmc_engine_fused<uint32_t, uint32_t, false, true>
                              : (const void*)cmc_engine_fused<uint32_t, uint32_t, true, true>;
    return variant == 0   ? (const void*)cmc_engine_fused<uint16_t, uint16_t, false, false>
           : variant == 1 ? (const void*)cmc_engine_fused<uint32_t, uint32_t, false, false>
                          : (const void*)cmc_engine_fused<uint32_t, uint32_t, true, false>;
}

const void* lane_kernel(int variant) {
    return variant == 0   ? (const void*)cmc_lanes<true, false>
           : variant == 1 ? (const void*)cmc_lanes<false, false>
                          : (const void*)cmc_lanes<false, true>;
}

const void* wave_kernel(int variant, bool global_cache) {
    if (variant == 0)
        return global_cache ? (const void*)cmc_waves<true, true> : (const void*)cmc_waves<true, false>;
    return global_cache ? (const void*)cmc_waves<false, true> : (const void*)cmc_waves<false, false>;
}

// Every engine kernel may use up to the device's opt-in shared memory.  Set
// once per device and never lowered, so launches of different plans -- and
// graphs captured from them -- are valid whatever ran in between.
int engine_smem_cap(size_t optin) {
    const void* fns[] = {engine_kernel(0, true), engine_kernel(1, true), engine_kernel(2, true),
                         engine_kernel(0, false), engine_kernel(1, false), engine_kernel(2, false),
                         (const void*)cmc_engine_split<uint16_t, uint16_t, false>,
                         (const void*)cmc_engine_split<uint32_t, uint32_t, false>,
                         (const void*)cmc_engine_split<uint32_t, uint32_t, true>,
                         fused_engine_kernel(0, true), fused_engine_kernel(1, true),
                         fused_engine_kernel(2, true), fused_engine_kernel(0, false),
                         fused_engine_kernel(1, false), fused_engine_kernel(2, false),
                         engine_kernel(0, true, true), engine_kernel(1, true, true),
                         lane_kernel(0), lane_kernel(1), lane_kernel(2),
                         wave_kernel(0, false), wave_kernel(0, true), wave_kernel(1, false), wave_kernel(1, true)};
    for (const void* fn : fns)
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(optin)) != cudaSuccess)
            return CMC_ECUDA;
    return CMC_OK;
}

int Ctx::init(int dev) {
    device = dev;
    int rc = cuda(cudaSetDevice(dev), "cudaSetDevice");
    if (rc) return rc;
    cudaDeviceProp prop{};
    if ((rc = cuda(cudaGetDeviceProperties(&prop, dev), "cudaGetDeviceProperties"))) return rc;
    if (prop.major < 10)
        return fail(CMC_EINVAL, "device %d (%s, sm_%d%d) is not an sm_100 GPU", dev, prop.name,
                    prop.major, prop.minor);
    sms = prop.multiProcessorCount;
    smem_optin = prop.sharedMemPerBlockOptin;
    memory_bytes = prop.totalGlobalMem;
    if (engine_smem_cap(smem_optin)) {
        cudaGetLastError();
        return fail(CMC_ECUDA, "cudaFuncSetAttribute on the engine kernels failed");
    }
    if ((rc = cuda(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "stream"))) return rc;
    if ((rc = cuda(cudaEventCreate(&ev_start), "event"))) return rc;
    if ((rc = cuda(cudaEventCreate(&ev_stop), "event"))) return rc;
    uint32_t t0[256];
    t0_table(t0);
    size_t cap = 0;
    if ((rc = grow(d_t0, cap, 256 + 44 + 32, "tables"))) return rc;
    uint32_t fips[44];
    expand_u64(0x0706050403020100ULL, 0x0f0e0d0c0b0a0908ULL, fips);
    if ((rc = cuda(cudaMemcpy(d_t0, t0, sizeof t0, cudaMemcpyHostToDevice), "upload T0"))) return rc;
    if ((rc = cuda(cudaMemcpy(d_t0 + 256, fips, sizeof fips, cudaMemcpyHostToDevice), "upload KAT key")))
        return rc;
    if ((rc = bitmap(0))) return rc;
    if (cudaHostAlloc((void**)&h_result, sizeof(CallResult), cudaHostAllocMapped) != cudaSuccess ||
        cudaHostGetDevicePointer((void**)&d_result, h_result, 0) != cudaSuccess ||
        cudaHostAlloc((void**)&h_job, sizeof(Job), cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        return fail(CMC_ENOMEM, "pinned call buffers");
    }
    const uint32_t kat_smem = kEngineTableBytes;
    if ((rc = cuda(cudaFuncSetAttribute((const void*)cmc_selftest,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, kat_smem),
                   "selftest attribute")))
        return rc;
    cmc_selftest<<<1, 32, kat_smem, stream>>>(d_t0, d_t0 + 256, d_t0 + 300, 256u);
    if ((rc = cuda(cudaGetLastError(), "selftest launch"))) return rc;
    uint32_t bad[32];
    if ((rc = cuda(cudaMemcpyAsync(bad, d_t0 + 300, sizeof bad, cudaMemcpyDeviceToHost, stream),
                   "selftest read")))
        return rc;
    if ((rc = cuda(cudaStreamSynchronize(stream), "selftest sync"))) return rc;
    for (int i = 0; i < 32; ++i)
        if (bad[i]) return fail(CMC_EKAT, "device AES known-answer test failed (lane %d, flags %u)", i, bad[i]);
    return CMC_OK;
}

Ctx::~Ctx() {
    if (device < 0) return;  // a planner that never touched a device holds nothing to free
    cudaSetDevice(device);
    cudaFree(d_t0);
    cudaFree(d_jobs);
    cudaFree(d_bits);
    cudaFree(d_out);
    cudaFree(d_slots);
    cudaFree(d_ghdr);
    cudaFree(d_job_failed);
    cudaFree(d_key);
    forget_graphs();
    cudaFreeHost(h_failed);
    cudaFreeHost(h_result);
    cudaFreeHost(h_job);
    if (ev_start) cudaEventDestroy(ev_start);
    if (ev_stop) cudaEventDestroy(ev_stop);
    if (stream) cudaStreamDestroy(stream);
}

int Ctx::upload_jobs(const std::vector<Job>& jobs, cudaStream_t st) {
    int rc = grow(d_jobs, jobs_cap, jobs.size(), "job table");
    if (rc) return rc;
    return cuda(cudaMemcpyAsync(d_jobs, jobs.data(), jobs.size() * sizeof(Job),
                                cudaMemcpyHostToDevice, st),
                "upload jobs");
}

int Ctx::launch_host(const cmc_params& p, const uint32_t key[44], uint32_t first, uint32_t count,
                     uint32_t* out, uint32_t* nfailed) {
    kernels = 0;
    if (!key || !out || !nfailed) return fail(CMC_EINVAL, "null argument");
    *nfailed = 0;
    if (count == 0) return CMC_OK;
    if (uint64_t(first) + count > 0x100000000ULL) return fail(CMC_EINVAL, "offset range overflows");
    int rc = cuda(cudaSetDevice(device), "cudaSetDevice");
    if (rc) return rc;
    cudaStream_t st = user_stream ? user_stream : stream;
    look_for_capture(st);
    std::vector<Job> jobs(1);
    if ((rc = make_job(p, first, count, 0, jobs[0]))) return rc;
    std::memcpy(jobs[0].batch_rk, key, 44 * 4);
    if ((rc = grow(d_jobs, jobs_cap, 1, "job table"))) return rc;
    *h_job = jobs[0];
    if ((rc = cuda(cudaMemcpyAsync(d_jobs, h_job, sizeof(Job), cudaMemcpyHostToDevice, st), "upload job"))) return rc;
    if ((rc = grow(d_out, out_cap, size_t(count) + 1, "failure list"))) return rc;
    // one synchronisation: the compaction writes count, control block and the
    // first offsets to host memory (t = 16, 256 trials: three copies and their
    // synchronisations took 20 of a call's 77 us)
    if ((rc = run(jobs, count, st, first, d_out, d_out + count, count, nullptr, nullptr, nullptr, true))) return rc;
    if ((rc = cuda(cudaStreamSynchronize(st), "launch sync"))) return rc;
    if ((rc = check_ctrl(h_result->ctrl))) return rc;
    const uint32_t nf = h_result->count;
    if (nf > count) return fail(CMC_ERANGE, "GPU failure count out of range");
    std::memcpy(out, h_result->offsets, size_t(std::min(nf, kInlineOffsets)) * 4);
    if (nf > kInlineOffsets &&
        (rc = cuda(cudaMemcpy(out + kInlineOffsets, d_out + kInlineOffsets, size_t(nf - kInlineOffsets) * 4,
                              cudaMemcpyDeviceToHost),
                   "read offsets")))
        return rc;
    *nfailed = nf;
    return CMC_OK;
}

int Ctx::launch_device(const cmc_params& p, const uint32_t* d_key_in, uint32_t first,
                       uint32_t count, uint32_t* d_offsets, uint32_t* d_nfailed, cudaStream_t st) {
    kernels = 0;
    if (!d_key_in || !d_offsets || !d_nfailed) return fail(CMC_EINVAL, "null argument");
    if (!st) st = stream;
    int rc = cuda(cudaSetDevice(device), "cudaSetDevice");
    if (rc) return rc;
    if (count == 0) return cuda(cudaMemsetAsync(d_nfailed, 0, 4, st), "memset count");
    look_for_capture(st);
    std::vector<Job> jobs(1);
    if ((rc = make_job(p, first, count, 0, jobs[0]))) return rc;
    if ((rc = upload_jobs(jobs, st))) return rc;
    if ((rc = cuda(cudaMemcpyAsync(d_jobs[0].batch_rk, d_key_in, 44 * 4, cudaMemcpyDeviceToDevice, st),
                   "copy batch key")))
        return rc;
    return run(jobs, count, st, first, d_offsets, d_nfailed, count, nullptr, nullptr);
}

// Plan of a server's launch over `shapes` within `budget` bytes.  Admission,
// size classes and launches plan the same jobs with different counts (trials are
// granted step by step), so a served plan depends on the shapes alone: no split
// for short launches.  A resident launch walks global slots with four isolated
// warps, whose number does not depend on the table size, so that jobs that come
// later fit; where not even one such slot per SM is within the budget it keeps
// the plan of an iteration, unpooled.
int Ctx::plan_served(const std::vector<Job>& shapes, uint64_t budget, bool resident, Plan& pl, uint64_t& pool) {
    const uint64_t was_budget = slot_budget;
    const uint32_t gs = force_global_slots, wk = force_walkers;
    const int iso = force_isolate, wc = force_walker_ctas, fp = force_pool;
    served = true;
    slot_budget = budget;
    const auto measured = [&](int rc) {
        pool = (pl.gslot_bytes + 255) / 256 * 256 + pl.gcache_bytes;
        return rc;
    };
    int rc;
    if (resident) {
        force_global_slots = 1;
        force_isolate = 1;
        force_walkers = 4;
        force_walker_ctas = 0;
        rc = measured(plan(shapes, pl));
        force_global_slots = gs;
        force_walkers = wk;
        force_isolate = iso;
        if (rc == CMC_OK && pool > budget) {
            force_pool = 0;
            rc = measured(plan(shapes, pl));
            force_pool = fp;
        }
        force_walker_ctas = wc;
    } else {
        rc = measured(plan(shapes, pl));
    }
    served = false;
    slot_budget = was_budget;
    return rc;
}

// Estimated AES-block cost of one trial of a job (map build + seeds), used to
// order a batch heaviest first.
double job_cost(const Job& j) {
    const double c = std::ldexp(1.0, 2 * int(j.half_bits)) / double(j.domain);
    const double direct = double(j.pnum) * j.k * 8.0 * c;
    const double build = 8.0 * std::ldexp(1.0, int(j.half_bits));
    const double map = j.method == kMethodCache    ? build + direct / 64.0
                       : j.method == kMethodGCache ? build + direct * 0.3
                                                   : direct;
    return 2.0 + map + 0.1 * j.pnum;
}

std::string Ctx::mix_key(const cmc_job* in, uint32_t n) const {
    std::vector<std::string> parts;
    for (uint32_t i = 0; i < n; ++i) {
        const cmc_params& p = in[i].params;
        char b[96];
        snprintf(b, sizeof b, "%u/%u/%u/%u/%u/%llu", p.mode, p.pnum, p.k, p.buckets, p.half_bits,
                 (unsigned long long)p.domain);
        parts.push_back(b);
    }
    std::sort(parts.begin(), parts.end());
    parts.erase(std::unique(parts.begin(), parts.end()), parts.end());
    std::string key;
    for (auto& x : parts) key += x + ";";
    return key;
}

// Everything a captured batched call bakes in: job shapes and counts in table
// order, plan classes, planner options, the buffers it touches and the sizes of
// those that a replay does not grow first.
std::string Ctx::graph_key(const std::vector<Job>& jobs, const std::vector<uint32_t>& bounds,
                           uint64_t total, uint64_t dev_cap) const {
    std::string key;
    auto add = [&](uint64_t v) {
        key += std::to_string(v);
        key += '/';
    };
    for (const Job& j : jobs)
        for (uint64_t v : {uint64_t(j.mode), uint64_t(j.input_mode), uint64_t(j.pnum), uint64_t(j.k), uint64_t(j.buckets),
                           uint64_t(j.kick), uint64_t(j.half_bits), uint64_t(j.method), j.domain, uint64_t(j.count)})
            add(v);
    key += '|';
    for (uint32_t x : bounds) add(x);
    key += '|';
    for (int64_t v : {int64_t(total), int64_t(dev_cap), int64_t(force_wg), int64_t(force_ng), int64_t(force_global_slots),
                      int64_t(force_walkers), int64_t(max_slots_per_group), int64_t(force_walker_ctas),
                      int64_t(force_isolate), int64_t(force_method), int64_t(spin_limit), int64_t(map_chains),
                      int64_t(fill_blocks), int64_t(use_fused), int64_t(force_lanes), int64_t(force_waves),
                      int64_t(force_pool), int64_t(pool_limit)})
        add(uint64_t(v));
    for (const void* p : {(const void*)d_jobs, (const void*)d_bits, (const void*)d_out, (const void*)d_slots,
                          (const void*)d_job_failed, (const void*)h_failed})
        add(uint64_t(reinterpret_cast<uintptr_t>(p)));
    for (size_t n : {bits_cap, slots_cap}) add(n);
    return key;
}

int Ctx::prepare_jobs(const cmc_job* in, uint32_t n, uint32_t sample_div, std::vector<Job>& out,
                      std::vector<uint32_t>& order, uint64_t& total, std::vector<uint32_t>& bounds) {
    if (!in || n == 0) return fail(CMC_EINVAL, "no jobs");
    std::vector<Job> tmp(n);
    for (uint32_t i = 0; i < n; ++i) {
        uint32_t count = in[i].count;
        if (sample_div > 1) count = std::max<uint32_t>(1, count / sample_div);
        if (count == 0) return fail(CMC_EINVAL, "job %u has no trials", i);
        if (uint64_t(in[i].first) + count > 0x100000000ULL)
            return fail(CMC_EINVAL, "job %u: offset range overflows", i);
        int rc = make_job(in[i].params, in[i].first, count, 0, tmp[i]);
        if (rc) return rc;
        batch_key(in[i].seed, in[i].batch, tmp[i].batch_rk);
        tmp[i].user = i;
    }
    // Plan classes: parameter sets whose own plans agree (slot placement,
    // warps per group, groups, walkers, entry width, cache kind) run under one
    // plan, so a small table never runs under
    // a plan made for a large one.  Classes run heaviest first; within a class, heaviest
    // trials first, so a launch ends on short ones.  Past kMaxClasses
    // signatures the lightest classes share the last launch.
    std::vector<uint32_t> cls(n, 0);
    if (force_walker_ctas <= 0) {
        std::map<std::string, uint32_t> ids;
        std::vector<double> weight;
        std::vector<uint32_t> sig(n);
        for (uint32_t i = 0; i < n; ++i) {
            Plan solo;
            int rc = plan(std::vector<Job>{tmp[i]}, solo);
            if (rc) return rc;
            const char cache = tmp[i].method == kMethodCache ? 's' : tmp[i].method == kMethodGCache ? 'g' : 'd';
            // (splitting classes further, by slot count, measured slower: 12
            // classes on the 64-set sweep gave 1.069 M trials/s against 1.090 M
            // with these 5 -- each class a CTA leaves costs it a walk drain)
            char key[96];
            snprintf(key, sizeof key, "%d/%u/%u/%u/%u/%d/%c", solo.slots_smem ? 1 : 0, solo.wg, solo.ng,
                     solo.nw, solo.isolate, solo.variant, cache);
            auto it = ids.emplace(key, uint32_t(ids.size())).first;
            sig[i] = it->second;
            if (weight.size() <= sig[i]) weight.resize(sig[i] + 1, 0.0);
            weight[sig[i]] += job_cost(tmp[i]) * tmp[i].count;
        }
        std::vector<uint32_t> rank(weight.size());
        for (uint32_t c = 0; c < rank.size(); ++c) rank[c] = c;
        std::stable_sort(rank.begin(), rank.end(), [&](uint32_t a, uint32_t b) { return weight[a] > weight[b]; });
        std::vector<uint32_t> pos(rank.size());
        for (uint32_t r = 0; r < rank.size(); ++r) pos[rank[r]] = std::min<uint32_t>(r, kMaxClasses - 1);
        for (uint32_t i = 0; i < n; ++i) cls[i] = pos[sig[i]];
    }
    order.resize(n);
    for (uint32_t i = 0; i < n; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) {
        return cls[a] != cls[b] ? cls[a] < cls[b] : job_cost(tmp[a]) > job_cost(tmp[b]);
    });
    bounds.assign(1, 0);
    for (uint32_t i = 1; i < n; ++i)
        if (cls[order[i]] != cls[order[i - 1]]) bounds.push_back(i);
    bounds.push_back(n);
    out.resize(n);
    total = 0;
    for (uint32_t i = 0; i < n; ++i) {
        out[i] = tmp[order[i]];
        out[i].trial_base = total;
        total += out[i].count;
    }
    if (total >= 0xffffffffULL) return fail(CMC_EINVAL, "more than 2^32 - 1 trials in one batched call");
    return CMC_OK;
}

namespace {

// Apply a tuned plan for the duration of one call.
struct ScopedPlan {
    Ctx& c;
    uint32_t wg;
    int isolate, method;
    ScopedPlan(Ctx& ctx, const TunedPlan* t) : c(ctx), wg(ctx.force_wg), isolate(ctx.force_isolate),
                                               method(ctx.force_method) {
        if (t) {
            c.force_wg = t->wg;
            c.force_isolate = t->isolate;
            c.force_method = t->method;
        }
    }
    ~ScopedPlan() {
        c.force_wg = wg;
        c.force_isolate = isolate;
        c.force_method = method;
    }
};

}  // namespace

int Ctx::run_jobs(const cmc_job* in, uint32_t n, uint64_t* out_failed, uint32_t* out_offsets,
                  uint32_t* out_jobs, uint64_t cap, uint64_t* out_total) {
    kernels = 0;
    if (!out_failed) return fail(CMC_EINVAL, "null out_failed");
    int rc = cuda(cudaSetDevice(device), "cudaSetDevice");
    if (rc) return rc;
    // a plan tuned at one size is kept for calls up to twice as large
    const auto it = tuned.find(mix_key(in, n));
    uint64_t asked = 0;
    for (uint32_t i = 0; in && i < n; ++i) asked += in[i].count;
    ScopedPlan scoped(*this, it == tuned.end() || asked > 2 * it->second.trials ? nullptr : &it->second);
    std::vector<Job> jobs;
    std::vector<uint32_t> order, bounds;
    uint64_t total = 0;
    if ((rc = prepare_jobs(in, n, 0, jobs, order, total, bounds))) return rc;
    cudaStream_t st = user_stream ? user_stream : stream;
    look_for_capture(st);
    if ((rc = upload_jobs(jobs, st))) return rc;
    if ((rc = grow(d_job_failed, job_failed_cap, n, "job counters"))) return rc;
    const uint64_t dev_cap = out_offsets ? std::min<uint64_t>(cap, total) : 0;
    if ((rc = grow(d_out, out_cap, size_t(dev_cap) + 1, "failure list"))) return rc;
    if (h_failed_cap < n) {
        cudaFreeHost(h_failed);
        h_failed = nullptr;
        h_failed_cap = 0;
        if (cudaHostAlloc((void**)&h_failed, n * sizeof(unsigned long long), cudaHostAllocDefault) !=
            cudaSuccess) {
            cudaGetLastError();
            return fail(CMC_ENOMEM, "pinned job counters");
        }
        h_failed_cap = n;
    }
    // The device side of the call: counters, the engine launches, the
    // compaction and the read-back into pinned memory.
    auto enqueue = [&]() -> int {
        int r = cuda(cudaMemsetAsync(d_job_failed, 0, n * sizeof(unsigned long long), st), "memset counters");
        if (r) return r;
        if ((r = run(jobs, total, st, 0, d_out, d_out + dev_cap, dev_cap, d_job_failed, nullptr, &bounds, true)))
            return r;
        return cuda(cudaMemcpyAsync(h_failed, d_job_failed, n * sizeof(unsigned long long),
                                    cudaMemcpyDeviceToHost, st), "read counters");
    };
    // A call shape seen before is captured into a CUDA graph on its second
    // call and replayed from the third: the job table is uploaded by copy
    // first, everything else is one graph launch.  The first call runs eagerly
    // so that buffers are sized and kernel attributes set before any capture.
    graph_state = "eager";
    if (use_graphs && force_walker_ctas <= 0) {
        const std::string key = graph_key(jobs, bounds, total, dev_cap);
        auto it = std::find_if(graphs.begin(), graphs.end(), [&](const GraphEntry& g) { return g.key == key; });
        if (it != graphs.end()) {
            if ((rc = cuda(cudaEventRecord(ev_start, st), "event"))) return rc;
            if ((rc = cuda(cudaGraphLaunch(it->exec, st), "graph launch"))) return rc;
            if ((rc = cuda(cudaEventRecord(ev_stop, st), "event"))) return rc;
            kernels = it->kernels;
            ctrl_count = it->ctrl_count;
            plan_text = it->plan_text;
            last_plan = it->plan;
            graph_state = "replayed";
        } else if (std::find(graph_seen.begin(), graph_seen.end(), key) != graph_seen.end()) {
            cudaGraph_t g = nullptr;
            capturing = fixed_memory = true;
            rc = cuda(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal), "begin capture");
            if (!rc) rc = enqueue();
            const cudaError_t e = cudaStreamEndCapture(st, &g);
            capturing = fixed_memory = false;
            cudaGraphExec_t ex = nullptr;
            const cudaError_t ie = (!rc && e == cudaSuccess && g) ? cudaGraphInstantiate(&ex, g, 0)
                                                                  : cudaErrorUnknown;
            if (ie == cudaSuccess) {
                if (graphs.size() >= 8) {
                    cudaGraphExecDestroy(graphs.front().exec);
                    graphs.erase(graphs.begin());
                }
                graphs.push_back(GraphEntry{key, ex, kernels, ctrl_count, plan_text, last_plan});
                if (g) cudaGraphDestroy(g);
                if ((rc = cuda(cudaEventRecord(ev_start, st), "event"))) return rc;
                if ((rc = cuda(cudaGraphLaunch(ex, st), "graph launch"))) return rc;
                if ((rc = cuda(cudaEventRecord(ev_stop, st), "event"))) return rc;
                graph_state = "captured";
            } else {
                // the shape could not be captured: run it eagerly
                const std::string why = rc ? err
                                      : std::string(cudaGetErrorName(e != cudaSuccess ? e : ie));
                if (g) cudaGraphDestroy(g);
                cudaGetLastError();
                if ((rc = enqueue())) return rc;
                graph_state = "eager(capture failed: " + why + ")";
            }
        } else {
            if ((rc = enqueue())) return rc;
            // keyed by the buffers as this call left them (it may have grown some)
            graph_seen.push_back(graph_key(jobs, bounds, total, dev_cap));
            if (graph_seen.size() > 64) graph_seen.erase(graph_seen.begin());
        }
    } else if ((rc = enqueue())) {
        return rc;
    }
    if (use_graphs) plan_text += " graph=" + graph_state;
    if ((rc = cuda(cudaStreamSynchronize(st), "batched sync"))) return rc;
    if ((rc = check_ctrl(h_result->ctrl))) return rc;
    std::vector<unsigned long long> failed(h_failed, h_failed + n);
    const uint32_t nf = h_result->count;
    uint64_t sum = 0;
    for (uint32_t i = 0; i < n; ++i) {
        out_failed[order[i]] = failed[i];
        sum += failed[i];
    }
    if (sum != nf) return fail(CMC_ERANGE, "per-job failure counts disagree with the bitmap");
    if (out_total) *out_total = nf;
    if (out_offsets && nf) {
        const uint64_t m = std::min<uint64_t>(nf, dev_cap);
        std::vector<uint32_t> g(h_result->offsets, h_result->offsets + std::min<uint64_t>(m, kInlineOffsets));
        if (m > kInlineOffsets) {
            g.resize(m);
            if ((rc = cuda(cudaMemcpy(g.data(), d_out, m * 4, cudaMemcpyDeviceToHost), "read failures"))) return rc;
        }
        // global index -> (original job, offset); global order is job-major in
        // the heavy-first order, so regroup by the caller's job order
        std::vector<std::pair<uint32_t, uint32_t>> pairs(m);
        for (uint64_t i = 0; i < m; ++i) {
            uint32_t lo = 0, hi = n;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) / 2;
                if (jobs[mid].trial_base <= g[i]) lo = mid; else hi = mid;
            }
            pairs[i] = {order[lo], jobs[lo].first + uint32_t(g[i] - jobs[lo].trial_base)};
        }
        std::sort(pairs.begin(), pairs.end());
        for (uint64_t i = 0; i < m; ++i) {
            out_offsets[i] = pairs[i].second;
            if (out_jobs) out_jobs[i] = pairs[i].first;
        }
    }
    return CMC_OK;
}

int Ctx::autotune(const cmc_job* in, uint32_t n, uint32_t sample_div) {
    int rc = cuda(cudaSetDevice(device), "cudaSetDevice");
    if (rc) return rc;
    cudaStream_t st = user_stream ? user_stream : stream;
    look_for_capture(st);
    if (!sample_div) sample_div = 64;
    std::vector<Job> jobs;
    std::vector<uint32_t> order, bounds;
    uint64_t total = 0;
    // device time of a call under t; CMC_EINVAL and CMC_ENOMEM: it does not fit
    auto time_call = [&](const TunedPlan& t, uint32_t div, double& ms) -> int {
        ScopedPlan scoped(*this, &t);
        int r = prepare_jobs(in, n, div, jobs, order, total, bounds);
        if (r || (r = upload_jobs(jobs, st))) return r;
        if ((r = run(jobs, total, st, 0, nullptr, nullptr, 0, d_job_failed, nullptr, &bounds))) return r;
        float f = 0;
        if ((r = cuda(cudaEventSynchronize(ev_stop), "tune sync"))) return r;
        if ((r = cuda(cudaEventElapsedTime(&f, ev_start, ev_stop), "tune time"))) return r;
        ms = f;
        return check_ctrl();
    };
    if ((rc = prepare_jobs(in, n, sample_div, jobs, order, total, bounds))) return rc;
    if ((rc = grow(d_job_failed, job_failed_cap, n, "job counters"))) return rc;
    bool any_cached = false;  // does the automatic choice use a round cache anywhere?
    for (const Job& j : jobs) any_cached = any_cached || j.method != kMethodDirect;
    std::vector<TunedPlan> cands{TunedPlan{0, -1, -1}};  // each class under its automatic plan
    for (int iso : {0, 1})
        for (uint32_t wg : {1u, 2u, 4u, 6u})
            for (int method : {-1, 0}) {
                if (method == 0 && !any_cached) continue;  // auto already picks direct
                cands.push_back(TunedPlan{wg, iso, method});
            }
    double best_ms = 1e300;
    TunedPlan best{};
    std::string best_text;
    uint64_t sampled = 0;
    for (const TunedPlan& t : cands) {
        double ms = 0;
        rc = time_call(t, sample_div, ms);
        if (rc == CMC_EINVAL || rc == CMC_ENOMEM) continue;  // skip the candidate
        if (rc) return rc;
        if (ms < best_ms) {
            best_ms = ms;
            best = t;
            best_text = plan_text;
            sampled = total;
        }
    }
    if (best_ms == 1e300) return fail(CMC_EINVAL, "no candidate plan fits this mix");
    // A sample may be a short launch where the call is not: the engines and the
    // splits of the automatic plan depend on the counts, a forced plan does not,
    // and it rules the lane and wave engines out.  So the sample's winner has to
    // win at the call's counts too (64 sets of 65,536 trials, sample 1/16: forced
    // plans won the sample, and ran at 1.30 M trials/s against 1.97 M).
    if (best.wg && sample_div > 1) {
        const TunedPlan forced = best;
        double with = 1e300, without = 1e300;
        rc = time_call(TunedPlan{}, 1, without);
        const std::string text = plan_text;
        if (rc && rc != CMC_ENOMEM) return rc;
        rc = time_call(forced, 1, with);
        if (rc && rc != CMC_ENOMEM && rc != CMC_EINVAL) return rc;
        if (rc || with > 0.97 * without) best = TunedPlan{};
        best_text = best.wg ? plan_text : text;
        best_ms = best.wg ? with : without;
        sampled = total;
    }
    best.trials = 0;
    for (uint32_t i = 0; i < n; ++i) best.trials += in[i].count;
    tuned[mix_key(in, n)] = best;
    char buf[96];
    snprintf(buf, sizeof buf, " | %.3f ms for %llu trials", best_ms, (unsigned long long)sampled);
    tune_text = best_text + buf;
    return CMC_OK;
}

}  // namespace cmc

using cmc::Ctx;

extern "C" {

int cmc_init(int device, cmc_ctx** out) {
    if (!out) return CMC_EINVAL;
    *out = nullptr;
    Ctx* c = new (std::nothrow) Ctx();
    if (!c) return CMC_ENOMEM;
    const int rc = c->init(device);
    if (rc) {
        cmc::g_thread_error = c->err;
        delete c;
        return rc;
    }
    *out = reinterpret_cast<cmc_ctx*>(c);
    return CMC_OK;
}

int cmc_destroy(cmc_ctx* ctx) {
    delete reinterpret_cast<Ctx*>(ctx);
    return CMC_OK;
}

const char* cmc_last_error(const cmc_ctx* ctx) {
    if (!ctx) return cmc::g_thread_error.c_str();
    return reinterpret_cast<const Ctx*>(ctx)->err.c_str();
}

int cmc_launch(cmc_ctx* ctx, const cmc_params* params, const uint32_t batch_key[44],
               uint32_t first, uint32_t count, uint32_t* out_offsets, uint32_t* out_nfailed) {
    if (!ctx || !params) return CMC_EINVAL;
    return reinterpret_cast<Ctx*>(ctx)->launch_host(*params, batch_key, first, count, out_offsets,
                                                     out_nfailed);
}

int cmc_launch_device(cmc_ctx* ctx, const cmc_params* params, const uint32_t* d_batch_key,
                      uint32_t first, uint32_t count, uint32_t* d_out_offsets,
                      uint32_t* d_out_nfailed, void* stream) {
    if (!ctx || !params) return CMC_EINVAL;
    return reinterpret_cast<Ctx*>(ctx)->launch_device(*params, d_batch_key, first, count,
                                                       d_out_offsets, d_out_nfailed,
                                                       static_cast<cudaStream_t>(stream));
}

int cmc_check(cmc_ctx* ctx) {
    if (!ctx) return CMC_EINVAL;
    Ctx* c = reinterpret_cast<Ctx*>(ctx);
    int rc = c->cuda(cudaDeviceSynchronize(), "synchronize");
    if (rc) return rc;
    return c->check_ctrl();
}

int cmc_run_jobs(cmc_ctx* ctx, const cmc_job* jobs, uint32_t njobs, uint64_t* out_failed,
                 uint32_t* out_offsets, uint32_t* out_jobs, uint64_t cap, uint64_t* out_total) {
    if (!ctx) return CMC_EINVAL;
    return reinterpret_cast<Ctx*>(ctx)->run_jobs(jobs, njobs, out_failed, out_offsets, out_jobs, cap,
                                                  out_total);
}

int cmc_autotune(cmc_ctx* ctx, const cmc_job* jobs, uint32_t njobs, uint32_t sample_div,
                 const char** out_choice) {
    if (!ctx) return CMC_EINVAL;
    Ctx* c = reinterpret_cast<Ctx*>(ctx);
    const int rc = c->autotune(jobs, njobs, sample_div);
    if (out_choice) *out_choice = c->tune_text.c_str();
    return rc;
}

int cmc_set_option(cmc_ctx* ctx, const char* name, int64_t value) {
    if (!ctx || !name) return CMC_EINVAL;
    Ctx* c = reinterpret_cast<Ctx*>(ctx);
    const std::string n(name);
    if (n == "warps_per_group" && value >= 0 && value <= 15) c->force_wg = uint32_t(value);
    else if (n == "groups" && value >= 0 && value <= cmc::kMaxGroups) c->force_ng = uint32_t(value);
    else if (n == "global_slots" && (value == 0 || value == 1)) c->force_global_slots = uint32_t(value);
    else if (n == "method" && value >= -1 && value <= 2) c->force_method = int(value);
    else if (n == "lanes" && value >= -1 && value <= int64_t(cmc::kMaxLaneWarps)) c->force_lanes = int(value);
    else if (n == "waves" && (value == -1 || value == 0 || value == 1 || value == 2 || value == 4 || value == 8))
        c->force_waves = int(value);
    else if (n == "pool" && value >= -1 && value <= 1) c->force_pool = int(value);
    else if (n == "graph" && (value == 0 || value == 1)) c->use_graphs = int(value);
    else if (n == "fused" && (value == 0 || value == 1)) c->use_fused = int(value);
    else if (n == "fill_blocks" && (value == 0 || (value >= 2 && value <= 4))) c->fill_blocks = uint32_t(value);
    else if (n == "map_chains" && (value == 0 || value == 1 || value == 2 || value == 4 || value == 8))
        c->map_chains = uint32_t(value);
    else if (n == "walkers" && value >= 0 && value <= 4) c->force_walkers = uint32_t(value);
    else if (n == "isolate_walkers" && value >= -1 && value <= 1) c->force_isolate = int(value);
    else if (n == "walker_ctas" && value >= -1 && value < c->sms) c->force_walker_ctas = int(value);
    else if (n == "slots_per_group" && value >= 0 && value <= 32)
        c->max_slots_per_group = value ? uint32_t(value) : 8u;
    else if (n == "pool_bytes" && value >= 0) {
        c->pool_limit = value ? uint64_t(value) : ~0ull;
        if (c->slots_cap > c->pool_limit) {
            cudaSetDevice(c->device);
            c->memory.release(c->d_slots);  // waits for the work that uses it
            c->d_slots = nullptr;
            c->slots_cap = 0;
            c->forget_graphs();
        }
    }
    else if (n == "spin_limit" && value >= 0 && value <= 0xffffffffLL)
        c->spin_limit = value ? uint32_t(value) : (1u << 26);
    else return c->fail(CMC_EINVAL, "unknown option or value out of range: %s=%lld", name, (long long)value);
    return CMC_OK;
}

int cmc_set_stream(cmc_ctx* ctx, void* stream) {
    if (!ctx) return CMC_EINVAL;
    reinterpret_cast<Ctx*>(ctx)->user_stream = static_cast<cudaStream_t>(stream);
    return CMC_OK;
}

double cmc_last_engine_ms(cmc_ctx* ctx) {
    if (!ctx) return -1.0;
    Ctx* c = reinterpret_cast<Ctx*>(ctx);
    if (c->kernels == 0) return -1.0;
    float ms = 0.f;
    // a failure here must not stay pending for the next launch's error check
    if (cudaEventSynchronize(c->ev_stop) != cudaSuccess ||
        cudaEventElapsedTime(&ms, c->ev_start, c->ev_stop) != cudaSuccess) {
        cudaGetLastError();
        return -1.0;
    }
    return ms;
}

int cmc_last_stats(cmc_ctx* ctx, uint64_t out[6]) {
    if (!ctx || !out) return CMC_EINVAL;
    Ctx* c = reinterpret_cast<Ctx*>(ctx);
    const cmc::Ctrl& s = c->last_ctrl;
    out[0] = s.walks;
    out[1] = s.probes;
    out[2] = s.slot_wait_cycles;
    out[3] = s.walker_idle_cycles;
    out[4] = s.walker_cycles;
    out[5] = s.error;
    return CMC_OK;
}

uint32_t cmc_last_kernel_count(const cmc_ctx* ctx) {
    return ctx ? reinterpret_cast<const Ctx*>(ctx)->kernels : 0;
}

int cmc_plan_describe(const cmc_params* params, uint32_t count, uint32_t sms, uint64_t smem_optin,
                      char* out, uint32_t cap) {
    if (!params || !out || cap == 0 || count == 0 || sms == 0 ||
        smem_optin < uint64_t(cmc::kEngineTableBytes) + cmc::kCtaSharedBytes + cmc::kGroupHeaderBytes) {
        cmc::set_thread_error("cmc_plan_describe: invalid argument");
        return CMC_EINVAL;
    }
    Ctx c;  // planner only: no device is selected and nothing is allocated
    c.sms = int(sms);
    c.smem_optin = size_t(smem_optin);
    std::vector<cmc::Job> jobs(1);
    int rc = c.make_job(*params, 0, count, 0, jobs[0]);
    cmc::Plan pl;
    if (!rc) rc = c.plan(jobs, pl);
    if (!rc) {
        cmc::LanePlan lanes;
        cmc::WavePlan waves;
        c.choose_engine(jobs, pl, lanes, waves);
        c.plan_text += cmc::lanes_text(lanes) + cmc::waves_text(waves);
    }
    snprintf(out, cap, "%s", (rc ? c.err : c.plan_text).c_str());
    if (rc) cmc::set_thread_error(c.err);
    return rc;
}

const char* cmc_last_plan(const cmc_ctx* ctx) {
    return ctx ? reinterpret_cast<const Ctx*>(ctx)->plan_text.c_str() : "";
}

}  // extern "C"
