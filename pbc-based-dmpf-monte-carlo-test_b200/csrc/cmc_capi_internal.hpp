// cmc_capi_internal.hpp -- the context behind the opaque cmc_ctx handle.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <string>
#include <vector>

#include "cmc.h"
#include "cmc_engine.cuh"

namespace cmc {

constexpr uint32_t kMaxClasses = 16;  // plan classes per batched call
static_assert(kMaxClasses <= kMaxFusedClasses, "every class fits a fused launch");

constexpr uint32_t kCtrlWords = 320;  // room for kMaxClasses control blocks
static_assert(kMaxClasses * sizeof(Ctrl) <= kCtrlWords * 4, "control blocks fit their room");
static_assert(kMaxClasses <= kResultCtrls, "a result holds every class's control block");

struct Plan {
    uint32_t ng = 0, wg = 0, ns = 0, nw = 1;
    uint32_t walker_ctas = 0;  // > 0: split engine with this many walker CTAs
    uint32_t isolate = 0;      // walker warps alone on SM sub-partition 3
    bool slots_smem = true;
    uint32_t slot_stride = 0, bins_bytes = 0, group_bytes = 0;
    uint32_t group_off = 0, slots_off = 0, smem_bytes = 0, threads = 0, ctas = 0;
    int variant = 0;  // 0: u16 map/bins, 1: u32 map/bins, 2: u32 + 64-bit PRP domain
    // What a server counts for this plan: its walk slots at full number and, for
    // 16-bit tables, without their items' buckets, and its round caches.
    uint64_t claim_bytes = 0;
    bool reduced = false;         // fewer walk slots than planned: Ctx::slot_budget
    uint64_t gslot_bytes = 0;     // global walk slots (0: slots in shared memory)
    uint32_t gcache_stride = 0;   // u16 entries per group's global round cache
    uint64_t gcache_bytes = 0;    // all groups' global round caches
    uint32_t pool_stage = 0;      // pooled direct passes: bytes per staging map (0: off)
    uint32_t pool_fold = 0;       // pooled direct passes: bytes per fold table (0: unfolded)
};

// How a launch runs in the lane engine (cmc_lanes.cu).
struct LanePlan {
    uint32_t warps = 0;         // per CTA (0: the group engine runs the launch)
    uint32_t share = 32;        // lanes per warp that take trials
    uint32_t ctas = 0, smem_bytes = 0;
    int variant = 0;            // as Plan::variant
    uint64_t region_bytes = 0;  // per lane
    uint64_t regions_bytes = 0, stock_bytes = 0;
    double cycles = 0;          // estimated
};

// How a launch runs in the wave engine (cmc_waves.cu).
struct WavePlan {
    uint32_t ng = 0, wg = 0;    // groups per CTA (0: not used), warps per group
    uint32_t wave = 0, min_wave = 1;  // trials per wave and group
    uint32_t ctas = 0, smem_bytes = 0, group_bytes = 0, cache_off = 0, map_off = 0;
    int variant = 0;            // as Plan::variant
    bool global_cache = false;
    uint32_t gcache_stride = 0;
    uint64_t region_bytes = 0;  // per trial of a wave
    uint64_t regions_bytes = 0, stock_bytes = 0, gcache_bytes = 0;
    double cycles = 0;          // estimated
};

// How a call runs: its plan classes, the kernels they run in (more than one
// class: a fused kernel) and their places in the context's pool.
struct LaunchPlan {
    std::vector<Plan> plans;
    std::vector<LanePlan> lanes;
    std::vector<WavePlan> waves;
    std::vector<double> work, trials;  // per class: AES blocks, trials
    std::vector<std::vector<uint32_t>> kernels;
    std::vector<uint64_t> region;
    uint64_t pool = 0;
    uint32_t heaviest = 0;
    std::string text;

    uint64_t pool_bytes(uint32_t c) const {
        const auto whole = [](uint64_t n) { return (n + 255) / 256 * 256; };
        if (waves[c].ng) return whole(waves[c].regions_bytes) + waves[c].stock_bytes + whole(waves[c].gcache_bytes);
        if (lanes[c].warps) return whole(lanes[c].regions_bytes) + lanes[c].stock_bytes;
        return whole(plans[c].gslot_bytes) + whole(plans[c].gcache_bytes);
    }
};

uint32_t choose_method(uint32_t h, uint64_t domain, double candidates, int force, bool may_allocate);
// Raises the engine kernels' dynamic shared-memory limit to the device's opt-in maximum.
int engine_smem_cap(size_t optin);
// The engine kernel for a plan's entry width (Plan::variant) and walk-slot
// placement, and the fused kernel of the same kind.
const void* engine_kernel(int variant, bool smem_slots, bool pooled = false);
const void* fused_engine_kernel(int variant, bool smem_slots);
const void* lane_kernel(int variant);
const void* wave_kernel(int variant, bool global_cache);
// Estimated cost of one trial in AES-block equivalents (seeds, map, 0.1 t for the walk).
double job_cost(const Job& j);

// The device-memory calls of a context's buffers (a test puts its own here).
struct DeviceMemory {
    cudaError_t (*alloc)(void**, size_t) = [](void** p, size_t n) { return cudaMalloc(p, n); };
    cudaError_t (*release)(void*) = [](void* p) { return cudaFree(p); };
    cudaError_t (*available)(size_t*) = [](size_t* n) {
        size_t all = 0;
        return cudaMemGetInfo(n, &all);
    };
};

// Planner options chosen by the autotuner for one mix of parameter sets.
struct TunedPlan {
    uint32_t wg = 0;
    int isolate = -1;
    int method = -1;
    uint64_t trials = 0;  // of the call it was tuned for
};

struct Ctx {
    int device = -1;
    int sms = 0;
    size_t smem_optin = 0;
    uint64_t memory_bytes = 180ull << 30;  // device memory (the planner's default: B200)
    cudaStream_t stream = nullptr;       // the context's own stream
    cudaStream_t user_stream = nullptr;  // cmc_set_stream override
    cudaEvent_t ev_start = nullptr, ev_stop = nullptr;
    uint32_t* d_t0 = nullptr;  // T0 table, FIPS KAT schedule, self-test output
    Ctrl* d_ctrl = nullptr;      // one control block per plan class of a launch, at the head of d_bits
    uint32_t ctrl_count = 1;     // control blocks the last run used
    Job* d_jobs = nullptr;
    size_t jobs_cap = 0;
    uint32_t* d_bits = nullptr;  // kCtrlWords of control blocks, then the failure bitmap
    size_t bits_cap = 0;
    CallResult* h_result = nullptr;  // mapped host memory: what a synchronous call reads back
    CallResult* d_result = nullptr;  // its device address
    Job* h_job = nullptr;            // pinned staging of cmc_launch's one job
    uint32_t* d_out = nullptr;
    size_t out_cap = 0;
    char* d_slots = nullptr;
    size_t slots_cap = 0;
    GSlotHeader* d_ghdr = nullptr;
    size_t ghdr_cap = 0;
    uint32_t* d_key = nullptr;
    unsigned long long* d_job_failed = nullptr;
    size_t job_failed_cap = 0;
    std::map<std::string, TunedPlan> tuned;  // autotuner results by job mix
    std::string tune_text;
    std::string err, plan_text;
    uint32_t kernels = 0;
    Plan last_plan;
    LaunchPlan call_plan;  // of the last call: keeps its vectors' memory for the next
    Ctrl last_ctrl{};
    // tuning overrides (0 = automatic)
    uint32_t force_wg = 0, force_ng = 0, force_global_slots = 0, force_walkers = 0;
    uint32_t max_slots_per_group = 8;
    int force_walker_ctas = -1;  // -1 auto, 0 in-SM walker, N split engine
    int force_isolate = -1;      // -1 auto, 0 contiguous warp roles, 1 isolated walkers
    // batched calls: captured CUDA graphs of the device side, by call shape
    struct GraphEntry {
        std::string key;
        cudaGraphExec_t exec = nullptr;
        uint32_t kernels = 0, ctrl_count = 1;
        std::string plan_text;
        Plan plan;
    };
    int use_graphs = 1;
    int use_fused = 1;  // batched calls: all plan classes in one persistent launch
    bool capturing = false;
    DeviceMemory memory;
    bool fixed_memory = false;  // a stream capture is under way: no buffer is allocated or freed
    std::vector<GraphEntry> graphs;  // most recent last, at most 8
    std::vector<std::string> graph_seen;
    unsigned long long* h_failed = nullptr;  // pinned per-job counts of the last batched call
    size_t h_failed_cap = 0;
    std::string graph_state;                 // "eager", "captured" or "replayed"
    int force_method = -1;  // -1 auto, 0 direct, 1 cache (shared if h <= 12, else global), 2 global cache
    int force_lanes = -1;   // lane engine: -1 auto, 0 off, N warps per CTA
    int force_waves = -1;   // wave engine: -1 auto, 0 off, N groups per CTA
    int force_pool = -1;    // pooled direct passes: -1 auto, 0 off, 1 on where they apply
    bool plan_no_dfold = false;  // plan() re-run without room for direct passes' fold tables
    uint64_t slot_budget = ~0ull;  // bytes for global walk slots and round caches
    uint64_t pool_limit = ~0ull;   // bytes the pool may take (option pool_bytes)
    uint64_t refused = 0, refused_room = 0;  // a pool the device did not have, and the room it had then
    bool group_engine = false;     // no lanes or waves: the call is short of memory
    bool served = false;       // planning a server's launch (plan_served)
    bool may_allocate = true;  // false: no global round cache, global slots only if unavoidable
    uint32_t spin_limit = 1u << 26;
    uint32_t map_chains = 0;  // lookup chains per lane from a round cache (0: automatic)
    uint32_t fill_blocks = 0; // round-cache fill: independent blocks per thread and step (0: automatic)

    ~Ctx();
    int init(int dev);
    int fail(int code, const char* fmt, ...);
    int cuda(cudaError_t e, const char* what);
    int grow_bytes(void*& ptr, size_t& cap, size_t need, size_t size, const char* what);
    void forget_graphs();
    void look_for_capture(cudaStream_t st);
    template <typename T>
    int grow(T*& ptr, size_t& cap, size_t need, const char* what);
    int make_job(const cmc_params& p, uint32_t first, uint32_t count, uint64_t base, Job& j);
    int plan(const std::vector<Job>& jobs, Plan& pl);
    int plan_served(const std::vector<Job>& shapes, uint64_t budget, bool resident, Plan& pl, uint64_t& pool);
    LanePlan plan_lanes(const std::vector<Job>& jobs, const Plan& group) const;
    WavePlan plan_waves(const std::vector<Job>& jobs, const Plan& group) const;
    void choose_engine(const std::vector<Job>& jobs, const Plan& group, LanePlan& lanes, WavePlan& waves) const;
    int plan_launch(const std::vector<Job>& jobs, const std::vector<uint32_t>& bounds, LaunchPlan& lp);
    int reserve_pool(uint64_t n);
    int fit_launch(const std::vector<Job>& jobs, const std::vector<uint32_t>& bounds, LaunchPlan& lp);
    int upload_jobs(const std::vector<Job>& jobs, cudaStream_t st);
    int run(const std::vector<Job>& jobs, uint64_t total, cudaStream_t st, uint32_t value_base,
            uint32_t* d_out, uint32_t* d_count, uint64_t out_cap, unsigned long long* job_failed,
            unsigned long long* job_done, const std::vector<uint32_t>* class_bounds = nullptr,
            bool read_back = false);
    int check_ctrl();
    int check_ctrl(const Ctrl* blocks);
    int bitmap(size_t words);
    int launch_host(const cmc_params& p, const uint32_t key[44], uint32_t first, uint32_t count,
                    uint32_t* out, uint32_t* nfailed);
    int launch_device(const cmc_params& p, const uint32_t* d_key, uint32_t first, uint32_t count,
                      uint32_t* d_offsets, uint32_t* d_nfailed, cudaStream_t st);
    int prepare_jobs(const cmc_job* in, uint32_t n, uint32_t sample_div, std::vector<Job>& out,
                     std::vector<uint32_t>& order, uint64_t& total, std::vector<uint32_t>& bounds);
    std::string mix_key(const cmc_job* in, uint32_t n) const;
    std::string graph_key(const std::vector<Job>& jobs, const std::vector<uint32_t>& bounds,
                          uint64_t total, uint64_t dev_cap) const;
    int run_jobs(const cmc_job* in, uint32_t n, uint64_t* out_failed, uint32_t* out_offsets,
                 uint32_t* out_jobs, uint64_t cap, uint64_t* out_total);
    int autotune(const cmc_job* in, uint32_t n, uint32_t sample_div);
};

}  // namespace cmc
