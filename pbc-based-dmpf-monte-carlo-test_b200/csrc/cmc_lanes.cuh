// cmc_lanes.cuh -- data shared by the lane engine (cmc_lanes.cu) and its planner.
#pragma once
#include <cstdint>

#include "cmc_engine.cuh"

namespace cmc {

constexpr uint32_t kLaneTableBytes = 2 * kEngineTableBytes;  // T0/T2 rows, then T1/T3 rows
constexpr uint32_t kLaneFoldBytes = 8 * 32 * 16;             // per warp: 8 Feistel rounds x 32 lanes x 16 B
constexpr uint32_t kMaxLaneWarps = 16;
// Table reads per pass before a lane on known buckets sits one out: measured
// at t = 64, 2^20 trials 20.5, 19.2, 19.0 and 19.1 ms with 1, 2, 4 and 8.
constexpr uint32_t kLaneHops = 4;

struct LaneArgs {
    const Job* jobs;
    uint32_t njobs;
    uint64_t total;                  // the launch runs global trials [gidx_begin, total)
    uint64_t gidx_begin;
    Ctrl* ctrl;
    uint32_t* fail_bits;             // bit g = global trial g failed
    unsigned long long* job_failed;  // per job (optional)
    const uint32_t* t0;              // 256-word T0 table in global memory
    char* regions;                   // one table of B entries per lane that takes trials
    uint64_t region_bytes;
    uint32_t hops;                   // table reads per pass before a lane sits one out
    uint32_t* stock;                 // kRecordBlockBytes per warp
    uint32_t share;                  // lanes per warp that take trials (<= 32)
};

}  // namespace cmc
