// cmc_waves.cuh -- data shared by the wave engine (cmc_waves.cu) and its planner.
#pragma once
#include <cstdint>

#include "cmc_engine.cuh"

namespace cmc {

// A group's shared region: [two set-up records, kWaveHeaderBytes][fold table]
// [round cache, when it is kept in shared memory].
constexpr uint32_t kWaveHeaderBytes = 1024;

struct WaveArgs {
    const Job* jobs;
    uint32_t njobs;
    uint64_t total;                  // the launch runs global trials [gidx_begin, total)
    uint64_t gidx_begin;
    Ctrl* ctrl;
    uint32_t* fail_bits;             // bit g = global trial g failed
    unsigned long long* job_failed;  // per job (optional)
    const uint32_t* t0;              // 256-word T0 table in global memory
    char* regions;                   // per group `wave` regions: [B table entries][t items' buckets]
    uint64_t region_bytes;
    uint32_t map_off;                // the buckets start this far into a region
    uint32_t wave, min_wave;         // trials per wave and group: at most (<= a group's threads), at least
    uint32_t* stock;                 // kRecordBlockBytes per warp
    uint16_t* gcache;                // global round caches, one per group (nullptr: shared memory)
    uint32_t gcache_stride;          // entries
    uint32_t ng, wg;                 // groups per CTA, warps per group
    uint32_t group_bytes, cache_off;
};

}  // namespace cmc
