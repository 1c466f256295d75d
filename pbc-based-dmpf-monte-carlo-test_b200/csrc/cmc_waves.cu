// cmc_waves.cu -- the wave engine: groups of warps build the bucket maps of a
// wave of trials from round caches, then walk the wave one trial per thread.
//
// For shapes whose round cache (8 * 2^h AES blocks) costs less than evaluating
// buckets one by one.  The group engine (cmc_engine.cu) gives walks of their
// own warps 10 to 128 lanes per SM; here every thread of a group walks a trial
// of the wave, and the SM's other groups fill round caches meanwhile.  A walk
// step waits for one table read: an entry holds its item's other buckets
// (Item in cmc_trial.cuh), so an evicted item's next bin is known at once.
//
// Fill: shared-memory lookups bound it, 106 per block for AES rounds 3..10 of
// the two-table form, one wavefront of 32 lanes per clock and SM.  The state
// after round 2 separates: with R = y << 8 | x it is U(x) ^ F(r, y), where U
// reads byte 0 of R ^ rk3 through state word 0 (the same for all Feistel rounds
// r, which enter state word 2 alone), so a thread keeps one x and its U in
// registers and runs over all (r, y): one broadcast 16-byte load of F instead
// of 16 lookups for rounds 1 and 2.
#include <cstdint>

#include "cmc_trial.cuh"
#include "cmc_waves.cuh"

namespace cmc {

namespace {

using T2 = Te<false>;

struct WaveHeader {
    uint32_t rec[2][kRecordWords];
    unsigned long long base;
    uint32_t n;
};
static_assert(sizeof(WaveHeader) <= kWaveHeaderBytes, "the planner reserves kWaveHeaderBytes");

__device__ __forceinline__ void wave_sync(uint32_t g, uint32_t nthreads) {
    asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(nthreads) : "memory");
}

// Stores of the fill loop as PTX: plain stores into the array that also holds
// the T-table cost an address instruction per table lookup (cmc_engine.cu).
__device__ __forceinline__ void st_cache_shared(uint32_t addr, uint32_t v) {
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"((unsigned short)v) : "memory");
}

__device__ __forceinline__ void st_cache_global(uint16_t* p, uint32_t v) {
    asm volatile("st.global.u16 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "h"((unsigned short)v) : "memory");
}

__device__ __forceinline__ uint4 lds_fold(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(addr));
    return v;
}

// U(x): the round-2 lookups that read state word 0; w has x ^ rk3 in byte 0.
__device__ __forceinline__ uint4 wave_u(const Lanes& L, uint32_t c0, uint32_t w) {
    const uint32_t a = c0 ^ T2::e3<0>(L, w);
    return make_uint4(T2::e0<3>(L, a), T2::e3<0>(L, a), T2::e2<1>(L, a), T2::e1<2>(L, a));
}

// Round cache entries (r << h) | R = F_r(R) & mask; of round 7 those that the
// buckets need (Job::last_rows; t = 1024, N = 2^20: 9 % of all blocks less).
template <bool GC>
__device__ __forceinline__ void wave_fill(const Lanes& L, const PrpKey& key, const Job& J, uint32_t c0, uint32_t k3,
                                          uint32_t fold, uint16_t* cache, uint32_t h, uint32_t mask,
                                          uint32_t gt, uint32_t nt) {
    const uint32_t cbase = GC ? 0 : (uint32_t)__cvta_generic_to_shared(cache);
    auto put = [&](uint32_t e, uint32_t v) {
        if constexpr (GC) st_cache_global(cache + e, v);
        else st_cache_shared(cbase + 2 * e, v);
    };
    if (h >= 8) {
        const uint32_t last = 7u << (h - 8), rows = J.last_rows;  // (r, y) pairs of rounds 0..6
        const uint32_t n = (8u << (h - 8)) - rows;
        const uint32_t parts = nt > 256 ? nt / 256 : 1, part = gt >> 8;
        const uint32_t n0 = n * part / parts & ~1u, n1 = part + 1 == parts ? n : n * (part + 1) / parts & ~1u;
        const uint32_t begin = n0 < last ? n0 : n0 + rows, end = n1 > last ? n1 + rows : n1;
        const uint32_t mid = rows && begin < last ? min(n1, last) : end;
        for (uint32_t x = gt & 255u; x < 256; x += nt) {
            const uint4 u = wave_u(L, c0, x ^ k3);
            uint32_t i = begin, stop = mid;
#pragma unroll 1
            for (;;) {  // [begin, mid), then [last + rows, end)
#pragma unroll 1
                for (; i < stop; i += 2) {
                    const uint4 f = lds_fold(fold + 16 * i), g = lds_fold(fold + 16 * i + 16);
                    const uint32_t a = prp_tail(L, key, u.x ^ f.x, u.y ^ f.y, u.z ^ f.z, u.w ^ f.w);
                    const uint32_t b = prp_tail(L, key, u.x ^ g.x, u.y ^ g.y, u.z ^ g.z, u.w ^ g.w);
                    put(256 * i + x, a & mask);
                    put(256 * i + 256 + x, b & mask);
                }
                if (stop == end) break;
                i = last + rows;
                stop = end;
            }
        }
        const uint32_t width = (uint32_t)J.width;
        for (uint32_t m = gt + 1; m <= J.last_cuts; m += nt) {
            const uint32_t at = m * width, R = at >> h;
            if ((at & mask) == 0 || R >= 256 * rows) continue;
            const uint4 u = wave_u(L, c0, (R & 255u) ^ k3), f = lds_fold(fold + 16 * (last + (R >> 8)));
            put((7u << h) + R, prp_tail(L, key, u.x ^ f.x, u.y ^ f.y, u.z ^ f.z, u.w ^ f.w) & mask);
        }
    } else {
        for (uint32_t e = gt; e < 8u << h; e += nt) {
            const uint4 u = wave_u(L, c0, (e & mask) ^ k3), f = lds_fold(fold + 16 * (e >> h));
            put(e, prp_tail(L, key, u.x ^ f.x, u.y ^ f.y, u.z ^ f.z, u.w ^ f.w) & mask);
        }
    }
}

// Buckets of all (item, copy) pairs from a round cache, CH lookup chains per
// lane; a warp runs over its own share of the pairs and a lane takes the next
// pair when its cycle-walk ends.  PART: the cache may hold a part of round 7
// (Job::last_rows).  Returns false if a bucket was out of range.
template <int CH, bool PART, typename MapT>
__device__ __forceinline__ bool wave_map(const Job& J, const uint32_t* rec, const uint16_t* cache, MapT* map,
                                         uint32_t gwi, uint32_t wg, uint32_t lane) {
    const uint32_t k = J.k, ncand = J.pnum * k, h = J.half_bits, mask = (uint32_t)J.mask;
    const uint32_t domain_m1 = (uint32_t)(J.domain - 1), width = (uint32_t)J.width, magic = J.width_magic;
    const uint32_t nbins = J.buckets;
    const bool sequential = J.input_mode == 0, cuts = J.last_cuts != 0;
    const uint32_t whole = J.last_rows ? 2 * (uint32_t)(J.domain >> h) : 0;  // high halves inside the domain
    const uint64_t shift = (uint64_t)rec[kStWalk + 4] | ((uint64_t)rec[kStWalk + 5] << 32);
    const uint64_t step = (uint64_t)rec[kStWalk + 6] | ((uint64_t)rec[kStWalk + 7] << 32);
    const uint64_t rmask = J.range_mask;
    const uint32_t share = (ncand + wg - 1) / wg;
    const uint32_t end = min(ncand, (gwi + 1) * share);
    uint32_t next = min(end, gwi * share);  // warp-uniform
    const unsigned below = (1u << lane) - 1u;
    uint32_t at[CH], l[CH], r[CH];  // halves as byte offsets into the cache, twice their value
    bool has[CH], any = false, ok = true;
    auto take = [&](int i, bool need) {
        const unsigned m = __ballot_sync(kFull, need);
        const uint32_t c = next + __popc(m & below);
        next = min(end, next + __popc(m));
        if (need) {
            has[i] = c < end;
            if (has[i]) {
                const uint32_t o = k == 3 ? __umulhi(c, 0xAAAAAAABu) >> 1 : c >> (k >> 1), j = c - o * k;
                const uint64_t e = sequential ? (uint64_t)o : (shift + (uint64_t)o * step) & rmask;
                const uint32_t y = (uint32_t)(e * k + j);
                at[i] = 4 * o + j;
                l[i] = 2 * (y >> h);
                r[i] = 2 * (y & mask);
            }
        }
    };
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        l[i] = r[i] = at[i] = 0;  // idle chains keep in-range indices
        has[i] = false;
        take(i, true);
        any |= has[i];
    }
    while (__any_sync(kFull, any)) {
#pragma unroll
        for (uint32_t rr = 0; rr < (PART ? 7 : 8); ++rr) {
            const char* round = reinterpret_cast<const char*>(cache) + ((size_t)rr << (h + 1));
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                const uint32_t nr = l[i] ^ 2u * *reinterpret_cast<const uint16_t*>(round + r[i]);
                l[i] = r[i];
                r[i] = nr;
            }
        }
        if constexpr (PART) {
            // The last round, where the bucket does not follow from the high half
            // (with any low half y is then in the domain and in the same bucket).
            const char* round = reinterpret_cast<const char*>(cache) + ((size_t)7 << (h + 1));
            bool decided[CH];
#pragma unroll
            for (int i = 0; i < CH; ++i) decided[i] = r[i] < whole;
            if (cuts) {
#pragma unroll
                for (int i = 0; i < CH; ++i) {
                    const uint32_t y0 = (r[i] >> 1) << h;
                    decided[i] = decided[i] && (div_width(y0, width, magic) + 1) * width - y0 > mask;
                }
            }
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                uint32_t f = 0;
                if (!decided[i]) f = *reinterpret_cast<const uint16_t*>(round + r[i]);
                const uint32_t nr = l[i] ^ 2u * f;
                l[i] = r[i];
                r[i] = nr;
            }
        }
        any = false;
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const uint32_t y = ((l[i] >> 1) << h) | r[i] >> 1;
            const bool done = has[i] && y <= domain_m1;
            if (done) {
                const uint32_t b = div_width(y, width, magic);
                ok = ok && b < nbins;
                __stcg(map + at[i], (MapT)(b < nbins ? b : 0u));
            }
            take(i, done);
            any |= has[i];
        }
    }
    return ok;
}

// The walks of a warp's trials, one per lane (`active`), by the steps of ItemWalk
// (cmc_trial.cuh), which the group engine uses: a change to the rules of a walk
// has to be made in both.  Returns whether this lane's failed.
//
// A step reads one bin per lane, all at the same place of the loop, and its two
// outcomes (item placed, item evicted) are selects, not branches.  A walk alone
// is bound by latency, the table read and the chain of instructions behind it;
// beside other groups' fills by the ALU pipe (79 % of a launch at t = 1024, under
// ncu).  The walk's digits are therefore decoded ahead, for all lanes together,
// and an item that returns to the bin it left costs no read (t = 1024, N = 2^20:
// 250 ALU instructions per step with 64-bit digit divisions and a loop over
// returning items, 3,500 cycles a step with 32 lanes and branches).
template <bool NARROW>
__device__ __forceinline__ bool walk_bgh(const Job& J, bool active, uint64_t walk, uint64_t rnd, char* region,
                                         uint32_t map_off, unsigned long long& probes) {
    // BGH25 random walk (cuckoo_core.hpp:123-133)
    using ItemT = Item<NARROW>;
    using Entry = typename ItemT::Entry;
    Entry* bins = reinterpret_cast<Entry*>(region);
    const Entry* map = reinterpret_cast<const Entry*>(region + map_off);
    const uint32_t k = J.k, last = J.pnum - 1, kick = J.kick;
    const bool four = k == 4;
    uint32_t item = 0, cur = 0, count = 0, which = 0, bin = 0;
    bool failed = false, again = false;
    Digits digits;
    digits.walk = walk;
    digits.rnd = rnd;
    ItemT it{};
    Entry ahead{}, mine{};  // the next item's buckets; what this lane wrote last
    if (active) {
        it = ItemT::from(ItemT::load(map));
        ahead = ItemT::load(map + 1);  // t >= 3
        which = digits.next(k);
        bin = it.get(which);
    }
    for (uint32_t s = 0; __any_sync(kFull, active); ++s) {
        if ((s & 7u) == 0 && active) digits.top_up(k);
        if (!active) continue;
        Entry old = mine;  // an item that returns to the bin it left finds the item that evicted it
        if (!again) old = ItemT::load(bins + bin);
        mine = it.pack(cur, which, four);
        ++probes;
        which = digits.next(k);
        const bool placed = ItemT::empty(old);
        uint32_t copy;
        it.unpack(old, bin, four, cur, copy);
        active = !(placed && item == last);
        item += placed;
        it = placed ? ItemT::from(ahead) : it;
        cur = placed ? item : cur;
        copy = placed ? 4u : copy;
        count = placed ? 0u : count + 1;
        if (placed) ahead = ItemT::load(map + min(item + 1, last));
        failed = count > kick;
        if (which == copy && !failed) {
            ++probes;
            const Entry back = it.pack(cur, which, four);
            it.unpack(mine, bin, four, cur, copy);
            mine = back;
            which = digits.next(k);
            failed = ++count > kick;
        }
        ItemT::store(bins + bin, mine);
        active = active && !failed;
        again = which == copy;
        bin = it.get(which);
    }
    return failed;
}

template <bool NARROW>
__device__ __forceinline__ bool walk_drrt(const Job& J, bool active, char* region, uint32_t map_off,
                                          unsigned long long& probes) {
    // DRRT18 cycling eviction (cuckoo_core.hpp:134-158)
    using ItemT = Item<NARROW>;
    using Entry = typename ItemT::Entry;
    Entry* bins = reinterpret_cast<Entry*>(region);
    const Entry* map = reinterpret_cast<const Entry*>(region + map_off);
    const uint32_t k = J.k, last = J.pnum - 1, kick = J.kick;
    const bool four = k == 4;
    uint32_t item = 0, cur = 0, count = 0, which = 0, bin = 0;
    bool failed = false, evicting = false;
    ItemT it{};
    Entry ahead{};
    if (active) {
        it = ItemT::from(ItemT::load(map));
        ahead = ItemT::load(map + 1);  // t >= 3
        bin = it.get(0);
    }
    while (__any_sync(kFull, active)) {
        if (!active) continue;
        const Entry old = ItemT::load(bins + bin);
        const Entry mine = it.pack(cur, which, four);
        ++probes;
        const bool placed = ItemT::empty(old), evict = evicting && !placed;
        if (placed || (evict && count < kick)) ItemT::store(bins + bin, mine);
        active = !(placed && item == last);
        item += placed;
        failed = evict && count >= kick;
        uint32_t out, copy;  // the item in the bin
        ItemT there = ItemT::from(old);
        there.unpack(old, bin, four, out, copy);
        // an evicted item goes to its next copy in another bin; the copy it sat
        // by is this bin
        uint32_t next = copy + 1 == k ? 0 : copy + 1;
        for (uint32_t tried = 1; evict && there.get(next) == bin; ++tried) {
            if (tried + 1 == k) {
                failed = true;
                break;
            }
            next = next + 1 == k ? 0 : next + 1;
        }
        // a new item tries its copies in order before it evicts
        const bool tried_all = !evicting && which + 1 == k;
        which = placed ? 0u : evict ? next : tried_all ? 0u : which + 1;
        count = evict ? count + 1 : 0u;
        it = placed ? ItemT::from(ahead) : evict ? there : it;
        cur = placed ? item : evict ? out : cur;
        evicting = !placed && (evicting || tried_all);
        if (placed) ahead = ItemT::load(map + min(item + 1, last));
        active = active && !failed;
        bin = it.get(which);
    }
    return failed;
}

}  // namespace

// NARROW: 8-byte table entries, else 16-byte ones (Item in cmc_trial.cuh).  GC:
// round caches in global memory (h <= 16), else in shared memory (h <= 12, or a
// single group's of h = 13).
template <bool NARROW, bool GC>
__global__ void __launch_bounds__(512, 1) cmc_waves(const WaveArgs a) {
    if (!table_base_ok()) {
        if (threadIdx.x == 0) atomicExch(&a.ctrl->error, kErrBase);
        return;
    }
    using ItemT = Item<NARROW>;
    using Entry = typename ItemT::Entry;
    using MapT = typename ItemT::Bucket;
    char* smem = cmc_dyn_smem;
    build_tables<false>(a.t0, smem);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nt = a.wg * 32, g = threadIdx.x / nt, gt = threadIdx.x - g * nt;
    const Lanes L{lane * 4, lane * 4 + 128, 256u};
    const uint32_t group = blockIdx.x * a.ng + g;
    char* gbase = smem + kEngineTableBytes + g * a.group_bytes;
    WaveHeader* hd = reinterpret_cast<WaveHeader*>(gbase);
    const uint32_t fold = (uint32_t)__cvta_generic_to_shared(gbase + kWaveHeaderBytes);
    uint16_t* cache = GC ? a.gcache + (size_t)group * a.gcache_stride : reinterpret_cast<uint16_t*>(gbase + a.cache_off);
    uint32_t* stock = a.stock + (size_t)group * a.wg * (kRecordBlockBytes / 4);
    char* regions = a.regions + (uint64_t)group * a.wave * a.region_bytes;
    unsigned long long probes = 0, walks = 0;
    bool first = true;

    for (;;) {
        if (gt == 0) {
            // Waves shrink towards the end of the launch (half of an even
            // share of what is left), as far as building a wave's maps takes
            // longer than walking it.  The first waves of a CTA's groups differ
            // in length, so that one group walks while others build maps.
            const unsigned long long size = a.total - a.gidx_begin;
            const unsigned long long seen = *(volatile unsigned long long*)&a.ctrl->next;
            const unsigned long long rem = seen < size ? size - seen : 0;
            const unsigned long long fair = rem / (2ull * gridDim.x * a.ng);
            const uint32_t cap = first ? max(a.min_wave, a.wave * (g + 1) / a.ng) : a.wave;
            const uint32_t n = (uint32_t)min(max(fair, (unsigned long long)a.min_wave), (unsigned long long)cap);
            const unsigned long long base = atomicAdd(&a.ctrl->next, (unsigned long long)n);
            hd->base = base;
            hd->n = base < size ? (uint32_t)min((unsigned long long)n, size - base) : 0u;
        }
        first = false;
        wave_sync(g, nt);
        const uint32_t n = hd->n;
        if (!n) break;
        // trial i of the wave belongs to lane i / wg of the group's warp i % wg
        uint32_t* mine = stock + (gt >> 5) * (kRecordBlockBytes / 4) + lane;
        const uint32_t own = lane * a.wg + (gt >> 5);
        const unsigned long long gi = a.gidx_begin + hd->base + own;
        if (own < n) make_record<false, false>(a.jobs, a.njobs, L, gi, mine);
        wave_sync(g, nt);
        bool ok = true;
        for (uint32_t i = 0; i < n; ++i) {
            uint32_t* rec = hd->rec[i & 1];
            {
                const uint32_t* st = stock + (i % a.wg) * (kRecordBlockBytes / 4) + i / a.wg;
                for (uint32_t w = gt; w < kRecordWords; w += nt) rec[w] = __ldcg(st + w * 32);
            }
            wave_sync(g, nt);  // also: every warp has left the previous trial's fill and map
            const Job& J = a.jobs[rec[kStJob]];
            const uint32_t h = J.half_bits, mask = (uint32_t)J.mask;
            const uint32_t k3 = rec[kStKey + 28] >> 16;
            // F(r, y) = the round-2 lookups that read state word 1 (byte 1 of
            // R ^ rk3, that is y) and the record's fold entry of r
            const uint32_t yb = h > 8 ? h - 8 : 0;
            for (uint32_t v = gt; v < 8u << yb; v += nt) {
                const uint32_t y = v & ((1u << yb) - 1u), r = v >> yb;
                const uint32_t b = rec[kStKey + 27] ^ T2::e2<1>(L, (y << 8) ^ k3);
                const uint32_t* f = rec + kStFold + 4 * r;
                reinterpret_cast<uint4*>(gbase + kWaveHeaderBytes)[v] =
                    make_uint4(f[0] ^ T2::e1<2>(L, b), f[1] ^ T2::e0<3>(L, b), f[2] ^ T2::e3<0>(L, b),
                               f[3] ^ T2::e2<1>(L, b));
            }
            char* region = regions + (uint64_t)i * a.region_bytes;
            {
                const uint32_t nb = (J.buckets * (uint32_t)sizeof(Entry) + 15) / 16;
                const uint4 ones = make_uint4(kFull, kFull, kFull, kFull);
                for (uint32_t v = gt; v < nb; v += nt) __stcg(reinterpret_cast<uint4*>(region) + v, ones);
            }
            PrpKey key;
#pragma unroll
            for (int w = 0; w < 24; ++w) key.kr[4 + w] = rol8(rec[kStKey + w]);
            key.kr[29] = rol8(rec[kStKey + 24]);
            key.kr[30] = rol8(rec[kStKey + 25]);
            key.k43lo = rec[kStKey + 28] & 0xffffu;
            wave_sync(g, nt);
            wave_fill<GC>(L, key, J, rec[kStKey + 26], k3, fold, cache, h, mask, gt, nt);
            wave_sync(g, nt);
            MapT* map = reinterpret_cast<MapT*>(region + a.map_off);
            // Four chains per lane hide a gather's latency from L2.  Where L1
            // holds much of the caches (256 KiB at h = 14; a single group's) two
            // are faster, as the warps' rounds, 2^(h+1) bytes each, stay closer
            // together: t=1500, k=4 (h = 14) 47.0 -> 44.7 ms, t=4139 (h = 16) in
            // one group 58.2 -> 48.6, in two 51.4 -> 56.4.
            if constexpr (GC) {
                ok = (h > 14 && a.ng > 1 ? wave_map<4, true>(J, rec, cache, map, gt >> 5, a.wg, lane)
                                         : wave_map<2, true>(J, rec, cache, map, gt >> 5, a.wg, lane)) && ok;
            } else {
                ok = (J.last_rows ? wave_map<2, true>(J, rec, cache, map, gt >> 5, a.wg, lane)
                                  : wave_map<2, false>(J, rec, cache, map, gt >> 5, a.wg, lane)) && ok;
            }
        }
        wave_sync(g, nt);
        auto get64 = [&](uint32_t w) {
            return (uint64_t)__ldcg(mine + w * 32) | ((uint64_t)__ldcg(mine + (w + 1) * 32) << 32);
        };
        const bool owner = own < n;
        const uint32_t job = owner ? __ldcg(mine + kStJob * 32) : 0u;
        const Job& J = a.jobs[job];
        char* region = regions + (uint64_t)min(own, n - 1) * a.region_bytes;
        bool failed = false;
        if (__any_sync(kFull, owner && J.mode == 1))
            failed = walk_bgh<NARROW>(J, owner && J.mode == 1, owner ? get64(kStWalk) : 0,
                                      owner ? get64(kStWalk + 2) : 0, region, a.map_off, probes);
        if (__any_sync(kFull, owner && J.mode != 1))
            failed = walk_drrt<NARROW>(J, owner && J.mode != 1, region, a.map_off, probes) || failed;
        if (owner) {
            ++walks;
            if (failed) {
                atomicOr(&a.fail_bits[gi >> 5], 1u << (gi & 31));
                if (a.job_failed) atomicAdd(&a.job_failed[job], 1ULL);
            }
        }
        if (!ok) {
            atomicExch(&a.ctrl->error, kErrRange);
            atomicExch(&a.ctrl->where, 3u);
        }
    }
    for (int o = 16; o; o >>= 1) {
        probes += __shfl_xor_sync(kFull, probes, o);
        walks += __shfl_xor_sync(kFull, walks, o);
    }
    if (lane == 0) {
        atomicAdd(&a.ctrl->probes, probes);
        atomicAdd(&a.ctrl->walks, walks);
    }
}

template __global__ void cmc_waves<true, false>(const WaveArgs);
template __global__ void cmc_waves<true, true>(const WaveArgs);
template __global__ void cmc_waves<false, false>(const WaveArgs);
template __global__ void cmc_waves<false, true>(const WaveArgs);

}  // namespace cmc
