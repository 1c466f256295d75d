// cmc_trial.cuh -- device code of one trial on one thread: AES round tables and
// set-up records (cmc_lanes.cu, cmc_waves.cu), walk digits and table entries
// (those and cmc_engine.cu), and the walk of the group engine's global slots
// (cmc_engine.cu).
#pragma once
#include <cstdint>

#include "cmc_aes.cuh"
#include "cmc_engine.cuh"

namespace cmc {

// Words of one trial's set-up record (TrialRecord), kept as [word][32 records]
// per warp.
constexpr uint32_t kRecordWords = 84;
constexpr uint32_t kRecordBlockBytes = kRecordWords * 32 * 4;

constexpr unsigned kFull = 0xffffffffu;
constexpr uint32_t kErrBase = 3;   // == -CMC_EKAT: table_base_ok() failed
constexpr uint32_t kErrRange = 5;  // == -CMC_ERANGE

// Lookup in the table pair P: P = 0 holds T0 (lb0) and T2 (lb2), P = 1 holds
// T1 and T3, kEngineTableBytes above it.
template <int P>
__device__ __forceinline__ uint32_t ldt(uint32_t off) {
    uint32_t v;
    if constexpr (P == 0)
        asm volatile("ld.shared.u32 %0, [%1+" CMC_STR(CMC_DYN_SMEM_BASE) "];" : "=r"(v) : "r"(off));
    else
        asm volatile("ld.shared.u32 %0, [%1+" CMC_STR(CMC_DYN_SMEM_BASE) "+65536];" : "=r"(v) : "r"(off));
    return v;
}
static_assert(kEngineTableBytes == 65536, "ldt addresses the second table pair");

// Byte B of w through the AES round table T0..T3: with FOUR from four tables,
// else from T0 and T2 and a rotation (T1 = ror8(T0), T3 = ror8(T2)).
template <bool FOUR>
struct Te {
    template <int B>
    static __device__ __forceinline__ uint32_t e0(const Lanes& L, uint32_t w) { return ldt<0>(toff<B>(w, L.lb0)); }
    template <int B>
    static __device__ __forceinline__ uint32_t e1(const Lanes& L, uint32_t w) {
        if constexpr (FOUR) return ldt<1>(toff<B>(w, L.lb0));
        else return ror8(e0<B>(L, w));
    }
    template <int B>
    static __device__ __forceinline__ uint32_t e2(const Lanes& L, uint32_t w) { return ldt<0>(toff<B>(w, L.lb2)); }
    template <int B>
    static __device__ __forceinline__ uint32_t e3(const Lanes& L, uint32_t w) {
        if constexpr (FOUR) return ldt<1>(toff<B>(w, L.lb2));
        else return ror8(e2<B>(L, w));
    }
    // One column of a full round.
    static __device__ __forceinline__ uint32_t column(const Lanes& L, uint32_t a, uint32_t b, uint32_t c,
                                                      uint32_t d, uint32_t k) {
        return xor3(xor3(e0<3>(L, a), e1<2>(L, b), e2<1>(L, c)), e3<0>(L, d), k);
    }
    static __device__ __forceinline__ void round(const Lanes& L, uint32_t s[4], const uint32_t* k) {
        const uint32_t t0 = column(L, s[0], s[1], s[2], s[3], k[0]);
        const uint32_t t1 = column(L, s[1], s[2], s[3], s[0], k[1]);
        const uint32_t t2 = column(L, s[2], s[3], s[0], s[1], k[2]);
        const uint32_t t3 = column(L, s[3], s[0], s[1], s[2], k[3]);
        s[0] = t0; s[1] = t1; s[2] = t2; s[3] = t3;
    }
    // Last round: the S-box byte of byte B of w, at its place B in the result
    // (T2 = (s, 3s, 2s, s) and T0 = (2s, s, s, 3s) from the top byte down hold
    // s at bytes 0 and 3, and 1 and 2).
    template <int B>
    static __device__ __forceinline__ uint32_t sub_at(const Lanes& L, uint32_t w) {
        if constexpr (B == 0 || B == 3) return e2<B>(L, w) & (0xffu << (8 * B));
        else return e0<B>(L, w) & (0xffu << (8 * B));
    }
    // Full AES-128 block under a plain schedule in global memory (the batch key).
    static __device__ __forceinline__ void encrypt(const Lanes& L, const uint32_t* rk, uint32_t s[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] ^= rk[i];
#pragma unroll 1
        for (int r = 4; r < 40; r += 4) {
            const uint32_t k[4] = {rk[r], rk[r + 1], rk[r + 2], rk[r + 3]};
            round(L, s, k);
        }
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            o[j] = (sub_at<3>(L, s[j]) | sub_at<2>(L, s[(j + 1) & 3]) | sub_at<1>(L, s[(j + 2) & 3]) |
                    sub_at<0>(L, s[(j + 3) & 3])) ^ rk[40 + j];
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = o[i];
    }
};

// The T-tables in shared memory, by all threads of the CTA: row x of a pair is
// [T0[x] x 32][T2[x] x 32], then [T1[x] x 32][T3[x] x 32].
template <bool FOUR>
__device__ __forceinline__ void build_tables(const uint32_t* t0, char* smem) {
    uint32_t* tw = reinterpret_cast<uint32_t*>(smem);
    for (uint32_t i = threadIdx.x; i < (FOUR ? 2 : 1) * kEngineTableBytes / 4; i += blockDim.x) {
        const uint32_t v = __ldg(&t0[(i >> 6) & 255u]);
        const uint32_t rot = ((i & 32) ? 16u : 0u) + (i >= kEngineTableBytes / 4 ? 8u : 0u);
        tw[i] = __funnelshift_r(v, v, rot);
    }
}

__device__ __forceinline__ uint64_t splitmix(uint64_t& s) {
    s += 0x9E3779B97F4A7C15ULL;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

// floor(y / width), y < 2^32, magic = floor((2^32 - 1) / width).
__device__ __forceinline__ uint32_t div_width(uint32_t y, uint32_t width, uint32_t magic) {
    uint32_t q = __umulhi(y, magic);
    uint32_t r = y - q * width;
    if (r >= width) { ++q; r -= width; }
    if (r >= width) { ++q; }
    return q;
}

// The next base-k digit (k = 2, 3, 4) of a walk's randomness: "if (r < k) r =
// splitmix(walk); which = r % k; r /= k" (cuckoo_core.hpp:126-127).
__device__ __forceinline__ uint32_t next_digit(uint64_t& walk, uint64_t& rnd, uint32_t k) {
    if (rnd < k) rnd = splitmix(walk);
    const uint64_t q = k == 3 ? __umul64hi(rnd, 0xAAAAAAAAAAAAAAABULL) >> 1 : rnd >> (k >> 1);
    const uint32_t d = (uint32_t)rnd - (uint32_t)q * k;
    rnd = q;
    return d;
}

// The digits of a walk decoded ahead, eight at a time: one 64-bit division by
// k^8 and eight 16-bit ones instead of eight 64-bit ones.  A randomness below
// k^8 gives its last digits (as long as it is k or more) and is replaced.
struct Digits {
    uint64_t walk = 0, rnd = 0;
    uint64_t buf = 0;  // n digits of two bits, the next one lowest
    uint32_t n = 0;

    // Appends up to eight digits (n <= 24 before).
    __device__ __forceinline__ void block(uint32_t k) {
        const uint32_t all = k == 3 ? 6561u : k == 2 ? 256u : 65536u;
        // floor(rnd / 3^8) for every 64-bit rnd: 0x9fd1... = ceil(2^76 / 3^8), within 2^12 / 3^8 of it
        const uint64_t q8 = k == 3 ? __umul64hi(rnd, 0x9fd1cd5aa3cca6d8ULL) >> 12 : rnd >> (k == 2 ? 8 : 16);
        const bool full = rnd >= all;
        uint32_t r = full ? (uint32_t)rnd - (uint32_t)q8 * all : (uint32_t)rnd;
        uint32_t word = 0, m = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            m += r >= k;
            // 21846 = ceil(2^16 / 3) divides r < 2^15 by 3
            const uint32_t q = k == 3 ? (r * 21846u) >> 16 : r >> (k >> 1);
            word |= (r - q * k) << (2 * i);
            r = q;
        }
        m = full ? 8u : m;
        buf |= (uint64_t)(word & ((1u << (2 * m)) - 1u)) << (2 * n);
        n += m;
        rnd = q8;
        if (!full) rnd = splitmix(walk);
    }
    // At least 17 digits.
    __device__ __forceinline__ void top_up(uint32_t k) {
        while (n <= 16) block(k);
    }
    __device__ __forceinline__ uint32_t next(uint32_t k) {
        while (n == 0) block(k);
        const uint32_t d = (uint32_t)buf & 3u;
        buf >>= 2;
        --n;
        return d;
    }
};

// The buckets of an item that its trial has evaluated so far (kUnknown for the
// others) and, packed with its ordinal, the table entry that holds it.  The
// buckets travel with the item: an evicted item brings along what is known of
// its other copies, so no bucket is evaluated twice and a probe needs one table
// read.  An entry is four fields -- 4 x 16 bits, or 4 x 32 for tables with
// B > 65535 or t > 16384: the buckets of copies 0..2, then ordinal and copy.
// With k = 4 (`four`) the bucket of copy 3 takes the place of the copy the item
// sits by, whose bucket is the bin itself.
template <bool NARROW>
struct Item;

template <>
struct Item<true> {
    using Entry = uint2;
    using Bucket = uint16_t;
    static constexpr uint32_t kUnknown = 0xffffu;
    uint32_t lo = 0xffffffffu, hi = 0xffffffffu;
    // an item from the four fields (its buckets)
    static __device__ __forceinline__ Item from(const Entry& e) {
        Item i;
        i.lo = e.x;
        i.hi = e.y;
        return i;
    }
    __device__ __forceinline__ uint32_t get(uint32_t j) const {
        return __byte_perm(lo, hi, 0x10u + 0x22u * j) & 0xffffu;
    }
    __device__ __forceinline__ void set(uint32_t j, uint32_t v) {
        lo = __byte_perm(lo, v, j == 0 ? 0x3254u : j == 1 ? 0x5410u : 0x3210u);
        hi = __byte_perm(hi, v, j == 2 ? 0x3254u : j == 3 ? 0x5410u : 0x3210u);
    }
    __device__ __forceinline__ Entry pack(uint32_t ord, uint32_t copy, bool four) const {
        Item e = *this;
        if (four && copy != 3) e.set(copy, hi >> 16);
        return make_uint2(e.lo, __byte_perm(e.hi, ord | copy << 14, 0x5410u));
    }
    __device__ __forceinline__ void unpack(const Entry& e, uint32_t bin, bool four, uint32_t& ord, uint32_t& copy) {
        ord = (e.y >> 16) & 0x3fffu;
        copy = e.y >> 30;
        lo = e.x;
        hi = e.y;
        if (four) {
            const uint32_t third = copy != 3 ? get(copy) : bin;
            if (copy != 3) set(copy, bin);
            set(3, third);
        }
    }
    static __device__ __forceinline__ Entry load(const Entry* p) { return __ldcg(p); }
    static __device__ __forceinline__ void store(Entry* p, const Entry& e) { __stcg(p, e); }
    static __device__ __forceinline__ bool empty(const Entry& e) { return e.y >= 0xffff0000u; }
};

template <>
struct Item<false> {
    using Entry = uint4;
    using Bucket = uint32_t;
    static constexpr uint32_t kUnknown = 0xffffffffu;
    uint32_t b0 = kUnknown, b1 = kUnknown, b2 = kUnknown, b3 = kUnknown;
    static __device__ __forceinline__ Item from(const Entry& e) {
        Item i;
        i.b0 = e.x; i.b1 = e.y; i.b2 = e.z; i.b3 = e.w;
        return i;
    }
    __device__ __forceinline__ uint32_t get(uint32_t j) const { return j == 0 ? b0 : j == 1 ? b1 : j == 2 ? b2 : b3; }
    __device__ __forceinline__ void set(uint32_t j, uint32_t v) {
        b0 = j == 0 ? v : b0;
        b1 = j == 1 ? v : b1;
        b2 = j == 2 ? v : b2;
        b3 = j == 3 ? v : b3;
    }
    __device__ __forceinline__ Entry pack(uint32_t ord, uint32_t copy, bool four) const {
        Item e = *this;
        if (four && copy != 3) e.set(copy, b3);
        return make_uint4(e.b0, e.b1, e.b2, ord | copy << 16);
    }
    __device__ __forceinline__ void unpack(const Entry& e, uint32_t bin, bool four, uint32_t& ord, uint32_t& copy) {
        ord = e.w & 0xffffu;
        copy = e.w >> 16;
        b0 = e.x;
        b1 = e.y;
        b2 = e.z;
        if (four) {
            b3 = copy != 3 ? get(copy) : bin;
            if (copy != 3) set(copy, bin);
        }
    }
    static __device__ __forceinline__ Entry load(const Entry* p) { return __ldcg(p); }
    static __device__ __forceinline__ void store(Entry* p, const Entry& e) { __stcg(p, e); }
    static __device__ __forceinline__ bool empty(const Entry& e) { return e.w == 0xffffffffu; }
};

// One trial's walk over a table of entries whose items carry their buckets, a
// probe per step: one table read, and both of its outcomes (item placed, item
// evicted) as selects.  The walk's digits are decoded ahead, for all lanes
// together (top_up), and an item that returns to the bin it left costs no read.
// Over the group engine's global slots against plain bins and a k-fold map, two
// reads a probe: t = 8000, N = 2^24, 16,384 trials 55.7 -> 44.2 ms.
//
// bgh_step and drrt_step are the loop bodies of walk_bgh and walk_drrt in
// cmc_waves.cu, which keep their state in local variables: through this struct
// the wave engine takes two registers more in its fill (t = 1024, 2^20 trials:
// 229 -> 248 ms).  A change to the rules of a walk has to be made in both.
template <bool NARROW>
struct ItemWalk {
    using ItemT = Item<NARROW>;
    using Entry = typename ItemT::Entry;
    Entry* bins;
    const Entry* map;  // the items' buckets
    uint32_t k, last, kick;
    Digits digits;
    ItemT it;           // the item in hand, number cur, and its copy to try
    Entry ahead, mine;  // the next item's buckets; what this walk wrote last
    uint32_t item, cur, count, which, bin;
    bool again, evicting, active, failed;

    __device__ __forceinline__ void begin(char* table, const char* buckets, uint32_t copies, uint32_t t, uint32_t limit,
                                          bool bgh, uint64_t walk, uint64_t rnd) {
        bins = reinterpret_cast<Entry*>(table);
        map = reinterpret_cast<const Entry*>(buckets);
        k = copies;
        last = t - 1;
        kick = limit;
        digits = Digits{};
        digits.walk = walk;
        digits.rnd = rnd;
        it = ItemT::from(ItemT::load(map));
        ahead = ItemT::load(map + 1);  // t >= 3
        mine = ahead;
        item = cur = count = 0;
        again = evicting = failed = false;
        active = true;
        which = bgh ? digits.next(k) : 0u;
        bin = it.get(which);
    }

    // BGH25 random walk (cuckoo_core.hpp:123-133); an item that returns to the
    // bin it left finds the item that evicted it, the second time in one step.
    __device__ __forceinline__ void bgh_step(uint32_t& steps) {
        const bool four = k == 4;
        Entry old = mine;
        if (!again) old = ItemT::load(bins + bin);
        mine = it.pack(cur, which, four);
        ++steps;
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
            ++steps;
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

    // DRRT18 cycling eviction (cuckoo_core.hpp:134-158).
    __device__ __forceinline__ void drrt_step(uint32_t& steps) {
        const bool four = k == 4;
        const Entry old = ItemT::load(bins + bin);
        const Entry entry = it.pack(cur, which, four);
        ++steps;
        const bool placed = ItemT::empty(old), evict = evicting && !placed;
        if (placed || (evict && count < kick)) ItemT::store(bins + bin, entry);
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
};

// Set-up record of one trial, word w of record e at stock[w * 32 + e].
enum TrialRecord : uint32_t {
    kStFold = 0,      // narrow: 32 fold words
    kStWalk = 32,     // walk, rnd, shift, step (two words each)
    kStGidx = 40,     // two words
    kStJob = 42,
    kStKey = 43,      // key words (LaneKey in cmc_lanes.cu; wide: one more, c2)
};

// Derives trial gi (cuckoo_bench.cu:226-238) and writes its record; one trial
// per lane.
template <bool FOUR, bool WIDE>
__device__ __forceinline__ void make_record(const Job* jobs, uint32_t njobs, const Lanes& L, uint64_t gi,
                                            uint32_t* st) {
    using T = Te<FOUR>;
    uint32_t lo = 0, hi = njobs;  // last job with trial_base <= gi
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (jobs[mid].trial_base <= gi) lo = mid; else hi = mid;
    }
    const Job& J = jobs[lo];
    const uint32_t offset = J.first + (uint32_t)(gi - J.trial_base);
    auto put = [&](uint32_t w, uint32_t v) { st[w * 32] = v; };
    auto put64 = [&](uint32_t w, uint64_t v) { put(w, (uint32_t)v); put(w + 1, (uint32_t)(v >> 32)); };
    put64(kStGidx, gi);
    put(kStJob, lo);
    {
        uint32_t s[4] = {0x57414c4bu, 0, offset, 0x524e4731u};
        T::encrypt(L, J.batch_rk, s);
        uint64_t walk = ((uint64_t)s[0] << 32) | s[1];
        const uint64_t shift = (((uint64_t)s[2] << 32) | s[3]) & J.range_mask;
        uint64_t input_state = shift ^ 0xd1b54a32d192ed03ULL;
        const uint64_t step = (splitmix(input_state) | 1ULL) & J.range_mask;
        const uint64_t rnd = splitmix(walk);
        put64(kStWalk, walk);
        put64(kStWalk + 2, rnd);
        put64(kStWalk + 4, shift);
        put64(kStWalk + 6, step);
    }
    uint32_t w[4] = {0x4b455931u, 0, offset, 0x50525031u};
    T::encrypt(L, J.batch_rk, w);
    // the key schedule (cuckoo_bench.cu:136-149), four words at a time
    const uint32_t k0 = w[0], k1 = w[1], k2 = w[2], k3 = w[3];
    uint32_t k4[4], k8[4];
    uint32_t rcon = 1;
    auto next = [&]() {
        const uint32_t v = (w[3] << 8) | (w[3] >> 24);
        const uint32_t t = T::template sub_at<0>(L, v) | T::template sub_at<1>(L, v) | T::template sub_at<2>(L, v) | T::template sub_at<3>(L, v);
        w[0] ^= t ^ (rcon << 24);
        rcon = (rcon << 1) ^ ((rcon & 0x80u) ? 0x1bu : 0u);
        w[1] ^= w[0];
        w[2] ^= w[1];
        w[3] ^= w[2];
    };
    next();
#pragma unroll
    for (int i = 0; i < 4; ++i) k4[i] = w[i];
    next();
#pragma unroll
    for (int i = 0; i < 4; ++i) k8[i] = w[i];
    if constexpr (WIDE) {
#pragma unroll
        for (int i = 0; i < 4; ++i) put(kStKey + i, k8[i]);
    }
#pragma unroll 1
    for (uint32_t i = 3; i < 10; ++i) {  // rk[12..39]
        next();
        if constexpr (WIDE) {
            for (int j = 0; j < 4; ++j) put(kStKey + 4 * (i - 2) + j, w[j]);
        } else if (i < 9) {
            for (int j = 0; j < 4; ++j) put(kStKey + 4 * (i - 3) + j, w[j]);
        } else {
            put(kStKey + 24, w[1]);
            put(kStKey + 25, w[2]);
        }
    }
    next();
    const uint32_t h = J.half_bits;
    const uint32_t s0 = 0x43455350u ^ k0, s1 = k1, s2 = h ^ k2, s3 = k3;
    if constexpr (WIDE) {
        put(kStKey + 32, T::template e0<3>(L, s0) ^ T::template e1<2>(L, s1) ^ T::template e2<1>(L, s2) ^ k4[0]);
        put(kStKey + 33, T::template e0<3>(L, s1) ^ T::template e1<2>(L, s2) ^ T::template e3<0>(L, s0) ^ k4[1]);
        put(kStKey + 34, T::template e1<2>(L, s0) ^ T::template e2<1>(L, s1) ^ T::template e3<0>(L, s2) ^ k4[3]);
        put(kStKey + 35, s3);
        put(kStKey + 36, w[3]);
        put(kStKey + 37, s1);
        put(kStKey + 38, T::template e0<3>(L, s2) ^ T::template e2<1>(L, s0) ^ k4[2]);
    } else {
        const uint32_t c0 = T::template e0<3>(L, s0) ^ T::template e1<2>(L, s1) ^ T::template e2<1>(L, s2) ^ k4[0];
        const uint32_t c1 = T::template e0<3>(L, s1) ^ T::template e1<2>(L, s2) ^ T::template e3<0>(L, s0) ^ k4[1];
        const uint32_t c3 = T::template e0<3>(L, s3) ^ T::template e1<2>(L, s0) ^ T::template e2<1>(L, s1) ^ T::template e3<0>(L, s2) ^ k4[3];
        const uint32_t c2b = T::template e0<3>(L, s2) ^ T::template e1<2>(L, s3) ^ T::template e2<1>(L, s0) ^ k4[2];
        put(kStKey + 26, c0);
        put(kStKey + 27, c1);
        put(kStKey + 28, (s3 << 16) | (w[3] & 0xffffu));
        const uint32_t f0 = T::template e3<0>(L, c3) ^ k8[0], f1 = T::template e2<1>(L, c3) ^ k8[1];
        const uint32_t f2 = T::template e1<2>(L, c3) ^ k8[2], f3 = T::template e0<3>(L, c3) ^ k8[3];
#pragma unroll 1
        for (uint32_t r = 0; r < 8; ++r) {
            const uint32_t c2 = c2b ^ T::template e3<0>(L, s1 ^ r);
            put(kStFold + 4 * r, f0 ^ T::template e2<1>(L, c2));
            put(kStFold + 4 * r + 1, f1 ^ T::template e1<2>(L, c2));
            put(kStFold + 4 * r + 2, f2 ^ T::template e0<3>(L, c2));
            put(kStFold + 4 * r + 3, f3 ^ T::template e3<0>(L, c2));
        }
    }
}

}  // namespace cmc
