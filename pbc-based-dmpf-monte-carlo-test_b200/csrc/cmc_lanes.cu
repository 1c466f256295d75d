// cmc_lanes.cu -- the lane engine: one trial per thread, buckets evaluated as
// the walk asks for them.
//
// The group engine (cmc_engine.cu) evaluates all k*t buckets of a trial before
// its walk.  A walk touches far fewer: placing t items into B buckets needs
// about -B ln(1 - t/B) distinct (item, copy) pairs -- 1.65 t of 3 t at
// t/B = 2/3 -- because an item whose first bucket is empty never looks at its
// other copies.  A walk alone is a serial chain of 8-round AES Feistel
// evaluations, so here every thread runs its own trial: its own key schedule
// in registers, its own table in global memory, one Feistel pass per step of
// the warp's loop.  The lanes of a warp are in lockstep only for the AES
// rounds; each is at its own probe of its own trial, a lane that cycle-walks
// takes another pass, and a lane whose trial ends takes the next one from the
// warp's stock, so all lanes compute in every pass.
//
// What bounds it: shared-memory lookups.  A block costs 106 table lookups for
// AES rounds 3..10, 10 for rounds 1 and 2 and four words of the trial's fold
// table = 120 wavefronts of 32 lanes, one per clock and SM.  The T-tables are
// kept as four (T0..T3, 128 KiB), which saves the rotation that each column of
// the group engine's two-table form spends on the ALU pipe (6 ALU operations
// per column instead of 7).  The walks' global loads and stores (a bin, a memo
// entry) are hidden behind the other warps' passes.
//
// There is no spin-wait in this kernel.
#include <cstdint>

#include "cmc_aes.cuh"
#include "cmc_lanes.cuh"

namespace cmc {

namespace {

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

template <int B>
__device__ __forceinline__ uint32_t te0(const Lanes& L, uint32_t w) { return ldt<0>(toff<B>(w, L.lb0)); }
template <int B>
__device__ __forceinline__ uint32_t te1(const Lanes& L, uint32_t w) { return ldt<1>(toff<B>(w, L.lb0)); }
template <int B>
__device__ __forceinline__ uint32_t te2(const Lanes& L, uint32_t w) { return ldt<0>(toff<B>(w, L.lb2)); }
template <int B>
__device__ __forceinline__ uint32_t te3(const Lanes& L, uint32_t w) { return ldt<1>(toff<B>(w, L.lb2)); }

// One column of a full AES round with four tables.
__device__ __forceinline__ uint32_t column4(const Lanes& L, uint32_t a, uint32_t b, uint32_t c, uint32_t d,
                                            uint32_t k) {
    return xor3(xor3(te0<3>(L, a), te1<2>(L, b), te2<1>(L, c)), te3<0>(L, d), k);
}

// Last round: the S-box byte of byte B of w, at its place B in the result
// (T2 = (s, 3s, 2s, s) and T0 = (2s, s, s, 3s) from the top byte down hold s
// at bytes 0 and 3, and 1 and 2).
template <int B>
__device__ __forceinline__ uint32_t sub_at(const Lanes& L, uint32_t w) {
    if constexpr (B == 0 || B == 3) return te2<B>(L, w) & (0xffu << (8 * B));
    else return te0<B>(L, w) & (0xffu << (8 * B));
}

// Four full columns.
__device__ __forceinline__ void round4(const Lanes& L, uint32_t s[4], const uint32_t* k) {
    const uint32_t t0 = column4(L, s[0], s[1], s[2], s[3], k[0]);
    const uint32_t t1 = column4(L, s[1], s[2], s[3], s[0], k[1]);
    const uint32_t t2 = column4(L, s[2], s[3], s[0], s[1], k[2]);
    const uint32_t t3 = column4(L, s[3], s[0], s[1], s[2], k[3]);
    s[0] = t0; s[1] = t1; s[2] = t2; s[3] = t3;
}

// Full AES-128 block under a plain schedule in global memory (the batch key).
__device__ __forceinline__ void encrypt4(const Lanes& L, const uint32_t* rk, uint32_t s[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] ^= rk[i];
#pragma unroll 1
    for (int r = 4; r < 40; r += 4) {
        const uint32_t k[4] = {rk[r], rk[r + 1], rk[r + 2], rk[r + 3]};
        round4(L, s, k);
    }
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
        o[j] = (sub_at<3>(L, s[j]) | sub_at<2>(L, s[(j + 1) & 3]) | sub_at<1>(L, s[(j + 2) & 3]) |
                sub_at<0>(L, s[(j + 3) & 3])) ^ rk[40 + j];
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] = o[i];
}

__device__ __forceinline__ uint64_t splitmix(uint64_t& s) {
    s += 0x9E3779B97F4A7C15ULL;
    uint64_t z = s;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

// A trial's key and the part of AES_k(0x43455350, r, h, R) that does not
// depend on R.  Rounds 1 and 2 of the PRP block: with w = R ^ rk3,
//   s0 = c0 ^ Te3[w b0], s1 = c1 ^ Te2[w b1], s2 = c2(r), s3 = c3   (h <= 16)
// and the Feistel round number r (< 8) enters c2 alone, through byte 0 of
// state word 1.  The lookups of round 2 that read s2 and s3 are therefore a
// table of 8 four-word entries per trial (fold), and a block spends 2 + 8
// lookups and one 16-byte fold load on its first two rounds.
template <bool WIDE>
struct LaneKey;

template <>
struct LaneKey<false> {
    static constexpr uint32_t kWords = 29;
    uint32_t k[26];   // rk[12..35] (rounds 3..8), rk[37], rk[38] (round 9)
    uint32_t c0, c1;
    uint32_t ends;    // rk[3] low half << 16 | rk[43] low half

    // Low 16 bits of AES_k(0x43455350, r, h, R).w3 for R < 2^16; f = fold entry of r.
    __device__ __forceinline__ uint32_t block(const Lanes& L, const uint4& f, uint32_t R) const {
        const uint32_t w = R ^ (ends >> 16);
        const uint32_t a = c0 ^ te3<0>(L, w), b = c1 ^ te2<1>(L, w);
        uint32_t s[4];
        s[0] = xor3(te0<3>(L, a), te1<2>(L, b), f.x);
        s[1] = xor3(te0<3>(L, b), te3<0>(L, a), f.y);
        s[2] = xor3(te2<1>(L, a), te3<0>(L, b), f.z);
        s[3] = xor3(te1<2>(L, a), te2<1>(L, b), f.w);
#pragma unroll
        for (int r = 0; r < 6; ++r) round4(L, s, k + 4 * r);
        const uint32_t u1 = column4(L, s[1], s[2], s[3], s[0], k[24]);
        const uint32_t u2 = column4(L, s[2], s[3], s[0], s[1], k[25]);
        return (sub_at<1>(L, u1) | sub_at<0>(L, u2)) ^ ends;  // bits above 15 are for the caller's mask
    }
};

template <>
struct LaneKey<true> {
    static constexpr uint32_t kWords = 38;
    uint32_t k[32];  // rk[8..39] (rounds 2..9)
    uint32_t c0, c1, c3, k3, k43;
    uint32_t k1;     // byte 0 of state word 1 before r is added

    // w3 of AES_k(0x43455350, r, h, R) for any 32-bit R: the four bytes of R
    // enter one state word each.  c2 holds c2 without its r-dependent lookup.
    __device__ __forceinline__ uint32_t block(const Lanes& L, uint32_t c2, uint32_t r, uint32_t R) const {
        const uint32_t w = R ^ k3;
        uint32_t s[4];
        s[0] = c0 ^ te3<0>(L, w);
        s[1] = c1 ^ te2<1>(L, w);
        s[2] = xor3(c2, te3<0>(L, k1 ^ r), te1<2>(L, w));
        s[3] = c3 ^ te0<3>(L, w);
#pragma unroll
        for (int i = 0; i < 8; ++i) round4(L, s, k + 4 * i);
        return (sub_at<3>(L, s[3]) | sub_at<2>(L, s[0]) | sub_at<1>(L, s[1]) | sub_at<0>(L, s[2])) ^ k43;
    }
};

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

// The buckets of an item that its trial has evaluated so far (kUnknown for the
// others) and, packed with its ordinal, the table entry that holds it.  The
// buckets travel with the item: an evicted item brings along what is known of
// its other copies, so no bucket is evaluated twice and a probe needs one table
// read.  The copy an item sits by has the bin itself as its bucket, so an entry
// is four fields -- 4 x 16 bits, or 4 x 32 for tables with B > 65535 or
// t > 16384: field 3 holds ordinal and copy, and the bucket of copy 3 (k = 4)
// takes the place of the copy the item sits by.
template <bool NARROW>
struct Item;

template <>
struct Item<true> {
    using Entry = unsigned long long;
    static constexpr uint32_t kUnknown = 0xffffu;
    static constexpr Entry kEmpty = ~0ull;
    uint64_t b = ~0ull;
    __device__ __forceinline__ uint32_t get(uint32_t j) const { return (uint32_t)(b >> (16 * j)) & 0xffffu; }
    __device__ __forceinline__ void set(uint32_t j, uint32_t v) {
        b = (b & ~(0xffffull << (16 * j))) | ((uint64_t)v << (16 * j));
    }
    __device__ __forceinline__ Entry pack(uint32_t ord, uint32_t copy) const {
        Item e = *this;
        if (copy != 3) e.set(copy, get(3));
        return (e.b & 0x0000ffffffffffffull) | ((uint64_t)(ord | copy << 14) << 48);
    }
    __device__ __forceinline__ void unpack(Entry e, uint32_t bin, uint32_t& ord, uint32_t& copy) {
        const uint32_t x = (uint32_t)(e >> 48);
        ord = x & 0x3fffu;
        copy = x >> 14;
        b = e;
        set(3, copy != 3 ? get(copy) : bin);
        if (copy != 3) set(copy, bin);
    }
    static __device__ __forceinline__ Entry load(const Entry* p) { return __ldcg(p); }
    static __device__ __forceinline__ void store(Entry* p, Entry e) { __stcg(p, e); }
    static __device__ __forceinline__ bool empty(Entry e) { return e == kEmpty; }
};

template <>
struct Item<false> {
    using Entry = uint4;
    static constexpr uint32_t kUnknown = 0xffffffffu;
    uint32_t b0 = kUnknown, b1 = kUnknown, b2 = kUnknown, b3 = kUnknown;
    __device__ __forceinline__ uint32_t get(uint32_t j) const { return j == 0 ? b0 : j == 1 ? b1 : j == 2 ? b2 : b3; }
    __device__ __forceinline__ void set(uint32_t j, uint32_t v) {
        b0 = j == 0 ? v : b0;
        b1 = j == 1 ? v : b1;
        b2 = j == 2 ? v : b2;
        b3 = j == 3 ? v : b3;
    }
    __device__ __forceinline__ Entry pack(uint32_t ord, uint32_t copy) const {
        Item e = *this;
        if (copy != 3) e.set(copy, b3);
        return make_uint4(e.b0, e.b1, e.b2, ord | copy << 16);
    }
    __device__ __forceinline__ void unpack(const Entry& e, uint32_t bin, uint32_t& ord, uint32_t& copy) {
        ord = e.w & 0xffffu;
        copy = e.w >> 16;
        b0 = e.x;
        b1 = e.y;
        b2 = e.z;
        b3 = copy != 3 ? get(copy) : bin;
        if (copy != 3) set(copy, bin);
    }
    static __device__ __forceinline__ Entry load(const Entry* p) { return __ldcg(p); }
    static __device__ __forceinline__ void store(Entry* p, const Entry& e) { __stcg(p, e); }
    static __device__ __forceinline__ bool empty(const Entry& e) { return e.w == 0xffffffffu; }
};

// Set-up record of one trial, word w of record e at stock[w * 32 + e].
enum LaneStock : uint32_t {
    kStFold = 0,      // narrow: 32 fold words
    kStWalk = 32,     // walk, rnd, shift, step (two words each)
    kStGidx = 40,     // two words
    kStJob = 42,
    kStKey = 43,      // LaneKey words (wide: one more, c2)
};
static_assert(kStKey + LaneKey<false>::kWords <= kLaneStockWords, "a narrow record fits");
static_assert(kStKey + LaneKey<true>::kWords + 1 <= kLaneStockWords, "a wide record fits");

// Derives trial gi (cuckoo_bench.cu:226-238) and writes its record; one trial
// per lane.
template <bool WIDE>
__device__ __forceinline__ void make_record(const LaneArgs& a, const Lanes& L, uint64_t gi, uint32_t* st) {
    uint32_t lo = 0, hi = a.njobs;  // last job with trial_base <= gi
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (a.jobs[mid].trial_base <= gi) lo = mid; else hi = mid;
    }
    const Job& J = a.jobs[lo];
    const uint32_t offset = J.first + (uint32_t)(gi - J.trial_base);
    auto put = [&](uint32_t w, uint32_t v) { st[w * 32] = v; };
    auto put64 = [&](uint32_t w, uint64_t v) { put(w, (uint32_t)v); put(w + 1, (uint32_t)(v >> 32)); };
    put64(kStGidx, gi);
    put(kStJob, lo);
    {
        uint32_t s[4] = {0x57414c4bu, 0, offset, 0x524e4731u};
        encrypt4(L, J.batch_rk, s);
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
    encrypt4(L, J.batch_rk, w);
    // the key schedule (cuckoo_bench.cu:136-149), four words at a time
    const uint32_t k0 = w[0], k1 = w[1], k2 = w[2], k3 = w[3];
    uint32_t k4[4], k8[4];
    uint32_t rcon = 1;
    auto next = [&]() {
        const uint32_t v = (w[3] << 8) | (w[3] >> 24);
        const uint32_t t = sub_at<0>(L, v) | sub_at<1>(L, v) | sub_at<2>(L, v) | sub_at<3>(L, v);
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
        put(kStKey + 32, te0<3>(L, s0) ^ te1<2>(L, s1) ^ te2<1>(L, s2) ^ k4[0]);
        put(kStKey + 33, te0<3>(L, s1) ^ te1<2>(L, s2) ^ te3<0>(L, s0) ^ k4[1]);
        put(kStKey + 34, te1<2>(L, s0) ^ te2<1>(L, s1) ^ te3<0>(L, s2) ^ k4[3]);
        put(kStKey + 35, s3);
        put(kStKey + 36, w[3]);
        put(kStKey + 37, s1);
        put(kStKey + 38, te0<3>(L, s2) ^ te2<1>(L, s0) ^ k4[2]);
    } else {
        const uint32_t c0 = te0<3>(L, s0) ^ te1<2>(L, s1) ^ te2<1>(L, s2) ^ k4[0];
        const uint32_t c1 = te0<3>(L, s1) ^ te1<2>(L, s2) ^ te3<0>(L, s0) ^ k4[1];
        const uint32_t c3 = te0<3>(L, s3) ^ te1<2>(L, s0) ^ te2<1>(L, s1) ^ te3<0>(L, s2) ^ k4[3];
        const uint32_t c2b = te0<3>(L, s2) ^ te1<2>(L, s3) ^ te2<1>(L, s0) ^ k4[2];
        put(kStKey + 26, c0);
        put(kStKey + 27, c1);
        put(kStKey + 28, (s3 << 16) | (w[3] & 0xffffu));
        const uint32_t f0 = te3<0>(L, c3) ^ k8[0], f1 = te2<1>(L, c3) ^ k8[1];
        const uint32_t f2 = te1<2>(L, c3) ^ k8[2], f3 = te0<3>(L, c3) ^ k8[3];
#pragma unroll 1
        for (uint32_t r = 0; r < 8; ++r) {
            const uint32_t c2 = c2b ^ te3<0>(L, s1 ^ r);
            put(kStFold + 4 * r, f0 ^ te2<1>(L, c2));
            put(kStFold + 4 * r + 1, f1 ^ te1<2>(L, c2));
            put(kStFold + 4 * r + 2, f2 ^ te0<3>(L, c2));
            put(kStFold + 4 * r + 3, f3 ^ te3<0>(L, c2));
        }
    }
}

}  // namespace

// NARROW: 8-byte table entries (14-bit ordinals, 16-bit buckets), else 16-byte
// ones.  WIDE: PRP domains above 2^32.
template <bool NARROW, bool WIDE>
__global__ void __launch_bounds__(512, 1) cmc_lanes(const LaneArgs a) {
    if (!table_base_ok()) {
        if (threadIdx.x == 0) atomicExch(&a.ctrl->error, kErrBase);
        return;
    }
    using ItemT = Item<NARROW>;
    using Entry = typename ItemT::Entry;
    char* smem = cmc_dyn_smem;
    {
        uint32_t* tw = reinterpret_cast<uint32_t*>(smem);
        for (uint32_t i = threadIdx.x; i < kLaneTableBytes / 4; i += blockDim.x) {
            const uint32_t v = __ldg(&a.t0[(i >> 6) & 255u]);
            const uint32_t rot = ((i & 32) ? 16u : 0u) + (i >= kEngineTableBytes / 4 ? 8u : 0u);
            tw[i] = __funnelshift_r(v, v, rot);
        }
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Lanes L{lane * 4, lane * 4 + 128, 256u};
    const uint32_t gwarp = blockIdx.x * (blockDim.x >> 5) + warp;
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    uint32_t* stock = a.stock + (size_t)gwarp * (kLaneStockBytes / 4);
    const uint32_t first_region = gwarp * a.share;  // lanes share..31 take no trials and have none
    Entry* bins = reinterpret_cast<Entry*>(a.regions + (uint64_t)(first_region + min(lane, a.share - 1)) * a.region_bytes);
    uint4* fold = reinterpret_cast<uint4*>(smem + kLaneTableBytes + warp * kLaneFoldBytes) + lane;

    LaneKey<WIDE> key;
    uint32_t* kw = reinterpret_cast<uint32_t*>(&key);
#pragma unroll
    for (uint32_t i = 0; i < LaneKey<WIDE>::kWords; ++i) kw[i] = 0;
    uint32_t c2 = 0;
    // the trial's walk
    uint64_t walk = 0, rnd = 0, gidx = 0, shift = 0, step = 0;
    uint32_t jidx = 0;
    ItemT it;  // the item in hand: ordinal cur, to be placed by copy `which`
    uint32_t item = 0, cur = 0, which = 0, count = 0, prev = 0, tried = 0, tgt = 0;
    uint32_t phase = 0;  // DRRT18: 0 placing a new item, 1 evicting
    bool busy = false, bad = false;
    bool known = false;  // tgt is the bucket of (cur, which) already: no pass needed
    // the value under evaluation
    uint32_t left = 0, right = 0;
    unsigned long long probes = 0, walks = 0;
    uint32_t stock_n = 0, stock_i = 0;  // warp-uniform
    bool more = true;

    for (;;) {
        // Lanes without a trial take one from the stock; an empty stock is
        // refilled by one claim, all its trials set up side by side.
        unsigned idle = __ballot_sync(kFull, !busy && lane < a.share);
        while (idle && (stock_i < stock_n || more)) {
            if (stock_i == stock_n) {
                // Claims shrink towards the end of the launch (half of an even
                // share of what is left, at least what idle lanes need), so
                // that no warp keeps a stock while others have nothing to do.
                uint32_t n = 0;
                unsigned long long base = 0;
                if (lane == 0) {
                    const unsigned long long size = a.total - a.gidx_begin;
                    const unsigned long long seen = *(volatile unsigned long long*)&a.ctrl->next;
                    const unsigned long long rem = seen < size ? size - seen : 0;
                    const unsigned long long fair = rem / (2ull * nwarps);
                    const uint32_t need = __popc(idle);
                    n = fair > need ? (uint32_t)min(fair, 32ull) : need;
                    base = atomicAdd(&a.ctrl->next, (unsigned long long)n);
                    n = base < size ? (uint32_t)min((unsigned long long)n, size - base) : 0u;
                }
                n = __shfl_sync(kFull, n, 0);
                base = __shfl_sync(kFull, base, 0);
                if (n == 0) {
                    more = false;
                    break;
                }
                if (lane < n) make_record<WIDE>(a, L, a.gidx_begin + base + lane, stock + lane);
                __syncwarp();
                stock_i = 0;
                stock_n = n;
            }
            const uint32_t rank = __popc(idle & ((1u << lane) - 1u));
            const uint32_t take = min((uint32_t)__popc(idle), stock_n - stock_i);
            const bool taking = ((idle >> lane) & 1u) && rank < take;
            if (taking) {
                const uint32_t* st = stock + stock_i + rank;
                auto get = [&](uint32_t w) { return st[w * 32]; };
                auto get64 = [&](uint32_t w) { return (uint64_t)st[w * 32] | ((uint64_t)st[(w + 1) * 32] << 32); };
#pragma unroll
                for (uint32_t i = 0; i < LaneKey<WIDE>::kWords; ++i) kw[i] = get(kStKey + i);
                if constexpr (WIDE) {
                    c2 = get(kStKey + LaneKey<WIDE>::kWords);
                } else {
#pragma unroll
                    for (uint32_t r = 0; r < 8; ++r)
                        fold[r * 32] = make_uint4(get(kStFold + 4 * r), get(kStFold + 4 * r + 1),
                                                  get(kStFold + 4 * r + 2), get(kStFold + 4 * r + 3));
                }
                walk = get64(kStWalk);
                rnd = get64(kStWalk + 2);
                shift = get64(kStWalk + 4);
                step = get64(kStWalk + 6);
                gidx = get64(kStGidx);
                jidx = get(kStJob);
            }
            stock_i += take;
            // the warp empties the tables of the lanes that took a trial
            const unsigned taken = __ballot_sync(kFull, taking);
            for (unsigned m = taken; m; m &= m - 1) {
                const uint32_t src = __ffs(m) - 1;
                const uint32_t j = __shfl_sync(kFull, jidx, src);
                char* rg = a.regions + (uint64_t)(first_region + src) * a.region_bytes;
                const uint32_t nb = (a.jobs[j].buckets * (uint32_t)sizeof(Entry) + 15) / 16;
                const uint4 ones = make_uint4(kFull, kFull, kFull, kFull);
                for (uint32_t i = lane; i < nb; i += 32) __stcg(reinterpret_cast<uint4*>(rg) + i, ones);
            }
            __syncwarp();
            if (taking) {
                const Job& J = a.jobs[jidx];
                item = 0; cur = 0; count = 0; phase = 0; prev = 0; tried = 0;
                bad = false;
                busy = true;
                known = false;
                it = ItemT{};
                which = 0;
                if (J.mode == 1) which = next_digit(walk, rnd, J.k);
                const uint64_t e = J.input_mode == 0 ? 0 : shift;
                const uint64_t y = e * J.k + which;
                left = (uint32_t)(y >> J.half_bits);
                right = (uint32_t)(y & J.mask);
            }
            idle &= ~taken;
        }
        if (!__any_sync(kFull, busy)) break;

        const Job& J = a.jobs[jidx];
        const uint32_t mask = (uint32_t)J.mask;
        // One Feistel pass (8 rounds) of every lane's value, unless every lane
        // is on a known bucket.
        if (__any_sync(kFull, busy && !known)) {
            uint32_t l = left, r = right;
#pragma unroll 1
            for (uint32_t rr = 0; rr < 8; ++rr) {
                uint32_t f;
                if constexpr (WIDE) f = key.block(L, c2, rr, r);
                else f = key.block(L, fold[rr * 32], r);
                const uint32_t nr = (l ^ f) & mask;
                l = r;
                r = nr;
            }
            left = l;
            right = r;
        }
        if (!busy) continue;
        const uint32_t h = J.half_bits;
        const uint32_t k = J.k, t = J.pnum, kick = J.kick;
        if (!known) {
            const uint64_t y = ((uint64_t)left << h) | right;
            if (y >= J.domain) continue;  // cycle-walk: another pass from this value
            if constexpr (WIDE) tgt = (uint32_t)(y / J.width);
            else tgt = div_width((uint32_t)y, (uint32_t)J.width, J.width_magic);
            if (tgt >= J.buckets) {
                bad = true;
                tgt = 0;
            }
            it.set(which, tgt);
        }
        // Probe until the next bucket has to be evaluated, at most a.hops table
        // reads: a lane still on known buckets then sits out one pass, so that
        // the others need not wait for it.
        known = false;
        bool done = false, failed = false;
        uint32_t reads = 0;
        if (J.mode == 1) {
            // BGH25 random walk (cuckoo_core.hpp:123-133)
            Entry old = ItemT::load(bins + tgt);
            for (;;) {
                ++probes;
                const Entry mine = it.pack(cur, which);
                ItemT::store(bins + tgt, mine);
                if (ItemT::empty(old)) {
                    cur = ++item;
                    count = 0;
                    done = item == t;
                    it = ItemT{};
                    if (!done) which = next_digit(walk, rnd, k);
                    break;
                }
                uint32_t copy;
                it.unpack(old, tgt, cur, copy);
                if (++count > kick) {
                    done = failed = true;
                    break;
                }
                which = next_digit(walk, rnd, k);
                const uint32_t m = it.get(which);
                if (m == ItemT::kUnknown) break;
                if (which == copy) {
                    old = mine;  // the copy it was evicted from: this bin again
                    continue;
                }
                tgt = m;
                if (++reads == a.hops) {
                    known = true;
                    break;
                }
                old = ItemT::load(bins + tgt);
            }
        } else {
            // DRRT18 cycling eviction (cuckoo_core.hpp:134-158)
            for (;;) {
                if (phase == 0) {
                    ++probes;
                    if (ItemT::empty(ItemT::load(bins + tgt))) {
                        ItemT::store(bins + tgt, it.pack(item, which));
                        cur = ++item;
                        which = 0;
                        it = ItemT{};
                        done = item == t;
                        break;
                    }
                    if (++which != k) break;
                    phase = 1;
                    which = 0;
                    count = 0;
                    tgt = it.get(0);
                } else if (tgt == prev) {
                    // this copy of the displaced item is the bin it left: its
                    // next copy, if it has one more
                    if (++tried == k - 1) {
                        done = failed = true;
                        break;
                    }
                    which = which + 1 == k ? 0 : which + 1;
                    tgt = it.get(which);
                    if (tgt == ItemT::kUnknown) break;
                    continue;
                } else {
                    ++count;
                }
                // evict from tgt
                ++probes;
                const Entry old = ItemT::load(bins + tgt);
                if (ItemT::empty(old)) {
                    ItemT::store(bins + tgt, it.pack(cur, which));
                    cur = ++item;
                    which = 0;
                    phase = 0;
                    it = ItemT{};
                    done = item == t;
                    break;
                }
                if (count >= kick) {
                    done = failed = true;
                    break;
                }
                ItemT::store(bins + tgt, it.pack(cur, which));
                it.unpack(old, tgt, cur, which);
                which = which + 1 == k ? 0 : which + 1;
                prev = tgt;
                tried = 0;
                tgt = it.get(which);
                if (tgt == ItemT::kUnknown) break;
                if (++reads == a.hops) {
                    known = true;
                    break;
                }
            }
        }
        if (done || bad) {
            if (bad) {
                atomicExch(&a.ctrl->error, kErrRange);
                atomicExch(&a.ctrl->where, 3u);
            }
            if (failed) {
                atomicOr(&a.fail_bits[gidx >> 5], 1u << (gidx & 31));
                if (a.job_failed) atomicAdd(&a.job_failed[jidx], 1ULL);
            }
            ++walks;
            busy = false;
        } else if (!known) {
            const uint64_t e = J.input_mode == 0 ? (uint64_t)cur : (shift + (uint64_t)cur * step) & J.range_mask;
            const uint64_t y0 = e * k + which;
            left = (uint32_t)(y0 >> h);
            right = (uint32_t)y0 & mask;
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

template __global__ void cmc_lanes<true, false>(const LaneArgs);
template __global__ void cmc_lanes<false, false>(const LaneArgs);
template __global__ void cmc_lanes<false, true>(const LaneArgs);

}  // namespace cmc
