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

#include "cmc_lanes.cuh"
#include "cmc_trial.cuh"

namespace cmc {

namespace {

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
        const uint32_t a = c0 ^ Te<true>::e3<0>(L, w), b = c1 ^ Te<true>::e2<1>(L, w);
        uint32_t s[4];
        s[0] = xor3(Te<true>::e0<3>(L, a), Te<true>::e1<2>(L, b), f.x);
        s[1] = xor3(Te<true>::e0<3>(L, b), Te<true>::e3<0>(L, a), f.y);
        s[2] = xor3(Te<true>::e2<1>(L, a), Te<true>::e3<0>(L, b), f.z);
        s[3] = xor3(Te<true>::e1<2>(L, a), Te<true>::e2<1>(L, b), f.w);
#pragma unroll
        for (int r = 0; r < 6; ++r) Te<true>::round(L, s, k + 4 * r);
        const uint32_t u1 = Te<true>::column(L, s[1], s[2], s[3], s[0], k[24]);
        const uint32_t u2 = Te<true>::column(L, s[2], s[3], s[0], s[1], k[25]);
        return (Te<true>::sub_at<1>(L, u1) | Te<true>::sub_at<0>(L, u2)) ^ ends;  // bits above 15 are for the caller's mask
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
        s[0] = c0 ^ Te<true>::e3<0>(L, w);
        s[1] = c1 ^ Te<true>::e2<1>(L, w);
        s[2] = xor3(c2, Te<true>::e3<0>(L, k1 ^ r), Te<true>::e1<2>(L, w));
        s[3] = c3 ^ Te<true>::e0<3>(L, w);
#pragma unroll
        for (int i = 0; i < 8; ++i) Te<true>::round(L, s, k + 4 * i);
        return (Te<true>::sub_at<3>(L, s[3]) | Te<true>::sub_at<2>(L, s[0]) | Te<true>::sub_at<1>(L, s[1]) | Te<true>::sub_at<0>(L, s[2])) ^ k43;
    }
};

static_assert(kStKey + LaneKey<false>::kWords <= kRecordWords, "a narrow record fits");
static_assert(kStKey + LaneKey<true>::kWords + 1 <= kRecordWords, "a wide record fits");

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
    build_tables<true>(a.t0, smem);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Lanes L{lane * 4, lane * 4 + 128, 256u};
    const uint32_t gwarp = blockIdx.x * (blockDim.x >> 5) + warp;
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    uint32_t* stock = a.stock + (size_t)gwarp * (kRecordBlockBytes / 4);
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
                if (lane < n) make_record<true, WIDE>(a.jobs, a.njobs, L, a.gidx_begin + base + lane, stock + lane);
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
                const Entry mine = it.pack(cur, which, k == 4);
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
                it.unpack(old, tgt, k == 4, cur, copy);
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
                        ItemT::store(bins + tgt, it.pack(item, which, k == 4));
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
                    ItemT::store(bins + tgt, it.pack(cur, which, k == 4));
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
                ItemT::store(bins + tgt, it.pack(cur, which, k == 4));
                it.unpack(old, tgt, k == 4, cur, which);
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
