// cf_binned.cuh -- large inserts by binning the batch to table segments.
//
// The work of a large insert is bringing each key to its bucket.  A batch of
// this path is binned by table segment in one or two passes without a
// histogram: hashed keys fill their segments evenly, so every bin has a fixed
// place with a few standard deviations of room, and a CTA takes its runs' places
// there with one atomic per bin and tile.  What does not fit (skewed batches,
// repeated keys) goes to the eviction list, which takes any key.  Entries are
// 4-byte ((bucket within the bin) << bits | tag) whenever that fits.
//
//   round 1: keys -> bins by primary bucket -> each segment staged in shared
//            memory, slots claimed by arrival rank (k_bin_insert); the entries
//            that find no slot are left at the front of their segment's bin;
//   round 2: those, by alternate bucket; round 3 (after a capped round 1): by
//            primary bucket again; what is left goes to the eviction kernels.
//
// Every count stays on the device: the host enqueues all launches of a batch
// and waits for none of them, unless the list is shorter than the batch (two waits,
// see list_room).  Used for batches whose slot order within a bucket
// is unspecified, in buckets of at most 16 slots; cf_segmented.cuh takes the rest.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "cf_segmented.cuh"

namespace cfb {

// Bins of one pass.  More bins mean shorter runs, and L2 takes only about 43 G
// partly written sectors per second: with 2048 bins (16-byte runs) a pass over
// 2^31 keys took 17 ms, with two passes of 256 bins the first takes 9.7.
constexpr uint32_t kBinMaxDigits = 512;
constexpr uint32_t kCursorStride = 8;  // one cursor per 32-byte sector: tiles take their places at the same time
constexpr int kBinThreads = 512;
constexpr int kBinInsertThreads = 256;
constexpr uint32_t kBinGroup = 256;  // segments whose leftovers a CTA gathers at a time

enum BinSource : int { BIN_KEYS = 0, BIN_SPLIT = 1, BIN_LEFT = 2 };

// Geometry of one binned batch (bin_geometry).
struct BinGeom {
    int sbl;            // log2 buckets of a segment
    int l2;             // segment bits split off in a second pass (0: one pass)
    uint32_t nseg;      // segments
    uint32_t d1;        // bins of the first pass
    uint32_t room1;     // entries of a first-pass bin (two passes)
    uint32_t room2;     // entries of a segment's bin
    int entry_bytes1;   // bytes of a first-pass entry (two passes): 4 or 8
    int entry_bytes2;   // bytes of an entry of a segment's bin
    uint64_t ent[2];    // entries of the two bin buffers
};

inline int ilog2(uint64_t v) { return 63 - __builtin_clzll(v); }
// ceil(log2(v)) for v >= 1
inline int clog2(uint64_t v) { return v <= 1 ? 0 : ilog2(v - 1) + 1; }

// Geometry of a binned insert of m keys into nb buckets of bb bytes, or false where
// the path does not apply.  Segments are at most 64 KiB (three CTAs per SM), and
// smaller in a small table, so that every SM gets one (2^20 slots: 256 segments
// of 8 KiB take 6 us a round, 32 of 64 KiB took 45).
inline bool bin_geometry(uint64_t nb, uint64_t bb, int bits, uint32_t alt_policy, uint64_t m, BinGeom* g) {
    if (m == 0 || m >= (1ull << 31)) return false;
    if (nb > (1ull << 32)) return false;  // bucket indexes are 32-bit here
    int sbl = ilog2(std::min<uint64_t>(kSegBytes / bb, nb));
    while (sbl > 5 && ((nb - 1) >> sbl) + 1 < 256) --sbl;
    const uint64_t nseg = ((nb - 1) >> sbl) + 1;
    // two passes of equal fan-out past kBinMaxDigits segments
    int l2 = nseg > kBinMaxDigits ? clog2(nseg) / 2 : 0;
    if (l2 && bits < 32 && l2 + sbl + bits > 32 && sbl + bits < 32 && ((nseg - 1) >> (32 - bits - sbl)) + 1 <= kBinMaxDigits)
        l2 = 32 - bits - sbl;  // unless some more first-pass bins keep the entries between the passes at 4 bytes
    if ((1ull << l2) > kBinMaxDigits || ((nseg - 1) >> l2) + 1 > kBinMaxDigits) return false;
    g->sbl = sbl;
    g->l2 = l2;
    g->nseg = static_cast<uint32_t>(nseg);
    g->d1 = static_cast<uint32_t>(((nseg - 1) >> l2) + 1);
    g->entry_bytes2 = bits < 32 ? 4 : 8;  // (at most 13 bits of bucket: 64 KiB of 8-byte buckets)
    g->entry_bytes1 = g->entry_bytes2 == 4 && l2 + sbl + bits <= 32 ? 4 : 8;
    // Room of a bin: the mean of its keys plus six standard deviations.  The AddSub
    // policy's primary buckets are the first half of the table.  Where a bucket is a
    // 32-bit hash modulo a count that is no power of two, the first buckets get one
    // hash value more than the last, which counts in large tables: 0.4 % of a bin's
    // keys at 10^9 slots, against six deviations of 0.3 % (0.7 M keys had no room).
    const uint64_t range = alt_policy == ALT_ADDSUB ? (nb + 1) / 2 : nb;
    const uint64_t hashes = ((1ull << 32) + range - 1) / range;  // of a first bucket, of 2^32
    auto room = [&](int log2_buckets) {
        const double mean = std::min(static_cast<double>(m), static_cast<double>(m) * std::ldexp(static_cast<double>(hashes), log2_buckets - 32));
        return (static_cast<uint64_t>(mean + 6.0 * std::sqrt(mean) + 64.0) + 7) / 8 * 8;
    };
    const uint64_t r2 = room(sbl), r1 = room(sbl + l2);
    g->ent[0] = l2 ? g->d1 * r1 : nseg * r2;
    g->ent[1] = nseg * r2;
    if (g->ent[0] >= (1ull << 32) || g->ent[1] >= (1ull << 32)) return false;
    g->room1 = static_cast<uint32_t>(r1);
    g->room2 = static_cast<uint32_t>(r2);
    return true;
}

// Device workspace of a binned batch.
struct BinWork {
    void* ent[2];
    uint32_t* pay[2];            // payloads beside ent, or null
    // Eviction list, (alternate bucket << bits) | tag: first the entries that
    // found no room in a bin (at most list_room of them), then the last round's.
    // list, ent[0] and ent[1] lie one after the other: with list_room below the
    // batch size (two passes only) the list runs on into ent[0], which is free
    // in the last round, and its second buffer starts m entries in.  Such a list
    // never fills up: past it in the first round the batch is given up, and
    // entries the first round leaves are binned again only where all would fit.
    uint64_t* list;
    uint32_t* list_pay;
    uint64_t list_room;
    unsigned long long* h_cnt;   // pinned
    uint32_t* cursor;            // per round: d1 (two passes) and nseg entry counts
    uint32_t* left;              // per segment: entries left by the round
    unsigned long long* cnt;     // list lengths: no room in a bin, after the fast BFS, after BFS, the last round's; left by the first round
    uint32_t* full;              // known-full bucket bitmap, or null
    uint64_t zero_bytes;         // cursor, cnt and full, one after the other: zero at the start of a batch
    int sms;
    uint32_t round1_cap;         // CF_OPT_ROUND1_CAP (0 = automatic)
    bool fresh;                  // the table is all zeros
};

template <typename EO>
struct BinArgs {
    const void* src;            // BIN_KEYS: keys; else entries of bins, `src_cap` apart
    const uint32_t* src_pay;    // payloads beside the source entries
    const uint32_t* src_count;  // entries of each source bin (may exceed src_cap: the rest overflowed)
    uint32_t src_cap;
    uint32_t src_bins;
    uint64_t n;                 // BIN_KEYS: keys
    uint64_t nb_mask;
    int low;                    // bits of the bucket index an output entry keeps
    int left_sbl;               // BIN_LEFT: log2 buckets of a source segment
    uint32_t digits;            // output bins per source (BIN_SPLIT), else in all
    EO* dst;
    uint32_t* dst_pay;
    uint32_t* cursor;           // entries taken so far, per output bin
    uint32_t dst_cap;
    uint64_t* over;             // entries without room, keyed by alternate bucket
    uint32_t* over_pay;
    unsigned long long* over_count;
    uint64_t over_room;         // entries the list holds (past it, in the first round only, they are counted)
    int over_alt;               // the entries binned here are keyed by primary bucket
};

// Entries per thread of a full-size tile: two CTAs per SM.
template <bool PAY>
constexpr int bin_ipt() {
    return PAY ? 7 : 10;
}
// Bytes of a source entry that k_bin copies to shared memory ahead of its tile.
template <class C, int SRC, typename EI>
constexpr int bin_in_bytes() {
    return SRC == BIN_KEYS ? C::key_bytes : static_cast<int>(sizeof(EI));
}
// Shared memory of k_bin for `digits` bins.
template <class C, int SRC, typename EI, bool PAY, int IPT>
constexpr size_t bin_smem(uint32_t digits) {
    return static_cast<size_t>(kBinThreads) * IPT *
               (8 + bin_in_bytes<C, SRC, EI>() + (PAY ? 4 : 0) + (PAY && SRC != BIN_KEYS ? 4 : 0) + (SRC == BIN_LEFT ? 4 : 0)) +
           static_cast<size_t>(digits) * 8;
}

// Asynchronous copy of one 4- or 8-byte word to shared memory; a thread that
// copies only what it reads itself needs just bin_copies_done.
template <int BYTES>
__device__ __forceinline__ void bin_copy(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void bin_copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// An entry (bucket b, tag) that finds no room in its bin goes to the eviction list:
// one atomic for the lanes that come here together (with one each, the lists of
// batches full of repeated keys were bound by it).
template <class C, bool PAY, typename EO>
__device__ __forceinline__ void bin_append(const BinArgs<EO>& a, uint64_t b, uint32_t tag, uint32_t pay) {
    if (a.over_alt) {
        b = alt_bucket<C>(b, tag, a.nb_mask);
        tag = alt_tag<C>(tag);
    }
    const uint32_t lanes = __activemask(), lane = threadIdx.x & 31;
    unsigned long long to = 0;
    if (lane == static_cast<uint32_t>(__ffs(lanes)) - 1u)
        to = atomicAdd(a.over_count, static_cast<unsigned long long>(__popc(lanes)));
    to = __shfl_sync(lanes, to, __ffs(lanes) - 1) + __popc(lanes & ((1u << lane) - 1u));
    if (to < a.over_room) {
        a.over[to] = pack_entry<C>(b, tag);
        if constexpr (PAY) a.over_pay[to] = pay;
    }
}

// Not inlined in the large tiles' kernels, whose 64 registers it disturbs (0.4 % of a
// 2^28-slot fill); the small tiles' keep their 40 to 48 only without the call.
template <class C, bool PAY, typename EO>
__device__ __noinline__ void bin_no_room(const BinArgs<EO>& a, uint64_t b, uint32_t tag, uint32_t pay) {
    bin_append<C, PAY>(a, b, tag, pay);
}

// One binning pass.  A tile of kBinThreads * IPT entries is ranked within its
// bins by shared-memory atomics, its runs' places are taken from the bins'
// cursors, and the tile is staged in bin order and written out run by run.
// BIN_KEYS: the source is the key array, hashed here.
// BIN_SPLIT: the source is bins of an earlier pass, each split into `digits`.
// BIN_LEFT: the source is the entries an insert round left at the front of its
//           segments' bins; each is re-keyed by its other bucket.
// The ranking and staging are bound by the shared-memory pipe and the hashing
// by the multiplier, so the two are run together: a thread hashes the next tile's
// entries between the stores that stage this one's, and the tile after that is
// on its way to shared memory meanwhile.  What is left is split evenly between
// issue (about 90 instructions per key), the multiplier, the ALU and the
// shared-memory pipe, each half busy.  Per pass over 2.04 G keys (2^31 slots,
// 256 bins): keys to 8-byte entries 9.7 ms, those to 4-byte entries 7.4 ms; the
// histogram and scatter passes they replace took 13.5 and 9.0.  Over 255 M keys
// (2^28 slots, 4-byte entries between the passes): 1.16 and 0.74 ms for 1.7 and 1.1.
// Three CTAs of 40 registers with 7 entries per thread, or 256-thread CTAs, came
// within 3 %; hashing before the staging instead of between it cost 10 %.
template <class C, int SRC, typename EI, typename EO, bool PAY, int IPT>
__global__ void __launch_bounds__(kBinThreads, 2) k_bin(const __grid_constant__ BinArgs<EO> a) {
    constexpr int NT = kBinThreads;
    constexpr uint32_t TILE = NT * IPT;
    constexpr bool WIDE = sizeof(EO) == 8;
    constexpr int IN = bin_in_bytes<C, SRC, EI>();
    using In = typename std::conditional<IN == 4, uint32_t, uint64_t>::type;
    static_assert(kBinMaxDigits <= NT, "thread d places bin d");
    extern __shared__ __align__(16) unsigned char bin_raw[];
    uint64_t* stage = reinterpret_cast<uint64_t*>(bin_raw);  // 4 bin << 32 | entry, or (8-byte entries) bucket << bits | tag
    In* in = reinterpret_cast<In*>(stage + TILE);            // the next tile's entries
    uint32_t* off = reinterpret_cast<uint32_t*>(in + TILE);  // 8 x (counts, then first staged position of each bin)
    uint32_t* base = off + a.digits;                         // output index of staged position q = base + q
    uint32_t* stage_pay = base + a.digits;
    uint32_t* in_pay = stage_pay + (PAY ? TILE : 0);
    uint32_t* in_seg = in_pay + (PAY && SRC != BIN_KEYS ? TILE : 0);  // BIN_LEFT: the entry's segment
    __shared__ uint32_t s_warp[NT / 32];
    __shared__ uint32_t s_pref[SRC == BIN_LEFT ? kBinGroup + 1 : 1];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t low_mask = static_cast<uint32_t>((1ull << a.low) - 1ull);
    for (uint32_t d = tid; d < a.digits; d += NT) off[d] = 0;

    // f(j) for every entry j of this thread in a tile of `count`
    auto for_tile = [&](uint32_t count, auto f) {
        if (count == TILE) {
#pragma unroll
            for (int j = 0; j < IPT; ++j) f(j);
        } else {
#pragma unroll
            for (int j = 0; j < IPT; ++j)
                if (static_cast<uint32_t>(j * NT) + tid < count) f(j);
        }
    };
    // load(count, bin0): starts the copies of this CTA's next tile (count = 0: there is none);
    // bin0 is its first output bin.  Every thread of the CTA calls it.
    uint64_t at = SRC == BIN_KEYS ? static_cast<uint64_t>(blockIdx.x) * TILE : blockIdx.x;  // key, or tile of the bins
    const uint32_t tiles = SRC == BIN_SPLIT ? (a.src_cap + TILE - 1) / TILE : 0u;           // per source bin
    const uint32_t group = SRC == BIN_LEFT ? (a.src_bins + gridDim.x - 1) / gridDim.x : 0u;
    const uint32_t g1 = (blockIdx.x + 1) * group < a.src_bins ? (blockIdx.x + 1) * group : a.src_bins;
    uint32_t s0 = blockIdx.x * group, ns = 0, total = 0, first = 0;  // BIN_LEFT: segments gathered, entries taken
    uint64_t pay0 = 0, pay1 = 0;  // BIN_KEYS: first key of the tile placed, and of the one before
    auto load = [&](uint32_t& count, uint32_t& bin0) {
        count = 0;
        bin0 = 0;
        if constexpr (SRC == BIN_KEYS) {
            if (at < a.n) {
                count = a.n - at < TILE ? static_cast<uint32_t>(a.n - at) : TILE;
                const typename C::Key* keys = static_cast<const typename C::Key*>(a.src) + at;
                for_tile(count, [&](int j) { bin_copy<IN>(in + j * NT + tid, keys + j * NT + tid); });
            }
            at += static_cast<uint64_t>(gridDim.x) * TILE;
        } else if constexpr (SRC == BIN_SPLIT) {
            for (; at < static_cast<uint64_t>(a.src_bins) * tiles && !count; at += gridDim.x) {
                // every bin's first tile, then every bin's second: earlier keys stay earlier
                const uint32_t bin = static_cast<uint32_t>(at % a.src_bins), f = static_cast<uint32_t>(at / a.src_bins) * TILE;
                const uint32_t got = a.src_count[bin * kCursorStride];
                const uint32_t have = got < a.src_cap ? got : a.src_cap;
                if (f >= have) continue;
                count = have - f < TILE ? have - f : TILE;
                bin0 = bin * a.digits;
                const uint64_t e0 = static_cast<uint64_t>(bin) * a.src_cap + f;
                for_tile(count, [&](int j) {
                    bin_copy<IN>(in + j * NT + tid, static_cast<const EI*>(a.src) + e0 + j * NT + tid);
                    if constexpr (PAY) bin_copy<4>(in_pay + j * NT + tid, a.src_pay + e0 + j * NT + tid);
                });
            }
        } else {
            while (first >= total) {  // the next segments with leftovers
                s0 += ns;
                if (s0 >= g1) return;
                ns = g1 - s0 < kBinGroup ? g1 - s0 : kBinGroup;
                __syncthreads();
                const uint32_t v = tid < ns ? a.src_count[s0 + tid] : 0u;  // at most the segment's room
                const uint32_t incl = warp_inclusive_scan(v);
                if (lane == 31) s_warp[warp] = incl;
                __syncthreads();
                const uint32_t x = lane < NT / 32 ? s_warp[lane] : 0u;
                const uint32_t before = __shfl_sync(0xFFFFFFFFu, warp_inclusive_scan(x) - x, warp);
                if (tid < ns) s_pref[tid + 1] = before + incl;
                if (tid == 0) s_pref[0] = 0;
                __syncthreads();
                total = s_pref[ns];
                first = 0;
            }
            count = total - first < TILE ? total - first : TILE;
            for_tile(count, [&](int j) {
                const uint32_t k = first + j * NT + tid;
                uint32_t lo = 0, hi = ns;  // s_pref[lo] <= k < s_pref[lo + 1]
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (s_pref[mid] <= k) lo = mid; else hi = mid;
                }
                const uint64_t e0 = static_cast<uint64_t>(s0 + lo) * a.src_cap + (k - s_pref[lo]);
                in_seg[j * NT + tid] = s0 + lo;
                bin_copy<IN>(in + j * NT + tid, static_cast<const EI*>(a.src) + e0);
                if constexpr (PAY) bin_copy<4>(in_pay + j * NT + tid, a.src_pay + e0);
            });
            first += TILE;
        }
    };
    // Entry j of the tile in shared memory: its bin and its output entry.
    using Val = typename std::conditional<WIDE, uint64_t, uint32_t>::type;
    Val val[IPT];
    uint32_t dr[IPT];  // 4 bin, then 4 bin << 16 | 8 x rank within the tile's run of that bin
    static_assert(TILE * 8 <= 65536 && kBinMaxDigits * 4 <= 65536, "bin and rank in one word");
    auto word_at = [](uint32_t* p, uint32_t byte) -> uint32_t& {
        return *reinterpret_cast<uint32_t*>(reinterpret_cast<unsigned char*>(p) + byte);
    };
    uint32_t pv[PAY ? IPT : 1];
    auto place = [&](int j) {
        const uint32_t i = j * NT + tid;
        uint32_t b, tag;
        if constexpr (SRC == BIN_KEYS) {
            uint64_t b64;
            candidates<C>(in[i], a.nb_mask, b64, tag);
            b = static_cast<uint32_t>(b64);
            if constexpr (PAY) pv[PAY ? j : 0] = static_cast<uint32_t>(pay0) + i;
        } else {
            const EI e = in[i];
            tag = static_cast<uint32_t>(e) & C::tag_mask;
            b = static_cast<uint32_t>(e >> C::bits);
            if constexpr (SRC == BIN_LEFT) {
                const uint64_t full = (static_cast<uint64_t>(in_seg[i]) << a.left_sbl) | b;
                b = static_cast<uint32_t>(alt_bucket<C>(full, tag, a.nb_mask));
                tag = alt_tag<C>(tag);
            }
            if constexpr (PAY) pv[PAY ? j : 0] = in_pay[i];
        }
        dr[j] = (b >> a.low) * 4;
        if constexpr (WIDE)
            val[j] = pack_entry<C>(b, tag);
        else
            val[j] = ((b & low_mask) << C::bits) | tag;
    };

    uint32_t count, bin0, next_count = 0, next_bin0 = 0;
    pay0 = at;
    load(count, bin0);
    if (count) {
        bin_copies_done();
#pragma unroll
        for (int j = 0; j < IPT; ++j) place(j);
        pay1 = at;
        load(next_count, next_bin0);
    }
    while (count) {
        __syncthreads();  // counts are zero, the last tile is written out
        for_tile(count, [&](int j) { dr[j] = (dr[j] << 16) + atomicAdd(&word_at(off, dr[j]), 8u); });
        __syncthreads();
        // this thread's bin: its place from the cursor (not needed before the
        // write-out, so the latency is hidden), its staged position from a scan
        const uint32_t c = tid < a.digits ? off[tid] / 8 : 0u;
        const uint32_t g = c ? atomicAdd(&a.cursor[(bin0 + tid) * kCursorStride], c) : 0u;
        const uint32_t incl = warp_inclusive_scan(c);
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        const uint32_t x = lane < NT / 32 ? s_warp[lane] : 0u;
        const uint32_t pos = __shfl_sync(0xFFFFFFFFu, warp_inclusive_scan(x) - x, warp) + incl - c;
        if (tid < a.digits) off[tid] = pos * 8;
        __syncthreads();
        bin_copies_done();
        pay0 = pay1;
        auto put = [&](int j) {
            const uint32_t d4 = dr[j] >> 16, p8 = word_at(off, d4) + (dr[j] & 0xFFFFu);
            *reinterpret_cast<uint64_t*>(bin_raw + p8) =
                WIDE ? static_cast<uint64_t>(val[j]) : static_cast<uint64_t>(d4) << 32 | val[j];
            if constexpr (PAY) stage_pay[p8 / 8] = pv[PAY ? j : 0];
        };
        if (count == TILE) {
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                put(j);
                place(j);  // (past the next tile's end: not used)
            }
        } else {
#pragma unroll
            for (int j = 0; j < IPT; ++j) {
                if (static_cast<uint32_t>(j * NT) + tid < count) put(j);
                place(j);
            }
        }
        uint32_t after = 0, after_bin0 = 0;
        if (next_count) {
            pay1 = at;
            load(after, after_bin0);
        }
        if (tid < a.digits) base[tid] = (bin0 + tid) * a.dst_cap + g - pos;
        const bool any_over = __syncthreads_or(c && g + c > a.dst_cap);
        for (uint32_t d = tid; d < a.digits; d += NT) off[d] = 0;
        const uint64_t wide_mask = static_cast<uint64_t>(low_mask) << C::bits | C::tag_mask;
        auto out = [&](uint32_t q, bool check) {
            const uint64_t y = stage[q];
            const uint32_t d4 = WIDE ? static_cast<uint32_t>(y >> (C::bits + a.low)) * 4 : static_cast<uint32_t>(y >> 32);
            const EO e = WIDE ? static_cast<EO>(y & wide_mask) : static_cast<EO>(y);
            const uint32_t o = word_at(base, d4) + q;
            if (check && o - (bin0 + d4 / 4) * a.dst_cap >= a.dst_cap) {  // no room left in its bin
                const uint64_t b = (static_cast<uint64_t>(bin0 + d4 / 4) << a.low) | (static_cast<uint64_t>(e) >> C::bits);
                const uint32_t tag = static_cast<uint32_t>(e) & C::tag_mask;
                if constexpr (IPT <= 4)
                    bin_append<C, PAY>(a, b, tag, PAY ? stage_pay[q] : 0u);
                else
                    bin_no_room<C, PAY>(a, b, tag, PAY ? stage_pay[q] : 0u);
            } else {
                a.dst[o] = e;
                if constexpr (PAY) a.dst_pay[o] = stage_pay[q];
            }
        };
        if (any_over)
            for (uint32_t q = tid; q < count; q += NT) out(q, true);
        else
            for_tile(count, [&](int j) { out(j * NT + tid, false); });
        count = next_count;
        bin0 = next_bin0;
        next_count = after;
        next_bin0 = after_bin0;
    }
}

// Segment-staged insert from bins: one CTA per segment.  The segment arrives in
// shared memory by one bulk copy (FRESH: the table is all zeros and the segment
// starts as zeros), every entry claims a slot of its bucket by arrival rank (one
// shared-memory atomic add on the bucket's claim word, as in k_seg_insert), and
// the segment leaves by one bulk copy.  FRESH claim words are plain arrival
// counters, because the claimable slots are 0 .. cap - 1 in every bucket.
// Entries that find no slot are moved to the front of the bin they came from
// (a step's entries are all in registers before any is overwritten, so one
// barrier per step orders the two) and counted in left[s]; in the last round
// they go to `list`, from entry *list_first on, as (alternate bucket << bits | tag).
// Bound by the shared-memory pipe (an atomic and a store per entry).  First
// round of 2.04 G keys: 4.1 ms (7.8 in k_seg_insert, whose steps had three
// barriers and wrote 8-byte leftovers with the other bucket worked out in
// place); the second and third 1.8 and 1.5 (2.8 and 2.0).
template <class C, typename E, bool PAY, bool FRESH>
__global__ void __launch_bounds__(kBinInsertThreads, 3)
    k_bin_insert(DevTable t, E* ent, uint32_t* pay, const uint32_t* count, uint32_t room, uint32_t nseg, int sbl, int round,
                 uint32_t* left, uint32_t cap, int last, uint64_t* list, uint32_t* list_pay,
                 unsigned long long* list_count, const unsigned long long* list_first, uint32_t* full) {
    static_assert(C::bs <= 16, "claim words keep a 16-bit counter above a 16-slot mask");
    extern __shared__ __align__(16) uint64_t seg[];
    __shared__ __align__(8) uint64_t seg_bar;
    __shared__ uint32_t s_left;
    __shared__ unsigned long long s_base;
    constexpr int WPB = C::bucket_bytes / 8;
    constexpr int TB = C::bits / 8;
    constexpr int U = sizeof(E) == 4 ? (PAY ? 8 : 16) : 8;  // entries per thread and step
    constexpr uint32_t STEP = kBinInsertThreads * U;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const uint32_t s = blockIdx.x;
    const uint32_t got = count[s * kCursorStride];
    const uint32_t n = got < room ? got : room;
    if (n == 0) {
        if (tid == 0) left[s] = 0;
        return;
    }
    const uint32_t sb = 1u << sbl;
    uint32_t* claim = reinterpret_cast<uint32_t*>(seg + static_cast<size_t>(sb) * WPB);
    uint8_t* seg_bytes = reinterpret_cast<uint8_t*>(seg);
    uint64_t* gseg = reinterpret_cast<uint64_t*>(t.buckets + (static_cast<uint64_t>(s) << sbl) * C::bucket_bytes);
    // the last segment of a table whose bucket count is not a multiple of the segment is partial
    const uint64_t rest = t.nb_mask + 1 - (static_cast<uint64_t>(s) << sbl);
    const uint32_t nbk = rest < sb ? static_cast<uint32_t>(rest) : sb;
    const uint32_t words = nbk * WPB;
    const bool bulk = words % 2 == 0;  // a whole number of 16-byte units
    E* in = ent + static_cast<uint64_t>(s) * room;
    uint32_t* in_pay = PAY ? pay + static_cast<uint64_t>(s) * room : nullptr;
    if (tid == 0) {
        mbar_init(&seg_bar, 1);
        fence_mbar_init();
        s_left = 0;
    }
    E ev[U], nx[U];
    uint32_t pv[PAY ? U : 1], pn[PAY ? U : 1];
    auto fetch = [&](uint32_t b0, E(&e)[U], uint32_t(&p)[PAY ? U : 1]) {
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const uint32_t k = b0 + j * kBinInsertThreads + tid;
            e[j] = 0;
            if (k < n) e[j] = in[k];
            if constexpr (PAY) {
                p[j] = 0;
                if (k < n) p[j] = in_pay[k];
            }
        }
    };
    fetch(0, nx, pn);
    __syncthreads();
    if constexpr (FRESH) {
        for (uint32_t w = tid; w < words; w += kBinInsertThreads) seg[w] = 0;
        for (uint32_t b = tid; b < sb; b += kBinInsertThreads) claim[b] = 0;
    } else if (bulk) {
        if (tid == 0) {
            mbar_arrive_expect_tx(&seg_bar, words * 8u);
            bulk_g2s(seg, gseg, words * 8u, &seg_bar);
        }
        const bool staged = mbar_wait(&seg_bar, 0, kMbarPollLimit);
        if (__syncthreads_or(!staged)) {
            // the copy did not land within its poll bound: report it, give it a
            // second bounded wait, and leave the segment untouched
            if (tid == 0) {
                atomicOr(&t.ctr[CTR_ERROR], ERR_WAIT_LIMIT);
                left[s] = 0;
            }
            mbar_wait(&seg_bar, 0, kMbarPollLimit);
            return;
        }
    } else {
        for (uint32_t w = tid; w < words; w += kBinInsertThreads) seg[w] = gseg[w];
        __syncthreads();
    }
    auto build_claims = [&]() {
        for (uint32_t b = tid; b < sb; b += kBinInsertThreads)
            claim[b] = b < nbk ? claimable_slots<C>(empty_mask<C>(seg + static_cast<size_t>(b) * WPB), cap) : 0u;
    };
    if constexpr (!FRESH) build_claims();
    uint32_t n_ok = 0;
    for (uint32_t b0 = 0; b0 < n; b0 += STEP) {
#pragma unroll
        for (int j = 0; j < U; ++j) {
            ev[j] = nx[j];
            if constexpr (PAY) pv[j] = pn[j];
        }
        if (b0 + STEP < n) fetch(b0 + STEP, nx, pn);
        // claim words ready; every entry of this step is in registers, so its place in the bin may be overwritten
        __syncthreads();
        if constexpr (!FRESH) {
            static_assert(kRankBatch % STEP == 0, "claim batches hold whole steps");
            if (b0 != 0 && b0 % kRankBatch == 0) {  // before an arrival counter can wrap
                build_claims();
                __syncthreads();
            }
        }
        uint32_t miss = 0;
#pragma unroll
        for (int j = 0; j < U; ++j) {
            if (b0 + j * kBinInsertThreads + tid < n) {
                const uint32_t fp = static_cast<uint32_t>(ev[j]) & C::tag_mask;
                const uint32_t lb = static_cast<uint32_t>(ev[j] >> C::bits);
                uint32_t slot;
                bool ok;
                if constexpr (FRESH) {
                    slot = atomicAdd(&claim[lb], 1u);
                    ok = slot < cap;
                } else {
                    const uint32_t old = atomicAdd(&claim[lb], 1u << 16);
                    const uint32_t m = old & 0xFFFFu, r = old >> 16;
                    ok = r < static_cast<uint32_t>(__popc(m));
                    // claimable slots are usually one run of bits: the r-th is low + r
                    const uint32_t low = static_cast<uint32_t>(__ffs(m)) - 1u, run = m >> (low & 31u);
                    slot = low + r;
                    if (ok && (run & (run + 1u)) != 0) slot = nth_set_bit16(m, r);
                }
                if (ok) {
                    uint8_t* at = seg_bytes + (static_cast<size_t>(lb) * C::bucket_bytes + slot * TB);
                    if constexpr (TB == 1)
                        *at = static_cast<uint8_t>(fp);
                    else if constexpr (TB == 2)
                        *reinterpret_cast<uint16_t*>(at) = static_cast<uint16_t>(fp);
                    else
                        *reinterpret_cast<uint32_t*>(at) = fp;
                    ++n_ok;
                } else {
                    miss |= 1u << j;
                }
            }
        }
        const uint32_t cnt = __popc(miss);
        const uint32_t incl = warp_inclusive_scan(cnt);
        uint32_t o = 0;
        if (lane == 31 && incl) o = atomicAdd(&s_left, incl);
        o = __shfl_sync(0xFFFFFFFFu, o, 31) + incl - cnt;
        if (miss) {
#pragma unroll
            for (int j = 0; j < U; ++j) {
                if ((miss >> j) & 1u) {
                    in[o] = ev[j];
                    if constexpr (PAY) in_pay[o] = pv[j];
                    ++o;
                }
            }
        }
    }
    fence_proxy_async_smem();  // this thread's tag stores, before the bulk copy reads them
    __syncthreads();
    if (bulk && tid == 0) {
        bulk_s2g(gseg, seg, words * 8u);
        bulk_commit();
    }
    if (!bulk)
        for (uint32_t w = tid; w < words; w += kBinInsertThreads) gseg[w] = seg[w];
    if (full && cap >= static_cast<uint32_t>(C::bs)) {
        // an uncapped round's full buckets, one bit each (sb is a multiple of 32 whenever the bitmap is kept)
        for (uint32_t c0 = 0; c0 < sb; c0 += kBinInsertThreads) {
            const uint32_t b = c0 + tid;
            bool is_full = false;
            if (b < nbk) {
                const uint32_t cw = claim[b];
                is_full = FRESH ? cw >= cap : (cw >> 16) >= static_cast<uint32_t>(__popc(cw & 0xFFFFu));
            }
            const uint32_t word = __ballot_sync(0xFFFFFFFFu, is_full);
            if (lane == 0 && b < sb) full[((static_cast<uint64_t>(s) << sbl) + b) >> 5] = word;
        }
    }
    const uint32_t nl = s_left;
    if (!last) {
        if (tid == 0) left[s] = nl;
    } else if (nl) {
        if (tid == 0) s_base = *list_first + atomicAdd(list_count, static_cast<unsigned long long>(nl));
        __syncthreads();  // also: every leftover is written
        for (uint32_t k = tid; k < nl; k += kBinInsertThreads) {
            const E e = in[k];
            uint32_t tag = static_cast<uint32_t>(e) & C::tag_mask;
            uint64_t b = (static_cast<uint64_t>(s) << sbl) | (static_cast<uint64_t>(e) >> C::bits);
            if (round != 2) {  // keyed by primary bucket
                b = alt_bucket<C>(b, tag, t.nb_mask);
                tag = alt_tag<C>(tag);
            }
            list[s_base + k] = pack_entry<C>(b, tag);
            if constexpr (PAY) list_pay[s_base + k] = in_pay[k];
        }
    }
    flush_counters(t.ctr, {{round == 2 ? CTR_SECONDARY : CTR_PRIMARY, static_cast<int32_t>(n_ok)},
                           {CTR_OCCUPIED, static_cast<int32_t>(n_ok)}});
    if (tid == 0) bulk_wait_all();
}

// Adds the entries that a round left in its segments' bins to *total.
static __global__ void __launch_bounds__(256) k_bin_left(const uint32_t* left, uint32_t nseg, unsigned long long* total) {
    uint32_t n = 0;
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < nseg; s += gridDim.x * blockDim.x) n += left[s];
    flush_counters(total, {{0, static_cast<int32_t>(n)}});
}

// Moves them to the list instead, keyed by alternate bucket: a warp per segment.
// For a list of half the batch that the next rounds might fill.
template <class C, typename E, bool PAY>
__global__ void __launch_bounds__(256) k_bin_to_list(const E* ent, const uint32_t* pay, const uint32_t* left, uint32_t room,
                                                     uint32_t nseg, int sbl, uint64_t nb_mask, uint64_t* list,
                                                     uint32_t* list_pay, unsigned long long* list_count) {
    const uint32_t lane = threadIdx.x & 31, nwarps = gridDim.x * (blockDim.x / 32);
    for (uint32_t s = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; s < nseg; s += nwarps) {
        const uint32_t n = left[s];
        if (n == 0) continue;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(list_count, static_cast<unsigned long long>(n));
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        for (uint32_t k = lane; k < n; k += 32) {
            const E e = ent[static_cast<uint64_t>(s) * room + k];
            const uint32_t tag = static_cast<uint32_t>(e) & C::tag_mask;
            const uint64_t b = (static_cast<uint64_t>(s) << sbl) | (static_cast<uint64_t>(e) >> C::bits);
            list[base + k] = pack_entry<C>(alt_bucket<C>(b, tag, nb_mask), alt_tag<C>(tag));
            if constexpr (PAY) list_pay[base + k] = pay[static_cast<uint64_t>(s) * room + k];
        }
    }
}

// The entries that found no room in a bin, keyed by alternate bucket: neither
// bucket has been tried, so both are; a stored key's entry is zeroed, the others
// stay in the list for the eviction kernels, which take many more keys at a time
// (evicting here, a thread per key: fills of 2^26 slots to 0.6 with half the batch
// repeats of 10^4 keys, BFS, 351 ms; 257 like this, 272 segment-staged).
template <class C>
__global__ void __launch_bounds__(256) k_bin_over(DevTable t, uint64_t* ent, const unsigned long long* n_dev) {
    const uint64_t m = *n_dev;
    uint32_t n_prim = 0, n_sec = 0;
    bool err = false;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < m;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const uint64_t e = ent[i];
        const uint32_t fp2 = static_cast<uint32_t>(e) & C::tag_mask, fp1 = alt_tag<C>(fp2);
        const uint64_t i2 = e >> C::bits, i1 = alt_bucket<C>(i2, fp2, t.nb_mask);
        uint64_t c[C::nchunks];
        uint64_t* bw = bucket_words<C>(t, i1);
        load_rlx<C::bucket_bytes>(bw, c);
        if (try_insert<C>(bw, c, fp1, err)) {
            ++n_prim;
            ent[i] = 0;
            continue;
        }
        bw = bucket_words<C>(t, i2);
        load_rlx<C::bucket_bytes>(bw, c);
        if (try_insert<C>(bw, c, fp2, err)) {
            ++n_sec;
            ent[i] = 0;
        }
    }
    flush_counters(t.ctr, {{CTR_OCCUPIED, static_cast<int32_t>(n_prim + n_sec)},
                           {CTR_PRIMARY, static_cast<int32_t>(n_prim)},
                           {CTR_SECONDARY, static_cast<int32_t>(n_sec)}});
    if (__any_sync(0xFFFFFFFFu, err) && (threadIdx.x & 31) == 0) atomicOr(&t.ctr[CTR_ERROR], ERR_CAS_LIMIT);
}

}  // namespace cfb
