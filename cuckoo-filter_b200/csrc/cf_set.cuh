// cf_set.cuh -- batched execution over many filters (a filter set).
//
// Thousands of independent filters with uneven key batches run in ONE launch
// of a persistent kernel.  The work list lives in device memory: item j is the
// key range [offs[j], offs[j+1]) of the concatenated key buffer, destined for
// filter filt[j] (offs is monotonic, offs[n_items] = total keys).  The grid
// strides over tiles of the concatenated keys; a CTA finds the items of its
// tile's first and last key by binary search over offs, and each thread searches
// between those and walks forward, so no per-item scratch or host-side tiling
// is needed and the launch can be captured in a CUDA graph and replayed with
// new keys in the same buffers.
//
// Per-key semantics are the single-filter kernels' (cf_kernels.cuh): the
// reference's insert / contains / remove (CuckooFilter.cuh:805-1116) applied
// to the filter the key belongs to.  Counters are per filter; each count is added
// with one atomic per run of lanes whose keys belong to one filter (one prefix
// scan finds the runs' sums), in the eviction with one per distinct filter
// (__match_any_sync).
//
// Tunables (template parameters, picked by the set's autotuner): KPT keys per
// thread, and for lookups the probe width W: W lanes cooperate on one key,
// each loading bucket_bytes / W bytes of each bucket, and vote by ballot.
#pragma once

#include <cstdint>

#include "cf_kernels.cuh"

namespace cfb {

// Item of key k in [lo, hi): the largest j with offs[j] <= k (empty items are skipped).
__device__ __forceinline__ uint32_t set_find_item(const uint64_t* __restrict__ offs, uint32_t lo, uint32_t hi, uint64_t k) {
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (offs[mid] <= k) lo = mid; else hi = mid;
    }
    return lo;
}

// The same over all items by the 32 lanes of a warp: four loads one after the other
// for 10^5 items where the search above makes 17.
__device__ __forceinline__ uint32_t set_find_item_warp(const uint64_t* __restrict__ offs, uint32_t n_items, uint64_t k) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0, hi = n_items;
    while (lo + 1 < hi) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint64_t at = lo + static_cast<uint64_t>(lane + 1) * step;
        const uint32_t le = __ballot_sync(0xFFFFFFFFu, at < hi && offs[at] <= k);
        const uint32_t c = static_cast<uint32_t>(__ffs(~le)) - 1u;  // (the last lane's is past hi)
        const uint32_t end = hi - lo;
        hi = (c + 1) * static_cast<uint64_t>(step) < end ? lo + (c + 1) * step : hi;
        lo += c * step;
    }
    return lo;
}

// Items of the tile [first, last]: range[0] of its first key, range[1] past that
// of its last (which is past range[0] whatever offs holds: both searches make the
// same probes until the one for the later key goes further).  Every thread of the
// CTA calls it, between two barriers of its own.
__device__ __forceinline__ void set_tile_items(const uint64_t* __restrict__ offs, uint32_t n_items, uint64_t first,
                                               uint64_t last, uint32_t (&range)[2]) {
    __syncthreads();
    const uint32_t warp = threadIdx.x / 32, lane = threadIdx.x & 31;
    if (warp == 0) {
        const uint32_t a = set_find_item_warp(offs, n_items, first);
        if (lane == 0) range[0] = a;
    }
    if (warp == (blockDim.x > 32 ? 1u : 0u)) {
        const uint32_t b = set_find_item_warp(offs, n_items, last) + 1;
        if (lane == 0) range[1] = b;
    }
    __syncthreads();
}

// A thread's walk over the items of its consecutive keys.
struct SetWalk {
    uint32_t item;
    uint64_t end;  // first key past the item (and past the empty ones after it)
    __device__ __forceinline__ SetWalk(const uint64_t* __restrict__ offs, const uint32_t (&range)[2], uint64_t k)
        : item(set_find_item(offs, range[0], range[1], k)), end(offs[item + 1]) {}
    // moves to the item of key k; true when that is another one
    __device__ __forceinline__ bool to(const uint64_t* __restrict__ offs, uint32_t n_items, uint64_t k) {
        if (k < end) return false;
        while (item + 1 < n_items && offs[item + 1] <= k) ++item;
        end = offs[item + 1];
        return true;
    }
};

constexpr uint64_t ERR_BAD_FILTER = 4;  // a work item named a filter outside the set

// Filter of item j, or n_filters (invalid) when the work list names a filter
// outside the set; such keys are skipped and flagged.
__device__ __forceinline__ uint32_t set_filter(const uint32_t* __restrict__ filt, uint32_t item, uint32_t n_filters) {
    const uint32_t f = filt[item];
    return f < n_filters ? f : n_filters;
}

// Adds each lane's values to the counters of its filter f: one atomic per
// counter when the active lanes share a filter, else one per distinct filter.
// All lanes of the warp must call it.
template <int N>
__device__ __forceinline__ void set_add_ctrs(const DevTable* __restrict__ descs, uint32_t f, bool active,
                                             const CounterAdd (&a)[N]) {
    const uint32_t lane = threadIdx.x & 31, act = __ballot_sync(0xFFFFFFFFu, active);
    if (!act) return;
    const uint32_t f0 = __shfl_sync(0xFFFFFFFFu, f, __ffs(act) - 1);
    uint32_t peers = act;
    const bool one = __all_sync(0xFFFFFFFFu, !active || f == f0);
    if (!one) peers = __match_any_sync(0xFFFFFFFFu, active ? f : 0xFFFFFFFFu);
    const bool leader = active && lane == static_cast<uint32_t>(__ffs(peers) - 1);
#pragma unroll
    for (int i = 0; i < N; ++i) {
        int32_t s = 0;
        if (one) {
            s = __reduce_add_sync(0xFFFFFFFFu, active ? a[i].v : 0);
        } else {
            for (uint32_t m = peers; m; m &= m - 1) s += __shfl_sync(peers, a[i].v, __ffs(m) - 1);
        }
        if (leader && s) atomicAdd(&descs[f].ctr[a[i].idx], static_cast<unsigned long long>(static_cast<long long>(s)));
    }
}

// Adds each lane's counts of its filter f, p and q (at most 32 each), where lanes of
// one filter mostly lie side by side: one atomic per counter and run of such lanes,
// add(ctr, sum of p, sum of q).  The runs' sums come from one prefix scan, so that
// warps of many small items do no more than others.  All lanes of the warp must call it.
template <class Add>
__device__ __forceinline__ void set_add_runs(const DevTable* __restrict__ descs, uint32_t f, bool active, uint32_t p,
                                             uint32_t q, Add add) {
    const uint32_t lane = threadIdx.x & 31, act = __ballot_sync(0xFFFFFFFFu, active);
    if (!act) return;
    const uint32_t g = active ? f : 0xFFFFFFFFu, before = __shfl_up_sync(0xFFFFFFFFu, g, 1);
    const uint32_t heads = __ballot_sync(0xFFFFFFFFu, lane == 0 || g != before);
    const uint32_t incl = warp_inclusive_scan(active ? p << 16 | q : 0u);
    const uint32_t prior = __shfl_up_sync(0xFFFFFFFFu, incl, 1);
    const uint32_t next = lane < 31 ? heads & (0xFFFFFFFEu << lane) : 0u;  // heads past this lane
    const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, next ? __ffs(next) - 2 : 31) - (lane ? prior : 0u);
    if (active && ((heads >> lane) & 1u) && total) add(descs[f].ctr, total >> 16, total & 0xFFFFu);
}

// Keys of a thread that are probed together: their bucket loads overlap, and two
// images leave registers for twice the warps that four would.
template <int KPT>
constexpr int set_batch() {
    return KPT < 2 ? 1 : 2;
}

// containsMany over the set, W = 1: each thread owns KPT consecutive keys.
// Bound by instruction issue: 512 filters of 1 K to 1 M slots, 14.2 M keys, took
// 219 us with a binary search over all items per thread, four images per
// thread and single-byte stores, and take 150.
template <class C, int KPT>
__global__ void __launch_bounds__(512) k_set_contains1(const DevTable* __restrict__ descs,
                                                       const uint32_t* __restrict__ filt,
                                                       const uint64_t* __restrict__ offs, uint32_t n_items, uint32_t n_filters,
                                                       const typename C::Key* __restrict__ keys, uint64_t n,
                                                       uint8_t* __restrict__ out, unsigned long long* err_flag) {
    constexpr int B = set_batch<KPT>();
    __shared__ uint32_t s_items[2];
    const uint64_t tile = static_cast<uint64_t>(blockDim.x) * KPT;
    const bool keys_vec = reinterpret_cast<uintptr_t>(keys) % (KPT * C::key_bytes < 32 ? KPT * C::key_bytes : 32) == 0;
    const bool out_vec = reinterpret_cast<uintptr_t>(out) % KPT == 0;
    bool bad = false;
    for (uint64_t base = blockIdx.x * tile; base < n; base += static_cast<uint64_t>(gridDim.x) * tile) {
        set_tile_items(offs, n_items, base, (base + tile < n ? base + tile : n) - 1, s_items);
        const uint64_t k0 = base + static_cast<uint64_t>(threadIdx.x) * KPT;
        if (k0 >= n) continue;
        uint64_t key[KPT];
        load_keys<C, KPT>(keys, k0, n, keys_vec, key);
        SetWalk walk(offs, s_items, k0);
        uint32_t f = set_filter(filt, walk.item, n_filters);
        DevTable cur = descs[f < n_filters ? f : 0];
        uint32_t hit = 0;
#pragma unroll
        for (int g = 0; g < KPT; g += B) {
            uint32_t live = 0;  // keys that exist and name a filter of the set
            uint8_t* tb[B];
            uint64_t mask[B], b[B];
            uint32_t fp[B];
            uint64_t c[B][C::nchunks];
#pragma unroll
            for (int j = 0; j < B; ++j) {
                const uint64_t k = k0 + g + j;
                if (k >= n) continue;
                if (walk.to(offs, n_items, k)) {
                    f = set_filter(filt, walk.item, n_filters);
                    cur = descs[f < n_filters ? f : 0];
                }
                if (f == n_filters) {
                    bad = true;
                    continue;
                }
                live |= 1u << j;
                tb[j] = cur.buckets;
                mask[j] = cur.nb_mask;
                candidates<C>(key[g + j], mask[j], b[j], fp[j]);
                load_nc<C::bucket_bytes>(tb[j] + b[j] * C::bucket_bytes, c[j]);
            }
            uint32_t in = 0;
#pragma unroll
            for (int j = 0; j < B; ++j)
                if (((live >> j) & 1u) && has_tag<C>(c[j], fp[j])) in |= 1u << j;
#pragma unroll
            for (int j = 0; j < B; ++j) {
                if (((live & ~in) >> j) & 1u) {
                    b[j] = alt_bucket<C>(b[j], fp[j], mask[j]);
                    load_nc<C::bucket_bytes>(tb[j] + b[j] * C::bucket_bytes, c[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < B; ++j)
                if ((((live & ~in) >> j) & 1u) && has_tag<C>(c[j], alt_tag<C>(fp[j]))) in |= 1u << j;
            hit |= in << g;
        }
        store_results<KPT>(out, k0, n, out_vec, hit);
    }
    if (bad) atomicOr(err_flag, ERR_BAD_FILTER);
}

// containsMany over the set, W lanes per key (W in {2, 4, 8}, a divisor of
// the bucket's 4-byte words): each group of W lanes owns KPT consecutive keys;
// lane r of the group loads bytes [r*PB, (r+1)*PB) of each bucket.
template <class C, int KPT, int W>
__global__ void __launch_bounds__(512) k_set_containsW(const DevTable* __restrict__ descs,
                                                       const uint32_t* __restrict__ filt,
                                                       const uint64_t* __restrict__ offs, uint32_t n_items, uint32_t n_filters,
                                                       const typename C::Key* __restrict__ keys, uint64_t n,
                                                       uint8_t* __restrict__ out, unsigned long long* err_flag) {
    constexpr int PB = C::bucket_bytes / W;
    bool bad = false;
    static_assert(PB == 4 || PB == 8, "a lane loads 4 or 8 bytes of a bucket");
    const uint32_t lane = threadIdx.x & 31, r = lane % W;
    const uint32_t gshift = lane - r;  // first lane of the group
    const uint32_t gmask = ((1u << W) - 1u) << gshift;
    const uint64_t groups = blockDim.x / W;
    const uint64_t tile = groups * KPT;
    for (uint64_t base = blockIdx.x * tile; base < n; base += static_cast<uint64_t>(gridDim.x) * tile) {
        const uint64_t k0 = base + static_cast<uint64_t>(threadIdx.x / W) * KPT;
        uint32_t item = k0 < n ? set_find_item(offs, 0, n_items, k0) : 0;
        DevTable t[KPT];
        uint64_t b[KPT];
        uint32_t fp[KPT];
        uint64_t piece[KPT];
        uint32_t valid = 0;
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            const uint64_t k = k0 + j;
            piece[j] = 0;
            fp[j] = 1;
            if (k < n) {
                while (item + 1 < n_items && offs[item + 1] <= k) ++item;
                const uint32_t f = set_filter(filt, item, n_filters);
                if (f == n_filters) {
                    bad = true;
                    continue;
                }
                valid |= 1u << j;
                t[j] = descs[f];
                candidates<C>(static_cast<uint64_t>(keys[k]), t[j].nb_mask, b[j], fp[j]);
                piece[j] = load_piece<PB>(t[j].buckets + b[j] * C::bucket_bytes + r * PB);
            }
        }
        uint32_t hit = 0;
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            const bool mine = ((valid >> j) & 1u) && piece_has<C, PB>(piece[j], fp[j]);
            if (__ballot_sync(0xFFFFFFFFu, mine) & gmask) hit |= 1u << j;
        }
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            if (((valid >> j) & 1u) && !((hit >> j) & 1u)) {
                b[j] = alt_bucket<C>(b[j], fp[j], t[j].nb_mask);
                fp[j] = alt_tag<C>(fp[j]);
                piece[j] = load_piece<PB>(t[j].buckets + b[j] * C::bucket_bytes + r * PB);
            }
        }
#pragma unroll
        for (int j = 0; j < KPT; ++j) {
            const bool mine = ((valid >> j) & 1u) && !((hit >> j) & 1u) && piece_has<C, PB>(piece[j], fp[j]);
            if (__ballot_sync(0xFFFFFFFFu, mine) & gmask) hit |= 1u << j;
            if (r == 0 && k0 + j < n) out[k0 + j] = static_cast<uint8_t>((hit >> j) & 1u);
        }
    }
    if (bad) atomicOr(err_flag, ERR_BAD_FILTER);
}

// deleteMany over the set: each thread owns KPT consecutive keys.  The keys of
// the thread's first filter are worked on together; those past the filter's end
// (a few threads per item) follow one at a time, so the common path keeps one
// table descriptor in registers.  Items of a few keys put several filters into a
// thread: 1.3 M keys of 10^5 filters, four keys per thread, took 62 us with one
// bucket load in flight, 110 with the warp's counts matched for every key past the
// first filter, and take 65.
template <class C, int KPT>
__global__ void __launch_bounds__(512, 2) k_set_delete(const DevTable* __restrict__ descs, const uint32_t* __restrict__ filt,
                                                       const uint64_t* __restrict__ offs, uint32_t n_items,
                                                       uint32_t n_filters, const typename C::Key* __restrict__ keys, uint64_t n,
                                                       uint8_t* __restrict__ out, unsigned long long* err_flag) {
    constexpr int B = set_batch<KPT>();
    __shared__ uint32_t s_items[2];
    const uint64_t tile = static_cast<uint64_t>(blockDim.x) * KPT;
    const bool keys_vec = reinterpret_cast<uintptr_t>(keys) % (KPT * C::key_bytes < 32 ? KPT * C::key_bytes : 32) == 0;
    const bool out_vec = reinterpret_cast<uintptr_t>(out) % KPT == 0;
    bool err = false, bad = false;
    for (uint64_t base = blockIdx.x * tile; base < n; base += static_cast<uint64_t>(gridDim.x) * tile) {
        set_tile_items(offs, n_items, base, (base + tile < n ? base + tile : n) - 1, s_items);
        const uint64_t k0 = base + static_cast<uint64_t>(threadIdx.x) * KPT;
        const uint32_t have = k0 < n ? (n - k0 < KPT ? static_cast<uint32_t>(n - k0) : KPT) : 0u;
        uint64_t key[KPT];
        if (have) load_keys<C, KPT>(keys, k0, n, keys_vec, key);
        SetWalk walk(offs, s_items, have ? k0 : base);
        uint32_t f = set_filter(filt, walk.item, n_filters);
        bad |= have && f == n_filters;
        const DevTable t = descs[f < n_filters ? f : 0];
        const uint32_t here = !have ? 0u : walk.end - k0 < have ? static_cast<uint32_t>(walk.end - k0) : have;
        const uint32_t live = f < n_filters ? (1u << here) - 1u : 0u;  // keys of the first filter
        uint32_t gone = 0;
#pragma unroll
        for (int g = 0; g < KPT; g += B) {
            uint64_t b[B];
            uint32_t fp[B];
            uint64_t c[B][C::nchunks];
#pragma unroll
            for (int j = 0; j < B; ++j) {
                if ((live >> (g + j)) & 1u) {
                    candidates<C>(key[g + j], t.nb_mask, b[j], fp[j]);
                    load_rlx<C::bucket_bytes>(bucket_words<C>(t, b[j]), c[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < B; ++j)
                if (((live >> (g + j)) & 1u) && try_remove<C>(bucket_words<C>(t, b[j]), c[j], fp[j], err)) gone |= 1u << (g + j);
#pragma unroll
            for (int j = 0; j < B; ++j) {
                if (((live & ~gone) >> (g + j)) & 1u) {
                    b[j] = alt_bucket<C>(b[j], fp[j], t.nb_mask);
                    load_rlx<C::bucket_bytes>(bucket_words<C>(t, b[j]), c[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < B; ++j)
                if ((((live & ~gone) >> (g + j)) & 1u) && !err &&
                    try_remove<C>(bucket_words<C>(t, b[j]), c[j], alt_tag<C>(fp[j]), err))
                    gone |= 1u << (g + j);
        }
        set_add_runs(descs, f, live != 0, __popc(gone), 0u, [](unsigned long long* ctr, uint32_t r, uint32_t) {
            atomicAdd(&ctr[CTR_REMOVED], static_cast<unsigned long long>(r));
            atomicAdd(&ctr[CTR_OCCUPIED], ~static_cast<unsigned long long>(r) + 1ull);
        });
        if (here < have) {  // keys past the first filter
            uint32_t r = 0;
            DevTable t2{};
            auto flush = [&]() {
                if (!r) return;
                atomicAdd(&t2.ctr[CTR_REMOVED], static_cast<unsigned long long>(r));
                atomicAdd(&t2.ctr[CTR_OCCUPIED], ~static_cast<unsigned long long>(r) + 1ull);
                r = 0;
            };
            for (uint32_t j = here; j < have; ++j) {
                if (walk.to(offs, n_items, k0 + j)) {
                    flush();
                    f = set_filter(filt, walk.item, n_filters);
                    bad |= f == n_filters;
                    if (f < n_filters) t2 = descs[f];
                }
                if (f == n_filters) continue;
                uint64_t b;
                uint32_t fp;
                uint64_t c[C::nchunks];
                candidates<C>(static_cast<uint64_t>(keys[k0 + j]), t2.nb_mask, b, fp);
                load_rlx<C::bucket_bytes>(bucket_words<C>(t2, b), c);
                bool ok = try_remove<C>(bucket_words<C>(t2, b), c, fp, err);
                if (!ok && !err) {
                    b = alt_bucket<C>(b, fp, t2.nb_mask);
                    load_rlx<C::bucket_bytes>(bucket_words<C>(t2, b), c);
                    ok = try_remove<C>(bucket_words<C>(t2, b), c, alt_tag<C>(fp), err);
                }
                if (ok) {
                    gone |= 1u << j;
                    ++r;
                }
            }
            flush();
        }
        if (have && out) store_results<KPT>(out, k0, n, out_vec, gone);
    }
    if (__any_sync(0xFFFFFFFFu, err) && (threadIdx.x & 31) == 0) atomicOr(err_flag, ERR_CAS_LIMIT);
    if (bad) atomicOr(err_flag, ERR_BAD_FILTER);
}

// insertMany over the set: each thread owns KPT consecutive keys; first empty
// slot of the primary, else of the alternate bucket; keys whose two buckets
// are full are parked per warp and evicted 32 at a time, one per lane (as
// k_insert does).
// Bound by instruction issue and by the compare-and-swaps' latency.  The same
// 14.2 M keys took 1041 us with one bucket load in flight per thread and three
// matched counter updates per key; 604 like this, 472 with the slot masks of
// cf_kernels.cuh.  Two CTAs of 512 threads (64 registers, some of them spilled in
// the eviction) beat the 128-register form, 765 us.
template <class C, int KPT>
__global__ void __launch_bounds__(512, 2) k_set_insert(const DevTable* __restrict__ descs, const uint32_t* __restrict__ filt,
                                                       const uint64_t* __restrict__ offs, uint32_t n_items,
                                                       uint32_t n_filters, const typename C::Key* __restrict__ keys, uint64_t n,
                                                       uint8_t* __restrict__ out, uint32_t policy_bfs, uint32_t max_ev,
                                                       unsigned long long* err_flag) {
    constexpr int B = set_batch<KPT>();
    constexpr int kBuf = 32 + 32 * KPT;
    __shared__ uint64_t s_defer[16 * kBuf];
    __shared__ uint32_t s_items[2];
    uint64_t* buf = s_defer + (threadIdx.x >> 5) * kBuf;
    const uint32_t lane = threadIdx.x & 31;
    uint32_t pending = 0;
    bool err = false, bad = false;
    const uint64_t tile = static_cast<uint64_t>(blockDim.x) * KPT;
    const bool keys_vec = reinterpret_cast<uintptr_t>(keys) % (KPT * C::key_bytes < 32 ? KPT * C::key_bytes : 32) == 0;
    const bool out_vec = reinterpret_cast<uintptr_t>(out) % KPT == 0;

    // evict the parked key index idx (or nothing when !v); warp-uniform call
    auto evict_parked = [&](uint64_t idx, bool v) {
        uint32_t f = 0;
        bool ok = false;
        EvictStats st;
        if (v) {
            // parked keys passed the filter check when they were first tried
            f = set_filter(filt, set_find_item(offs, 0, n_items, idx), n_filters);
            ok = evict_key<C>(descs[f], static_cast<uint64_t>(keys[idx]), policy_bfs, max_ev, st, err);
            if (ok && out) out[idx] = 1;
        }
        set_add_ctrs(descs, f, v,
                     {{CTR_EVICTED_INSERTS, 1},
                      {CTR_FAILED, ok ? 0 : 1},
                      {CTR_EVICTIONS, static_cast<int32_t>(st.evictions)},
                      {CTR_LOST, static_cast<int32_t>(st.lost)},
                      {CTR_DUP, static_cast<int32_t>(st.dup)},
                      {CTR_OCCUPIED, static_cast<int32_t>((ok ? 1u : 0u) - st.lost + st.dup)}});
    };

    for (uint64_t base = blockIdx.x * tile; base < n; base += static_cast<uint64_t>(gridDim.x) * tile) {
        set_tile_items(offs, n_items, base, (base + tile < n ? base + tile : n) - 1, s_items);
        const uint64_t k0 = base + static_cast<uint64_t>(threadIdx.x) * KPT;
        const uint32_t have = k0 < n ? (n - k0 < KPT ? static_cast<uint32_t>(n - k0) : KPT) : 0u;
        uint64_t key[KPT];
        if (have) load_keys<C, KPT>(keys, k0, n, keys_vec, key);
        SetWalk walk(offs, s_items, have ? k0 : base);
        uint32_t f = set_filter(filt, walk.item, n_filters);
        bad |= have && f == n_filters;
        const DevTable t = descs[f < n_filters ? f : 0];
        const uint32_t here = !have ? 0u : walk.end - k0 < have ? static_cast<uint32_t>(walk.end - k0) : have;
        uint32_t live = f < n_filters ? (1u << here) - 1u : 0u;  // keys of the first filter
        uint32_t prim = 0, sec = 0;                              // one bit per key
#pragma unroll
        for (int g = 0; g < KPT; g += B) {
            uint64_t b[B];
            uint32_t fp[B];
            uint64_t c[B][C::nchunks];
#pragma unroll
            for (int j = 0; j < B; ++j) {
                if ((live >> (g + j)) & 1u) {
                    candidates<C>(key[g + j], t.nb_mask, b[j], fp[j]);
                    load_rlx<C::bucket_bytes>(bucket_words<C>(t, b[j]), c[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < B; ++j)
                if (((live >> (g + j)) & 1u) && try_insert<C>(bucket_words<C>(t, b[j]), c[j], fp[j], err)) prim |= 1u << (g + j);
#pragma unroll
            for (int j = 0; j < B; ++j) {
                if (((live & ~prim) >> (g + j)) & 1u) {
                    b[j] = alt_bucket<C>(b[j], fp[j], t.nb_mask);
                    load_rlx<C::bucket_bytes>(bucket_words<C>(t, b[j]), c[j]);
                }
            }
#pragma unroll
            for (int j = 0; j < B; ++j)
                if ((((live & ~prim) >> (g + j)) & 1u) && !err &&
                    try_insert<C>(bucket_words<C>(t, b[j]), c[j], alt_tag<C>(fp[j]), err))
                    sec |= 1u << (g + j);
        }
        auto stored = [](unsigned long long* ctr, uint32_t p, uint32_t q) {
            if (p) atomicAdd(&ctr[CTR_PRIMARY], static_cast<unsigned long long>(p));
            if (q) atomicAdd(&ctr[CTR_SECONDARY], static_cast<unsigned long long>(q));
            if (p + q) atomicAdd(&ctr[CTR_OCCUPIED], static_cast<unsigned long long>(p + q));
        };
        set_add_runs(descs, f, live != 0, __popc(prim), __popc(sec), stored);
        if (here < have) {  // keys past the first filter
            uint32_t p = 0, q = 0;
            DevTable t2{};
            for (uint32_t j = here; j < have; ++j) {
                if (walk.to(offs, n_items, k0 + j)) {
                    stored(t2.ctr, p, q);
                    p = q = 0;
                    f = set_filter(filt, walk.item, n_filters);
                    bad |= f == n_filters;
                    if (f < n_filters) t2 = descs[f];
                }
                if (f == n_filters) continue;
                live |= 1u << j;
                uint64_t b;
                uint32_t fp;
                uint64_t c[C::nchunks];
                candidates<C>(static_cast<uint64_t>(keys[k0 + j]), t2.nb_mask, b, fp);
                load_rlx<C::bucket_bytes>(bucket_words<C>(t2, b), c);
                if (try_insert<C>(bucket_words<C>(t2, b), c, fp, err)) {
                    prim |= 1u << j;
                    ++p;
                } else if (!err) {
                    b = alt_bucket<C>(b, fp, t2.nb_mask);
                    load_rlx<C::bucket_bytes>(bucket_words<C>(t2, b), c);
                    if (try_insert<C>(bucket_words<C>(t2, b), c, alt_tag<C>(fp), err)) {
                        sec |= 1u << j;
                        ++q;
                    }
                }
            }
            stored(t2.ctr, p, q);
        }
        if (have && out) store_results<KPT>(out, k0, n, out_vec, prim | sec);
        // park the keys whose buckets are both full
        const uint32_t hard = live & ~(prim | sec);
        const uint32_t cnt = __popc(hard);
        const uint32_t incl = warp_inclusive_scan(cnt);
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        uint32_t pos = pending + incl - cnt;
#pragma unroll
        for (int j = 0; j < KPT; ++j)
            if ((hard >> j) & 1u) buf[pos++] = k0 + j;
        pending += total;
        __syncwarp();
        while (pending >= 32) {
            pending -= 32;
            const uint64_t idx = buf[pending + lane];
            __syncwarp();
            evict_parked(idx, true);
        }
    }
    evict_parked(lane < pending ? buf[lane] : 0, lane < pending);
    if (__any_sync(0xFFFFFFFFu, err) && lane == 0) atomicOr(err_flag, ERR_CAS_LIMIT);
    if (bad) atomicOr(err_flag, ERR_BAD_FILTER);
}

}  // namespace cfb
