// cf_api.cu -- C ABI of the B200 cuckoo filter (declared in include/cuckoo_b200.h).
//
// Host side of the reference's CuckooFilter<Config> (CuckooFilter.cuh:140-785):
// the filter owns its table and counters; the synchronous calls mirror the
// reference's (launch, cudaStreamSynchronize, read the occupancy counter).  The
// device-side filter descriptor is passed to kernels by value, never as a host
// `this` pointer.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "../../include/cuckoo_b200.h"
#include "cf_registry.cuh"

using namespace cfb;

// Rows of published counters of a filter.  A synchronous random insert or delete
// holds one from before its launch until its stream has been waited for; a call
// that finds none free reads the counters back with a copy instead.
constexpr unsigned int kPubSlots = 64;

struct cf_filter {
    cf_config cfg;
    const OpsTable* ops;
    uint64_t num_buckets;
    uint64_t table_bytes;
    uint8_t* d_table;
    unsigned long long* d_ctr;  // CTR_COUNT device counters
    unsigned long long* h_ctr;  // pinned mirror
    // Counters as the last CTA of a synchronous random insert or delete leaves
    // them: kPubSlots rows of kPublished, the rows' tickets (zero while a row is
    // free) and one bit per free row.
    unsigned long long* h_pub;
    unsigned int* d_ticket;
    std::atomic<uint64_t> pub_free;
    int device;
    int block;
    int max_grid[KID_COUNT_KERNELS];
    int max_grid_aux;
    int sms;
    // segment-staged path
    bool seg_ok;            // the segment-staged path applies: packed (bucket, tag) entries fit in 64 bits
    bool rg_ok;             // the region-staged path applies
    SegGeom geom;
    void* ws;               // workspace (grown on demand, freed with the filter)
    uint64_t ws_bytes;
    uint64_t ws_limit;      // CF_OPT_WORKSPACE_LIMIT (0 = automatic)
    uint64_t seg_min_keys;  // CF_OPT_SEGMENTED_MIN_KEYS (0 = automatic)
    uint64_t round2_min;    // CF_OPT_ROUND2_SEGMENTED_MIN_KEYS (0 = automatic)
    uint32_t round1_cap;    // CF_OPT_ROUND1_CAP (0 = automatic)
    unsigned long long* h_cnt;
    // region-staged path
    RegionGeom rgeom;
    uint64_t rg_min_keys;   // CF_OPT_REGION_MIN_KEYS (0 = automatic)
    uint32_t staging;       // CF_OPT_STAGING (cf_staging)
    uint64_t rg_bytes;      // CF_OPT_REGION_BYTES (0 = kRgRegionBytes)
    uint32_t lookup_kpt;    // CF_OPT_LOOKUP_KPT (0 = default)
    uint32_t probe_width;   // CF_OPT_PROBE_WIDTH (0 or 1 = one lane per key)
    // The table is all zeros (set by cf_create and cf_clear, which synchronize;
    // cleared by every call that may write the table).  Never set again once
    // cf_table has handed out the table's address (table_exposed).
    std::atomic<bool> known_empty;
    bool table_exposed;
    // Staged batches (segment-staged, binned, region-staged) of a filter share its
    // workspace and write whole segments of the table back, so they run one after
    // the other whatever their streams: staged_mu is held while one is enqueued
    // (until it has ended, in a synchronous call), and staged_ev marks the end of the
    // last asynchronous one, on the stream with id staged_stream, while staged_pending.
    std::mutex staged_mu;
    cudaEvent_t staged_ev;
    unsigned long long staged_stream;
    std::atomic<bool> staged_pending;
    uint32_t persistent;    // CF_OPT_PERSISTENT (0 = one tile per CTA, 1 = persistent grid)
    uint32_t chain_hist;    // CF_OPT_CHAIN_HISTOGRAM
};

namespace {

thread_local char g_err[512] = "";

int fail(int status, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return status;
}

int cuda_fail(cudaError_t e, const char* what) {
    return fail(e == cudaErrorMemoryAllocation ? CF_ERR_NO_MEMORY : CF_ERR_CUDA, "%s: %s", what,
                cudaGetErrorString(e));
}

#define CF_CUDA(expr, what)                          \
    do {                                             \
        cudaError_t e_ = (expr);                     \
        if (e_ != cudaSuccess) return cuda_fail(e_, what); \
    } while (0)

const std::vector<OpsTable>& registry() {
    static std::vector<OpsTable> v = [] {
        std::vector<OpsTable> r;
        for (auto* add : {register_bits8, register_bits8_more, register_bits16, register_bits16_more,
                          register_bits16_policy, register_bits32, register_bits32_more})
            add(r);
        return r;
    }();
    return v;
}

const OpsTable* find_ops(const cf_config* c) {
    for (const OpsTable& o : registry())
        if (o.key_bytes == c->key_bytes && o.bits == c->bits_per_tag && o.bucket_size == c->bucket_size &&
            o.word_bytes == c->word_bytes && o.alt_policy == c->alt_policy)
            return &o;
    return nullptr;
}

int validate(const cf_config* c) {
    if (!c) return fail(CF_ERR_INVALID, "config is NULL");
    if (c->key_bytes != 4 && c->key_bytes != 8) return fail(CF_ERR_INVALID, "key_bytes must be 4 or 8");
    if (c->bits_per_tag != 8 && c->bits_per_tag != 16 && c->bits_per_tag != 32)
        return fail(CF_ERR_INVALID, "bits_per_tag must be 8, 16 or 32");
    if (c->bucket_size == 0 || (c->bucket_size & (c->bucket_size - 1)))
        return fail(CF_ERR_INVALID, "bucket_size must be a power of two");
    if (c->word_bytes != 8 && c->word_bytes != 4) return fail(CF_ERR_INVALID, "word_bytes must be 4 or 8");
    if (c->eviction_policy != CF_EVICT_BFS && c->eviction_policy != CF_EVICT_DFS)
        return fail(CF_ERR_INVALID, "eviction_policy must be CF_EVICT_BFS or CF_EVICT_DFS");
    if (c->max_evictions < 1 || c->max_evictions > kMaxEvictionsCap)
        return fail(CF_ERR_INVALID, "max_evictions must be in [1, %u]", kMaxEvictionsCap);
    if (c->block_size != 0 && (c->block_size % 32 != 0 || c->block_size > 512))
        return fail(CF_ERR_INVALID, "block_size must be 0 or a multiple of 32 up to 512");
    if (c->alt_policy != CF_ALT_XOR && c->alt_policy != CF_ALT_ADDSUB && c->alt_policy != CF_ALT_OFFSET)
        return fail(CF_ERR_INVALID, "alt_policy must be CF_ALT_XOR, CF_ALT_ADDSUB or CF_ALT_OFFSET");
    if (!find_ops(c))
        return fail(CF_ERR_UNSUPPORTED,
                    "no kernels for key_bytes=%u bits_per_tag=%u bucket_size=%u word_bytes=%u alt_policy=%u",
                    c->key_bytes, c->bits_per_tag, c->bucket_size, c->word_bytes, c->alt_policy);
    return CF_OK;
}

uint64_t num_buckets_for(uint64_t capacity, uint32_t bucket_size) {
    // std::ceil((double)capacity / bucketSize), then nextPowerOfTwo (helpers.cuh:31-45).
    const double req = std::ceil(static_cast<double>(capacity) / static_cast<double>(bucket_size));
    uint64_t r = static_cast<uint64_t>(req);
    if (r != 0 && (r & (r - 1)) == 0) return r;
    uint64_t n = r - 1;
    n |= n >> 1;
    n |= n >> 2;
    n |= n >> 4;
    n |= n >> 8;
    n |= n >> 16;
    n |= n >> 32;
    return n + 1;
}

// calculateNumBuckets of each policy (bucket_policies.cuh:80-83, :166-176, :346-349).
uint64_t num_buckets_policy(uint64_t capacity, uint32_t bucket_size, uint32_t alt_policy) {
    if (alt_policy == CF_ALT_XOR) return num_buckets_for(capacity, bucket_size);
    uint64_t r = static_cast<uint64_t>(std::ceil(static_cast<double>(capacity) / static_cast<double>(bucket_size)));
    if (alt_policy == CF_ALT_ADDSUB && (r % 2) != 0) r += 1;
    return r;
}

DevTable dev(const cf_filter* f) {
    return DevTable{f->d_table, f->num_buckets - 1, f->d_ctr, f->chain_hist ? f->d_ctr + CTR_HIST0 : nullptr};
}

LaunchCfg launch(const cf_filter* f, int kid, void* stream) {
    LaunchCfg L{static_cast<cudaStream_t>(stream), f->block, f->max_grid[kid]};
    L.full_grid = f->persistent == 0;
    return L;
}

LaunchCfg launch_aux(const cf_filter* f, void* stream) {
    return LaunchCfg{static_cast<cudaStream_t>(stream), 256, f->max_grid_aux};
}

struct DeviceGuard {
    int prev = -1;
    bool ok = true;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) ok = cudaSetDevice(dev) == cudaSuccess;
    }
    ~DeviceGuard() {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
    }
};

int check_filter(const cf_filter* f) {
    if (!f) return fail(CF_ERR_INVALID, "filter is NULL");
    return CF_OK;
}

int check_batch(const cf_filter* f, const void* keys, uint64_t n) {
    if (int s = check_filter(f)) return s;
    if (n && !keys) return fail(CF_ERR_INVALID, "keys is NULL with n > 0");
    return CF_OK;
}

int check_counters(const unsigned long long* c, uint64_t* occupied_out) {
    if (c[CTR_ERROR] & ERR_CAS_LIMIT)
        return fail(CF_ERR_DEVICE, "a compare-and-swap retry bound was hit on the device");
    if (c[CTR_ERROR] & ERR_WAIT_LIMIT)
        return fail(CF_ERR_DEVICE, "a bulk copy did not complete within its poll bound on the device");
    if (occupied_out) *occupied_out = c[CTR_OCCUPIED];
    return CF_OK;
}

// Synchronize, read the counters, surface device-side errors.
int finish(cf_filter* f, void* stream, uint64_t* occupied_out) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    CF_CUDA(cudaMemcpyAsync(f->h_ctr, f->d_ctr, CTR_COUNT * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s),
            "counter read-back");
    CF_CUDA(cudaStreamSynchronize(s), "stream synchronize");
    return check_counters(f->h_ctr, occupied_out);
}

// A row of published counters held by one synchronous call, or none when all are
// in use.  It goes back only once the kernel that uses it has ended (which leaves
// the ticket at zero): a call whose launch or wait failed keeps it from reuse.
struct PubRow {
    cf_filter* f;
    int row = -1;
    explicit PubRow(cf_filter* filter) : f(filter) {
        uint64_t free = f->pub_free.load(std::memory_order_relaxed);
        while (free) {
            const int r = __builtin_ctzll(free);
            if (f->pub_free.compare_exchange_weak(free, free & ~(1ull << r), std::memory_order_acquire)) {
                row = r;
                return;
            }
        }
    }
    DevTable table() const {
        DevTable t = dev(f);
        if (row >= 0) {
            t.pub = f->h_pub + row * kPublished;
            t.ticket = f->d_ticket + row;
        }
        return t;
    }
    // Waits for the random insert or delete launched with table(), whose last CTA
    // has written the row.
    int finish(void* stream, uint64_t* occupied_out) const {
        if (row < 0) return ::finish(f, stream, occupied_out);
        CF_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)), "stream synchronize");
        unsigned long long c[kPublished];
        const volatile unsigned long long* pub = f->h_pub + row * kPublished;
        for (int i = 0; i < kPublished; ++i) c[i] = pub[i];
        f->pub_free.fetch_or(1ull << row, std::memory_order_release);
        return check_counters(c, occupied_out);
    }
};

// A capturing stream, or one that cannot be asked (another stream's capture forbids it).
bool is_capturing(cudaStream_t s) {
    cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &c) == cudaSuccess) return c != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return true;
}

// Work enqueued on `stream` from here on follows the last asynchronous staged
// batch.  Not under capture: an event from outside cannot be waited for there, and
// the graph's launches are ordered by whoever launches it.  Holds staged_mu.
int follow_staged_locked(cf_filter* f, void* stream) {
    if (!f->staged_pending) return CF_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (is_capturing(s)) return CF_OK;
    unsigned long long id = 0;  // of the stream itself: a handle can be used again for another
    if (cudaStreamGetId(s, &id) == cudaSuccess) {
        if (id == f->staged_stream) return CF_OK;
    } else {
        cudaGetLastError();
    }
    CF_CUDA(cudaStreamWaitEvent(s, f->staged_ev, 0), "wait for the batch before");
    return CF_OK;
}

// The same for a call that is not a staged batch itself.
int follow_staged(cf_filter* f, void* stream) {
    if (!f->staged_pending.load(std::memory_order_acquire)) return CF_OK;
    std::lock_guard<std::mutex> lock(f->staged_mu);
    return follow_staged_locked(f, stream);
}

// The same for the blocking reads and writes of the counters, which go to the
// legacy default stream (non-blocking streams do not order themselves with it).
int follow_staged(cf_filter* f) { return follow_staged(f, nullptr); }

// Marks the end of an asynchronous staged batch.
int note_staged_locked(cf_filter* f, void* stream) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (is_capturing(s)) return CF_OK;
    CF_CUDA(cudaStreamGetId(s, &f->staged_stream), "stream id");
    CF_CUDA(cudaEventRecord(f->staged_ev, s), "mark the end of the batch");
    f->staged_pending.store(true, std::memory_order_release);
    return CF_OK;
}

// A staged batch: run() enqueues it; with `wait` the call returns when it has
// ended, with the occupied count.
template <class Run>
int staged_batch(cf_filter* f, void* stream, bool wait, uint64_t* occupied_out, Run run) {
    std::lock_guard<std::mutex> lock(f->staged_mu);
    if (int st = follow_staged_locked(f, stream)) return st;
    int st = run();
    if (wait && st == CF_OK) {
        st = finish(f, stream, occupied_out);
        if (st == CF_OK) {
            f->staged_pending.store(false, std::memory_order_release);
            return CF_OK;
        }
    }
    // (an error may have left part of the batch in flight)
    const int noted = note_staged_locked(f, stream);
    return st ? st : noted;
}

void init_geometry(cf_filter* f) {
    const uint64_t bb = f->ops->bucket_bytes;
    uint64_t sb = kSegBytes / bb;
    if (sb > f->num_buckets) sb = f->num_buckets;
    f->geom.sb_log2 = ilog2(sb);  // a power of two at most the bucket count
    sb = 1ull << f->geom.sb_log2;
    // the last segment is partial when the bucket count (AddSub and Offset
    // policies) is not a multiple of the segment
    f->geom.nseg = (f->num_buckets + sb - 1) / sb;
    f->geom.seg_shift = static_cast<int>(f->cfg.bits_per_tag) + f->geom.sb_log2;
    const int seg_bits = clog2(f->geom.nseg);
    f->geom.passes = seg_bits == 0 ? 1 : (seg_bits + kRadixBits - 1) / kRadixBits;
    // (bucket << bits) | tag must fit in 64 bits for every bucket index
    f->seg_ok = clog2(f->num_buckets) + static_cast<int>(f->cfg.bits_per_tag) <= 64 && f->ops->seg_chunk;
    f->rg_ok = f->seg_ok && f->ops->rg_chunk;
    // regions of ~kRgRegionBytes (or CF_OPT_REGION_BYTES), at most kRgMaxRegions
    // of them; the last region is partial when the bucket count is not a power
    // of two (AddSub and Offset policies)
    const int nb_log2 = clog2(f->num_buckets);
    const uint64_t rbytes = f->rg_bytes ? f->rg_bytes : kRgRegionBytes;
    int rl = rbytes > bb ? ilog2(rbytes / bb) : 0;
    if (rl < nb_log2 - 8) rl = nb_log2 - 8;
    if (rl > nb_log2) rl = nb_log2;
    f->rgeom.rl = rl;
    f->rgeom.nreg = static_cast<uint32_t>(((f->num_buckets - 1) >> rl) + 1);
}

// Words of the known-full bucket bitmap (one bit per bucket of the segment
// geometry), kept when the segment insert runs k_seg_insert (at most 64
// slots per bucket) on segments of at least 32 buckets; else 0.
uint64_t full_words(const cf_filter* f) {
    if (f->cfg.bucket_size > 64 || f->geom.sb_log2 < 5) return 0;
    return (f->geom.nseg << f->geom.sb_log2) >> 5;
}

// Bytes of workspace for a chunk of `cap` keys: two entry buffers (8 B per
// key), and with per-key results two payload buffers (4 B) and a result bitmap;
// besides, per table, the radix histogram, the segment starts, the list
// counters and the known-full bucket bitmap.
uint64_t ws_need(const cf_filter* f, uint64_t cap, int grid, bool payload) {
    const uint64_t hist = static_cast<uint64_t>(kRadix) * grid * 4;
    const uint64_t start = (f->geom.nseg + 1) * 4;
    auto al = [](uint64_t x) { return (x + 255) & ~255ull; };
    // result bitmap: two bits per key (a region-staged lookup keeps one hit bit per staged entry)
    const uint64_t per_key = payload ? al(cap * 4) * 2 + al((2 * cap + 31) / 32 * 4) : 0;
    return al(cap * 8) * 2 + per_key + al(hist) + al(start) + al(64) + al(full_words(f) * 4);
}

// Automatic workspace limit (CF_OPT_WORKSPACE_LIMIT = 0, the default): the
// device memory free now plus the workspace already held (it is freed before a
// larger one is allocated), less a reserve of 1/16 of the device (at least
// 1 GiB) left to the caller.  The reference allocates what each sorted insert
// needs (CuckooFilter.cuh:475-508); this keeps the whole batch in one chunk
// whenever that fits, and keeps the workspace for the next call.
constexpr uint64_t kMinAutoWorkspace = 256ull << 20;

uint64_t auto_workspace_limit(const cf_filter* f) {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
        cudaGetLastError();
        return 4ull << 30;
    }
    const uint64_t reserve = std::max<uint64_t>(1ull << 30, total_b / 16);
    const uint64_t avail = f->ws_bytes + free_b;
    return avail > reserve + kMinAutoWorkspace ? avail - reserve : kMinAutoWorkspace;
}

int ensure_workspace(cf_filter* f, uint64_t n, bool payload, SegWork* w) {
    // radix passes: one wave of each payload mode's scatter kernel, fixed per-CTA chunks
    int rs_grid[3];
    CF_CUDA(rs_scatter_grid<0>(f->sms, &rs_grid[0]), "radix launch setup");
    CF_CUDA(rs_scatter_grid<1>(f->sms, &rs_grid[1]), "radix launch setup");
    CF_CUDA(rs_scatter_grid<2>(f->sms, &rs_grid[2]), "radix launch setup");
    const int rg_grid = f->sms * 4;
    const int grid = std::max(std::max(rs_grid[0], std::max(rs_grid[1], rs_grid[2])) * kRsHistSub,
                              (rg_grid * static_cast<int>(kRgMaxRegions) + kRadix - 1) / kRadix);
    const uint64_t fixed = ws_need(f, 0, grid, payload) + 4096;
    const uint64_t kMaxChunk = 1ull << 31;  // 32-bit positions and payloads
    uint64_t limit = f->ws_limit;
    bool fits_held = false;  // automatic limit, and the whole batch fits the workspace already held
    if (limit == 0) {  // automatic: the whole batch when device memory allows
        const uint64_t whole = ws_need(f, std::min(n, kMaxChunk), grid, payload);
        fits_held = whole <= f->ws_bytes;
        limit = fits_held ? f->ws_bytes : auto_workspace_limit(f);
    }
    uint64_t cap = 0, need = 0;
    for (;;) {
        cap = n;
        if (fits_held) {
            // one chunk (the fit below is conservative and would split off a
            // sliver of the batch)
        } else if (limit > fixed) {
            const uint64_t fit = (limit - fixed) / (payload ? 25 : 16);
            if (cap > fit) cap = fit;
        } else {
            cap = 0;
        }
        if (cap > kMaxChunk) cap = kMaxChunk;
        if (cap < n) cap = cap / 32 * 32;
        if (cap < 1024 && n > cap) cap = 1024;
        need = ws_need(f, cap, grid, payload);
        if (f->ws_bytes >= need) break;
        if (f->ws) cudaFree(f->ws);
        f->ws = nullptr;
        f->ws_bytes = 0;
        const cudaError_t e = cudaMalloc(&f->ws, need);
        if (e == cudaSuccess) {
            f->ws_bytes = need;
            break;
        }
        // automatic limit: another allocation may have taken the memory since
        // it was measured; retry with half the chunk
        if (e != cudaErrorMemoryAllocation || f->ws_limit != 0 || need <= kMinAutoWorkspace)
            return cuda_fail(e, "workspace allocation");
        cudaGetLastError();
        f->ws = nullptr;
        limit = std::max(kMinAutoWorkspace, need / 2);
    }
    auto al = [](uint64_t x) { return (x + 255) & ~255ull; };
    uint8_t* p = static_cast<uint8_t*>(f->ws);
    w->ent[0] = reinterpret_cast<uint64_t*>(p);
    p += al(cap * 8);
    w->ent[1] = reinterpret_cast<uint64_t*>(p);
    p += al(cap * 8);
    w->hist = reinterpret_cast<uint32_t*>(p);
    p += al(static_cast<uint64_t>(kRadix) * grid * 4);
    w->start = reinterpret_cast<uint32_t*>(p);
    p += al((f->geom.nseg + 1) * 4);
    w->cnt = reinterpret_cast<unsigned long long*>(p);
    p += al(64);
    w->full_words = full_words(f);
    w->full = w->full_words ? reinterpret_cast<uint32_t*>(p) : nullptr;
    p += al(w->full_words * 4);
    w->pay[0] = w->pay[1] = nullptr;
    w->bitmap = nullptr;
    if (payload) {
        w->pay[0] = reinterpret_cast<uint32_t*>(p);
        p += al(cap * 4);
        w->pay[1] = reinterpret_cast<uint32_t*>(p);
        p += al(cap * 4);
        w->bitmap = reinterpret_cast<uint32_t*>(p);
    }
    w->h_cnt = f->h_cnt;
    w->cap = cap;
    for (int i = 0; i < 3; ++i) w->rs_grid[i] = rs_grid[i];
    w->rg_grid = rg_grid;
    w->sms = f->sms;
    return CF_OK;
}

// Keys from which the alternate-bucket round of a segment-staged batch is staged too
// rather than probed at random: a random probe costs one DRAM transaction (about
// 50 G/s for reads of a table past L2, 23 for read-modify-writes), staging the segments'
// bytes, read and for inserts written back.  For inserts that pays off from about
// one key per 64 table bytes, for lookups and deletes from several keys per bucket.
uint64_t auto_threshold(const cf_filter* f, int op) {
    if (op == SEG_INSERT) return f->table_bytes / 64;
    return f->num_buckets * 8;
}

// Batch size from which a batch is staged.  Inserts: one key per bucket, and
// enough keys to pay for a dozen launches: 2^17, or 2^20 for batches that cannot
// fill an empty table beyond three quarters (fewer evictions, which random inserts
// pay most for; the load before the batch is not known on the host, and tops-up
// from 0.6 and 0.8 to 0.9 were faster at random than segment-staged too).  Binned against random, us, 16-bit tags, filling an empty table:
// 2^14 slots to 0.95 80 and 58, to 0.6 52 and 25; 2^17 to 0.6 60 and 28; 2^20 to 0.6
// 66 and 40, to 0.95 107 and 110; 2^22 to 0.6 80 and 92, to 0.95 156 and 236.
// (Batches full of repeats are the exception: keys that must fail walk to the end
// beside the others.  2^18 slots to 0.6, half the batch repeats of 100 keys, DFS: 4.3 ms
// at random, 3.0 segment-staged.)
// Below one key per bucket random inserts win at every size (2^26 8-bit slots,
// 0.76 keys per bucket: 105 us a batch in the first half of the fill, 170 in the
// second, against 309 and 382 segment-staged).
// Deletes: eight keys per bucket.  Lookups: never.
// Random lookups were faster for every table and batch measured (256 KiB to
// 2 GiB, 2 to 64 keys per bucket, random against segment-staged G/s: 97 and 21
// in 8 MiB, 65 and 25 in 128 MiB, 36 and 24 in 512 MiB, 31.4 and 21.7 in 2 GiB).
uint64_t segmented_threshold(const cf_filter* f, int op, uint64_t n) {
    if (f->seg_min_keys) return f->seg_min_keys;
    if (op == SEG_DELETE) return f->num_buckets * 8;
    if (op != SEG_INSERT) return UINT64_MAX;
    const bool to_high_load = n >= f->num_buckets * f->cfg.bucket_size / 4 * 3;
    return std::max<uint64_t>(f->num_buckets, to_high_load ? 1ull << 17 : 1ull << 20);
}

int run_segmented(cf_filter* f, int op, const void* keys, uint64_t n, uint8_t* out, void* stream) {
    if (n == 0) return CF_OK;
    SegWork w{};
    if (int st = ensure_workspace(f, n, out != nullptr, &w)) return st;
    w.round2_segmented_min = f->round2_min ? f->round2_min : auto_threshold(f, op);
    w.round1_cap = f->round1_cap;
    // an insert into a table known to be empty: its first chunk's first
    // round stages zeroed segments instead of loading them
    bool fresh = op == SEG_INSERT && f->known_empty;
    f->known_empty = false;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const uint64_t kb = f->cfg.key_bytes;
    for (uint64_t c0 = 0; c0 < n; c0 += w.cap) {
        const uint64_t m = n - c0 < w.cap ? n - c0 : w.cap;
        w.fresh = fresh;
        fresh = false;
        CF_CUDA(f->ops->seg_chunk(dev(f), f->geom, w, op, static_cast<const uint8_t*>(keys) + c0 * kb, m,
                                  out ? out + c0 : nullptr, s, f->cfg.eviction_policy == CF_EVICT_BFS ? 1u : 0u,
                                  f->cfg.max_evictions),
                "segment-staged batch");
    }
    return CF_OK;
}

// The whole batch through the binned path; *taken is false (and nothing has
// been stored) when its workspace does not fit the limit or the batch is skewed.
int run_binned(cf_filter* f, const void* keys, uint64_t n, uint8_t* out, void* stream, bool* taken) {
    *taken = false;
    // A captured insert would replay what holds only now (an empty table, this
    // workspace), so a capturing stream is left to the segment-staged path, whose
    // host waits end the capture with an error.
    BinGeom g{};
    if (is_capturing(static_cast<cudaStream_t>(stream)) || !f->ops->bin_insert || !f->seg_ok ||
        !bin_geometry(f->num_buckets, f->ops->bucket_bytes, f->cfg.bits_per_tag, f->cfg.alt_policy, n, &g))
        return CF_OK;
    auto al = [](uint64_t x) { return (x + 255) & ~255ull; };
    const uint64_t words = f->cfg.bucket_size <= 64 && g.sbl >= 5 ? (static_cast<uint64_t>(g.nseg) << g.sbl) >> 5 : 0;
    // a buffer holds first-pass bins in one round and segments' bins in another
    const uint64_t eb1 = g.l2 ? g.entry_bytes1 : g.entry_bytes2, eb2 = g.entry_bytes2;
    const uint64_t b0 = std::max(g.ent[0] * eb1, g.l2 ? 0 : g.ent[1] * eb2), b1 = g.ent[1] * eb2;
    const uint64_t cursors = 3ull * ((g.l2 ? g.d1 : 0u) + g.nseg) * 4 * kCursorStride;
    // The list of entries without room holds the whole batch, or half of it (two
    // passes only) where the memory counts (8 GB at 2^30 keys) and the waits that
    // go with it do not, or where only that fits the limit.  What the first round leaves
    // goes to random inserts if a short list might not hold it (AddSub fill of 10^9 slots:
    // 79 ms for 38), so the list has its full length, if it can, where that may be: in a
    // table that is not empty, and where the primary buckets hold less than five
    // eighths of the batch (the AddSub policy's are half of the table).
    // list, ent[0] and ent[1] side by side hold two lists of n entries in the end.
    uint64_t room = 0, ents = 0, pays = 0, need = 0;
    auto size = [&](uint64_t list_room) {
        room = list_room;
        ents = std::max(al(room * 8) + al(b0) + al(b1), al(2 * n * 8));
        pays = out ? std::max(al(room * 4) + al(g.ent[0] * 4) + al(g.ent[1] * 4), al(2 * n * 4)) : 0;
        need = ents + pays + al(cursors) + al(g.nseg * 4ull) + al(64) + al(words * 4);
    };
    const bool can_halve = g.l2 && b0 >= n * 8 && (!out || g.ent[0] >= n);
    const uint64_t bs = f->cfg.bucket_size, cap1 = f->round1_cap ? f->round1_cap : bs - bs * kRound1SlackSixteenths / 16;
    const uint64_t primary = f->cfg.alt_policy == CF_ALT_ADDSUB ? f->num_buckets / 2 : f->num_buckets;
    const bool leaves_few = f->known_empty && cap1 * primary >= n / 8 * 5;
    size(can_halve && n >= (1ull << 27) && leaves_few ? n / 2 : n);
    if (need > f->ws_bytes) {
        const uint64_t limit = f->ws_limit ? f->ws_limit : auto_workspace_limit(f);
        if (need > limit && can_halve) size(n / 2);
        if (need > limit) return CF_OK;
        if (need > f->ws_bytes) {
            if (f->ws) cudaFree(f->ws);
            f->ws = nullptr;
            f->ws_bytes = 0;
            if (cudaMalloc(&f->ws, need) != cudaSuccess) {
                cudaGetLastError();
                f->ws = nullptr;
                return CF_OK;  // the segment-staged path sizes its chunks to what there is
            }
            f->ws_bytes = need;
        }
    }
    BinWork w{};
    uint8_t* p = static_cast<uint8_t*>(f->ws);
    w.list = reinterpret_cast<uint64_t*>(p);
    w.ent[0] = p + al(room * 8);
    w.ent[1] = p + al(room * 8) + al(b0);
    p += ents;
    if (out) {
        w.list_pay = reinterpret_cast<uint32_t*>(p);
        w.pay[0] = reinterpret_cast<uint32_t*>(p + al(room * 4));
        w.pay[1] = reinterpret_cast<uint32_t*>(p + al(room * 4) + al(g.ent[0] * 4));
        p += pays;
    }
    w.left = reinterpret_cast<uint32_t*>(p);
    p += al(g.nseg * 4ull);
    w.cursor = reinterpret_cast<uint32_t*>(p);
    p += al(cursors);
    w.cnt = reinterpret_cast<unsigned long long*>(p);
    p += al(64);
    w.full = words ? reinterpret_cast<uint32_t*>(p) : nullptr;
    w.zero_bytes = al(cursors) + al(64) + words * 4;
    w.list_room = room;
    w.h_cnt = f->h_cnt;
    w.sms = f->sms;
    w.round1_cap = f->round1_cap;
    w.fresh = f->known_empty;
    f->known_empty = false;
    bool skewed = false;
    CF_CUDA(f->ops->bin_insert(dev(f), g, w, keys, n, out, static_cast<cudaStream_t>(stream),
                               f->cfg.eviction_policy == CF_EVICT_BFS ? 1u : 0u, f->cfg.max_evictions, &skewed),
            "binned insert");
    if (skewed) f->known_empty = w.fresh;  // nothing has been stored
    *taken = !skewed;
    return CF_OK;
}

// Region-staged path (cf_region.cuh): keys from which it beats random probes.
// A random probe costs one DRAM transaction (~50 G/s on B200); the region path
// streams ~30 bytes per key plus the table once (lookups) or about twice
// (inserts and deletes), at close to HBM bandwidth.
uint64_t region_threshold(const cf_filter* f, int op) {
    if (f->rg_min_keys) return f->rg_min_keys;
    (void)op;
    return UINT64_MAX;  // automatic choice: not yet (measured slower than the other paths)
}

int run_region(cf_filter* f, int op, const void* keys, uint64_t n, uint8_t* out, void* stream) {
    if (n == 0) return CF_OK;
    if (op != SEG_CONTAINS) f->known_empty = false;
    SegWork w{};
    if (int st = ensure_workspace(f, n, op == SEG_CONTAINS || out != nullptr, &w)) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const uint64_t kb = f->cfg.key_bytes;
    // lookups stage two entries per key (32-bit entry offsets) and gather each
    // partition chunk's results in shared memory: at most 2^29 keys per chunk
    uint64_t cap = w.cap;
    if (op == SEG_CONTAINS) {
        const uint64_t lim = std::min<uint64_t>(1ull << 29, static_cast<uint64_t>(w.rg_grid) * 1000000ull);
        if (cap > lim) cap = lim;
    }
    for (uint64_t c0 = 0; c0 < n; c0 += cap) {
        const uint64_t m = n - c0 < cap ? n - c0 : cap;
        CF_CUDA(f->ops->rg_chunk(dev(f), f->rgeom, w, op, static_cast<const uint8_t*>(keys) + c0 * kb, m,
                                 out ? out + c0 : nullptr, s, f->cfg.eviction_policy == CF_EVICT_BFS ? 1u : 0u,
                                 f->cfg.max_evictions),
                "region-staged batch");
    }
    return CF_OK;
}

// Execution path of a batch: random probes, segment-staged or region-staged.
enum Path { PATH_RANDOM, PATH_SEGMENT, PATH_REGION };

Path choose_path(const cf_filter* f, int op, uint64_t n, bool sorted_insert) {
    if (!f->seg_ok) return PATH_RANDOM;
    switch (f->staging) {
        case CF_STAGING_RANDOM: return sorted_insert ? PATH_SEGMENT : PATH_RANDOM;
        case CF_STAGING_SEGMENT: return PATH_SEGMENT;
        case CF_STAGING_REGION: return f->rg_ok ? PATH_REGION : PATH_SEGMENT;
        default: break;
    }
    if (f->rg_ok && n >= region_threshold(f, op)) return PATH_REGION;
    if (sorted_insert) return PATH_SEGMENT;
    if (n >= segmented_threshold(f, op, n)) return PATH_SEGMENT;
    return PATH_RANDOM;
}

int do_insert(cf_filter* f, const DevTable& t, const void* keys, uint64_t n, uint8_t* out, void* stream) {
    f->known_empty = false;
    CF_CUDA(f->ops->insert(t, keys, n, out, launch(f, KID_INSERT, stream),
                           f->cfg.eviction_policy == CF_EVICT_BFS ? 1u : 0u, f->cfg.max_evictions),
            "insert launch");
    return CF_OK;
}

template <class C>
void host_candidates_t(uint64_t mask, const void* keys, uint64_t n, uint64_t* i1, uint64_t* i2, uint32_t* fp) {
    const auto* k = static_cast<const typename C::Key*>(keys);
    for (uint64_t i = 0; i < n; ++i) {
        uint64_t b;
        uint32_t f;
        candidates<C>(static_cast<uint64_t>(k[i]), mask, b, f);
        if (i1) i1[i] = b;
        if (i2) i2[i] = alt_bucket<C>(b, f, mask);
        if (fp) fp[i] = f;
    }
}

// Bucket size does not enter the hashing; 16 slots stands in for any.
template <int POL>
void host_candidates_p(uint32_t kb, uint32_t bits, uint64_t nbm, const void* keys, uint64_t n, uint64_t* i1,
                       uint64_t* i2, uint32_t* fp) {
    if (kb == 8) {
        if (bits == 8) host_candidates_t<Cfg<8, 8, 16, 8, POL>>(nbm, keys, n, i1, i2, fp);
        else if (bits == 16) host_candidates_t<Cfg<8, 16, 16, 8, POL>>(nbm, keys, n, i1, i2, fp);
        else host_candidates_t<Cfg<8, 32, 8, 8, POL>>(nbm, keys, n, i1, i2, fp);
    } else {
        if (bits == 8) host_candidates_t<Cfg<4, 8, 16, 8, POL>>(nbm, keys, n, i1, i2, fp);
        else if (bits == 16) host_candidates_t<Cfg<4, 16, 16, 8, POL>>(nbm, keys, n, i1, i2, fp);
        else host_candidates_t<Cfg<4, 32, 8, 8, POL>>(nbm, keys, n, i1, i2, fp);
    }
}

void host_candidates(uint32_t pol, uint32_t kb, uint32_t bits, uint64_t nbm, const void* keys, uint64_t n,
                     uint64_t* i1, uint64_t* i2, uint32_t* fp) {
    if (pol == CF_ALT_ADDSUB) host_candidates_p<ALT_ADDSUB>(kb, bits, nbm, keys, n, i1, i2, fp);
    else if (pol == CF_ALT_OFFSET) host_candidates_p<ALT_OFFSET>(kb, bits, nbm, keys, n, i1, i2, fp);
    else host_candidates_p<ALT_XOR>(kb, bits, nbm, keys, n, i1, i2, fp);
}

}  // namespace

namespace cfb {
// Error reporting for the other translation units of the C ABI (filter sets).
int api_fail(int status, const char* msg) { return fail(status, "%s", msg); }
int api_cuda_fail(cudaError_t e, const char* what) { return cuda_fail(e, what); }
int api_validate(const cf_config* cfg) { return validate(cfg); }
uint64_t api_num_buckets(uint64_t capacity, uint32_t bucket_size, uint32_t alt_policy) {
    return num_buckets_policy(capacity, bucket_size, alt_policy);
}
}  // namespace cfb

extern "C" {

int cf_abi_version(void) { return CF_ABI_VERSION; }

uint64_t cf_launch_count(void) { return launch_counter().load(std::memory_order_relaxed); }

const char* cf_last_error(void) { return g_err; }

const char* cf_status_string(int status) {
    switch (status) {
        case CF_OK: return "CF_OK";
        case CF_ERR_INVALID: return "CF_ERR_INVALID";
        case CF_ERR_UNSUPPORTED: return "CF_ERR_UNSUPPORTED";
        case CF_ERR_CUDA: return "CF_ERR_CUDA";
        case CF_ERR_NO_MEMORY: return "CF_ERR_NO_MEMORY";
        case CF_ERR_DEVICE: return "CF_ERR_DEVICE";
        case CF_ERR_NOT_LOADED: return "CF_ERR_NOT_LOADED";
        default: return "CF_ERR_UNKNOWN";
    }
}

int cf_config_supported(const cf_config* cfg) { return cfg && find_ops(cfg) != nullptr; }

uint64_t cf_num_buckets_for(uint64_t capacity, uint32_t bucket_size) {
    if (bucket_size == 0) return 0;
    return num_buckets_for(capacity, bucket_size);
}

uint64_t cf_num_buckets_for_policy(uint64_t capacity, uint32_t bucket_size, uint32_t alt_policy) {
    if (bucket_size == 0 || alt_policy > CF_ALT_OFFSET) return 0;
    return num_buckets_policy(capacity, bucket_size, alt_policy);
}

int cf_create(const cf_config* cfg, uint64_t capacity, cf_filter** out) {
    if (!out) return fail(CF_ERR_INVALID, "out is NULL");
    *out = nullptr;
    if (int s = validate(cfg)) return s;
    if (capacity == 0) return fail(CF_ERR_INVALID, "capacity must be > 0");
    int device = 0;
    {
        cudaError_t e = cudaGetDevice(&device);
        if (e != cudaSuccess) return fail(CF_ERR_NOT_LOADED, "no CUDA device: %s", cudaGetErrorString(e));
    }
    cf_filter* f = new cf_filter{};
    f->cfg = *cfg;
    f->ops = find_ops(cfg);
    f->device = device;
    f->num_buckets = num_buckets_policy(capacity, cfg->bucket_size, cfg->alt_policy);
    f->table_bytes = f->num_buckets * f->ops->bucket_bytes;
    f->block = cfg->block_size ? static_cast<int>(cfg->block_size) : 256;
    int sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    for (int k = 0; e == cudaSuccess && k < KID_COUNT_KERNELS; ++k) {
        int bps = 0;
        e = f->ops->occupancy(k, f->block, &bps);
        f->max_grid[k] = sms * (bps > 0 ? bps : 1);
    }
    f->max_grid_aux = sms * 8;
    f->sms = sms;
    init_geometry(f);
    f->ws_limit = 0;  // automatic
    if (e == cudaSuccess) e = cudaHostAlloc(&f->h_cnt, 4 * sizeof(unsigned long long), cudaHostAllocDefault);
    if (e == cudaSuccess) e = cudaMalloc(&f->d_table, f->table_bytes);
    constexpr size_t kCtrBytes = CTR_COUNT * sizeof(unsigned long long) + kPubSlots * sizeof(unsigned int);
    if (e == cudaSuccess) e = cudaMalloc(&f->d_ctr, kCtrBytes);
    if (e == cudaSuccess) f->d_ticket = reinterpret_cast<unsigned int*>(f->d_ctr + CTR_COUNT);
    if (e == cudaSuccess)
        e = cudaHostAlloc(&f->h_ctr, (CTR_COUNT + kPubSlots * kPublished) * sizeof(unsigned long long), cudaHostAllocDefault);
    if (e == cudaSuccess) f->h_pub = f->h_ctr + CTR_COUNT;
    static_assert(kPubSlots == 64, "one bit of pub_free per row");
    f->pub_free = ~0ull;
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&f->staged_ev, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaMemset(f->d_table, 0, f->table_bytes);
    if (e == cudaSuccess) e = cudaMemset(f->d_ctr, 0, kCtrBytes);
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        int s = cuda_fail(e, "filter allocation");
        cf_destroy(f);
        return s;
    }
    f->known_empty = true;
    *out = f;
    return CF_OK;
}

int cf_destroy(cf_filter* f) {
    if (!f) return CF_OK;
    DeviceGuard g(f->device);
    if (f->d_table) cudaFree(f->d_table);
    if (f->d_ctr) cudaFree(f->d_ctr);
    if (f->h_ctr) cudaFreeHost(f->h_ctr);
    if (f->h_cnt) cudaFreeHost(f->h_cnt);
    if (f->ws) cudaFree(f->ws);
    if (f->staged_ev) cudaEventDestroy(f->staged_ev);
    delete f;
    return CF_OK;
}

int cf_get_info(const cf_filter* f, cf_info* out) {
    if (int s = check_filter(f)) return s;
    if (!out) return fail(CF_ERR_INVALID, "out is NULL");
    out->num_buckets = f->num_buckets;
    out->capacity = f->num_buckets * f->cfg.bucket_size;
    out->size_in_bytes = f->table_bytes;
    out->bucket_bytes = f->ops->bucket_bytes;
    out->device = f->device;
    return CF_OK;
}

// Enqueues an insert; with `wait` it returns when the insert has ended, with the occupied count.
int insert_any(cf_filter* f, const void* keys, uint64_t n, uint8_t* out, void* stream, bool sorted, bool wait,
               uint64_t* occupied_out) {
    switch (choose_path(f, SEG_INSERT, n, sorted)) {
        case PATH_REGION:
            return staged_batch(f, stream, wait, occupied_out,
                                [&] { return run_region(f, SEG_INSERT, keys, n, out, stream); });
        case PATH_SEGMENT:
            return staged_batch(f, stream, wait, occupied_out, [&]() -> int {
                // At least one key per bucket: slot order within a bucket is
                // unspecified, and the batch is binned (fills to 0.95, segment-staged
                // against binned: 2^20 slots 420 -> 198 us, 2^28 6.58 -> 4.75 ms with a
                // sample looked up, 2^31 45.8 -> 36.5 ms).  Buckets of more than 16
                // slots, batches that do not fit the workspace limit in one piece and
                // skewed ones with a short list stay segment-staged, and so do those
                // of a caller who asks for that path or sets an option of it.
                bool taken = false;
                if (n >= f->num_buckets && f->staging != CF_STAGING_SEGMENT && !f->round2_min)
                    if (int st = run_binned(f, keys, n, out, stream, &taken)) return st;
                return taken ? CF_OK : run_segmented(f, SEG_INSERT, keys, n, out, stream);
            });
        default: break;
    }
    if (int s = follow_staged(f, stream)) return s;
    if (!wait) return do_insert(f, dev(f), keys, n, out, stream);
    if (!n) return finish(f, stream, occupied_out);
    const PubRow row(f);
    if (int s = do_insert(f, row.table(), keys, n, out, stream)) return s;
    return row.finish(stream, occupied_out);
}

int cf_insert_async(cf_filter* f, const void* d_keys, uint64_t n, uint8_t* d_out, void* stream) {
    if (int s = check_batch(f, d_keys, n)) return s;
    DeviceGuard g(f->device);
    return insert_any(f, d_keys, n, d_out, stream, false, false, nullptr);
}

int cf_insert(cf_filter* f, const void* d_keys, uint64_t n, uint8_t* d_out, void* stream, uint64_t* occupied_out) {
    if (int s = check_batch(f, d_keys, n)) return s;
    DeviceGuard g(f->device);
    return insert_any(f, d_keys, n, d_out, stream, false, true, occupied_out);
}

int cf_insert_sorted(cf_filter* f, const void* d_keys, uint64_t n, uint8_t* d_out, void* stream,
                     uint64_t* occupied_out) {
    if (int s = check_batch(f, d_keys, n)) return s;
    DeviceGuard g(f->device);
    // (bucket << bits) | tag must fit 64 bits for the staged paths; else the plain path
    return insert_any(f, d_keys, n, d_out, stream, true, true, occupied_out);
}

int cf_contains_async(cf_filter* f, const void* d_keys, uint64_t n, uint8_t* d_out, void* stream) {
    if (int s = check_batch(f, d_keys, n)) return s;
    if (n && !d_out) return fail(CF_ERR_INVALID, "d_out is NULL with n > 0");
    DeviceGuard g(f->device);
    switch (choose_path(f, SEG_CONTAINS, n, false)) {
        case PATH_REGION:
            return staged_batch(f, stream, false, nullptr,
                                [&] { return run_region(f, SEG_CONTAINS, d_keys, n, d_out, stream); });
        case PATH_SEGMENT:
            return staged_batch(f, stream, false, nullptr,
                                [&] { return run_segmented(f, SEG_CONTAINS, d_keys, n, d_out, stream); });
        default: break;
    }
    if (int s = follow_staged(f, stream)) return s;
    LaunchCfg L = launch(f, KID_CONTAINS, stream);
    L.kpt = static_cast<int>(f->lookup_kpt);
    L.width = static_cast<int>(f->probe_width);
    CF_CUDA(f->ops->contains(dev(f), d_keys, n, d_out, L), "contains launch");
    return CF_OK;
}

int cf_contains(cf_filter* f, const void* d_keys, uint64_t n, uint8_t* d_out, void* stream) {
    if (int s = cf_contains_async(f, d_keys, n, d_out, stream)) return s;
    DeviceGuard g(f->device);
    CF_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)), "stream synchronize");
    return CF_OK;
}

int do_delete(cf_filter* f, const DevTable& t, const void* keys, uint64_t n, uint8_t* out, void* stream) {
    LaunchCfg L = launch(f, KID_DELETE, stream);
    L.width = static_cast<int>(f->probe_width);
    CF_CUDA(f->ops->remove(t, keys, n, out, L), "delete launch");
    return CF_OK;
}

// Enqueues a delete; with `wait` it returns when the delete has ended, with the occupied count.
int delete_any(cf_filter* f, const void* keys, uint64_t n, uint8_t* out, void* stream, bool wait, uint64_t* occupied_out) {
    f->known_empty = false;
    switch (choose_path(f, SEG_DELETE, n, false)) {
        case PATH_REGION:
            return staged_batch(f, stream, wait, occupied_out,
                                [&] { return run_region(f, SEG_DELETE, keys, n, out, stream); });
        case PATH_SEGMENT:
            return staged_batch(f, stream, wait, occupied_out,
                                [&] { return run_segmented(f, SEG_DELETE, keys, n, out, stream); });
        default: break;
    }
    if (int s = follow_staged(f, stream)) return s;
    if (!wait) return do_delete(f, dev(f), keys, n, out, stream);
    if (!n) return finish(f, stream, occupied_out);
    const PubRow row(f);
    if (int s = do_delete(f, row.table(), keys, n, out, stream)) return s;
    return row.finish(stream, occupied_out);
}

int cf_delete_async(cf_filter* f, const void* d_keys, uint64_t n, uint8_t* d_out, void* stream) {
    if (int s = check_batch(f, d_keys, n)) return s;
    DeviceGuard g(f->device);
    return delete_any(f, d_keys, n, d_out, stream, false, nullptr);
}

int cf_delete(cf_filter* f, const void* d_keys, uint64_t n, uint8_t* d_out, void* stream, uint64_t* occupied_out) {
    if (int s = check_batch(f, d_keys, n)) return s;
    DeviceGuard g(f->device);
    return delete_any(f, d_keys, n, d_out, stream, true, occupied_out);
}

int cf_clear(cf_filter* f, void* stream) {
    if (int s = check_filter(f)) return s;
    DeviceGuard g(f->device);
    if (int st = follow_staged(f, stream)) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    CF_CUDA(cudaMemsetAsync(f->d_table, 0, f->table_bytes, s), "table clear");
    CF_CUDA(cudaMemsetAsync(f->d_ctr, 0, CTR_COUNT * sizeof(unsigned long long), s), "counter clear");
    CF_CUDA(cudaStreamSynchronize(s), "stream synchronize");
    f->known_empty = !f->table_exposed;
    return CF_OK;
}

int cf_occupied(cf_filter* f, uint64_t* out) {
    if (int s = check_filter(f)) return s;
    if (!out) return fail(CF_ERR_INVALID, "out is NULL");
    DeviceGuard g(f->device);
    if (int s = follow_staged(f)) return s;
    unsigned long long v = 0;
    CF_CUDA(cudaMemcpy(&v, f->d_ctr + CTR_OCCUPIED, sizeof(v), cudaMemcpyDeviceToHost), "occupancy read");
    *out = v;
    return CF_OK;
}

int cf_count_occupied_slots(cf_filter* f, uint64_t* out) {
    if (int s = check_filter(f)) return s;
    if (!out) return fail(CF_ERR_INVALID, "out is NULL");
    DeviceGuard g(f->device);
    if (int s = follow_staged(f)) return s;
    unsigned long long* d_res = nullptr;
    CF_CUDA(cudaMalloc(&d_res, sizeof(unsigned long long)), "scratch allocation");
    unsigned long long v = 0;
    cudaError_t e = cudaMemset(d_res, 0, sizeof(v));
    if (e == cudaSuccess) e = f->ops->count(dev(f), f->num_buckets, d_res, launch_aux(f, nullptr));
    if (e == cudaSuccess) e = cudaMemcpy(&v, d_res, sizeof(v), cudaMemcpyDeviceToHost);
    cudaFree(d_res);
    CF_CUDA(e, "occupied-slot count");
    *out = v;
    return CF_OK;
}

int cf_get_stats(cf_filter* f, cf_stats* out) {
    if (int s = check_filter(f)) return s;
    if (!out) return fail(CF_ERR_INVALID, "out is NULL");
    DeviceGuard g(f->device);
    if (int s = follow_staged(f)) return s;
    unsigned long long c[CTR_COUNT];
    CF_CUDA(cudaMemcpy(c, f->d_ctr, sizeof(c), cudaMemcpyDeviceToHost), "counter read");
    out->occupied = c[CTR_OCCUPIED];
    out->primary = c[CTR_PRIMARY];
    out->secondary = c[CTR_SECONDARY];
    out->evicted_inserts = c[CTR_EVICTED_INSERTS];
    out->evictions = c[CTR_EVICTIONS];
    out->failed = c[CTR_FAILED];
    out->lost = c[CTR_LOST];
    out->removed = c[CTR_REMOVED];
    out->duplicates = c[CTR_DUP];
    return CF_OK;
}

int cf_get_chain_histogram(cf_filter* f, uint64_t* bins) {
    if (int s = check_filter(f)) return s;
    if (!bins) return fail(CF_ERR_INVALID, "bins is NULL");
    DeviceGuard g(f->device);
    if (int s = follow_staged(f)) return s;
    unsigned long long h[kChainBins];
    CF_CUDA(cudaMemcpy(h, f->d_ctr + CTR_HIST0, sizeof(h), cudaMemcpyDeviceToHost), "histogram read");
    for (int i = 0; i < kChainBins; ++i) bins[i] = h[i];
    return CF_OK;
}

int cf_reset_stats(cf_filter* f) {
    if (int s = check_filter(f)) return s;
    DeviceGuard g(f->device);
    if (int s = follow_staged(f)) return s;
    CF_CUDA(cudaMemset(f->d_ctr + 1, 0, (CTR_COUNT - 1) * sizeof(unsigned long long)), "counter reset");
    return CF_OK;
}

int cf_table(cf_filter* f, void** d_table, uint64_t* bytes) {
    if (int s = check_filter(f)) return s;
    if (d_table) {  // the caller may write the table at any time
        f->known_empty = false;
        f->table_exposed = true;
    }
    if (d_table) *d_table = f->d_table;
    if (bytes) *bytes = f->table_bytes;
    return CF_OK;
}

int cf_load_table(cf_filter* f, const void* src, uint64_t bytes, void* stream) {
    if (int s = check_filter(f)) return s;
    if (!src) return fail(CF_ERR_INVALID, "src is NULL");
    if (bytes != f->table_bytes)
        return fail(CF_ERR_INVALID, "image is %llu bytes, table is %llu", static_cast<unsigned long long>(bytes),
                    static_cast<unsigned long long>(f->table_bytes));
    DeviceGuard g(f->device);
    f->known_empty = false;
    if (int st = follow_staged(f, stream)) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    CF_CUDA(cudaMemcpyAsync(f->d_table, src, bytes, cudaMemcpyDefault, s), "table load");
    CF_CUDA(cudaMemsetAsync(f->d_ctr + CTR_OCCUPIED, 0, sizeof(unsigned long long), s), "counter reset");
    CF_CUDA(f->ops->count(dev(f), f->num_buckets, f->d_ctr + CTR_OCCUPIED, launch_aux(f, stream)), "recount");
    CF_CUDA(cudaStreamSynchronize(s), "stream synchronize");
    return CF_OK;
}

int cf_set_option(cf_filter* f, int option, uint64_t value) {
    if (int s = check_filter(f)) return s;
    switch (option) {
        case CF_OPT_WORKSPACE_LIMIT:
            f->ws_limit = value;
            return CF_OK;
        case CF_OPT_SEGMENTED_MIN_KEYS:
            f->seg_min_keys = value;
            return CF_OK;
        case CF_OPT_ROUND2_SEGMENTED_MIN_KEYS:
            f->round2_min = value;
            return CF_OK;
        case CF_OPT_REGION_MIN_KEYS:
            f->rg_min_keys = value;
            return CF_OK;
        case CF_OPT_STAGING:
            if (value > CF_STAGING_REGION) return fail(CF_ERR_INVALID, "unknown staging mode %llu",
                                                       static_cast<unsigned long long>(value));
            f->staging = static_cast<uint32_t>(value);
            return CF_OK;
        case CF_OPT_LOOKUP_KPT:
            if (value != 0 && value != 1 && value != 2 && value != 4)
                return fail(CF_ERR_INVALID, "lookup keys per thread must be 0, 1, 2 or 4");
            f->lookup_kpt = static_cast<uint32_t>(value);
            return CF_OK;
        case CF_OPT_PROBE_WIDTH:
            if (value > 1 && ((value & (value - 1)) != 0 || value > 32 ||
                              !((f->ops->coop_widths >> __builtin_ctzll(value)) & 1u)))
                return fail(CF_ERR_INVALID,
                            "probe width %llu not supported for %u-byte buckets (lanes of 4 or 8 bytes, at most 64 slots)",
                            static_cast<unsigned long long>(value), f->ops->bucket_bytes);
            f->probe_width = static_cast<uint32_t>(value);
            return CF_OK;
        case CF_OPT_PERSISTENT:
            if (value > 1) return fail(CF_ERR_INVALID, "persistent must be 0 or 1");
            f->persistent = static_cast<uint32_t>(value);
            return CF_OK;
        case CF_OPT_CHAIN_HISTOGRAM:
            if (value > 1) return fail(CF_ERR_INVALID, "chain histogram must be 0 or 1");
            f->chain_hist = static_cast<uint32_t>(value);
            return CF_OK;
        case CF_OPT_ROUND1_CAP:
            if (value > f->cfg.bucket_size)
                return fail(CF_ERR_INVALID, "round-1 cap must be 0 (automatic) or 1..bucket_size");
            f->round1_cap = static_cast<uint32_t>(value);
            return CF_OK;
        case CF_OPT_REGION_BYTES:
            if (value & (value - 1)) return fail(CF_ERR_INVALID, "region bytes must be 0 or a power of two");
            f->rg_bytes = value;
            init_geometry(f);
            return CF_OK;
        default:
            return fail(CF_ERR_INVALID, "unknown option %d", option);
    }
}

int cf_get_option(cf_filter* f, int option, uint64_t* value) {
    if (int s = check_filter(f)) return s;
    if (!value) return fail(CF_ERR_INVALID, "value is NULL");
    switch (option) {
        case CF_OPT_WORKSPACE_LIMIT: *value = f->ws_limit; return CF_OK;
        case CF_OPT_SEGMENTED_MIN_KEYS: *value = f->seg_min_keys; return CF_OK;
        case CF_OPT_WORKSPACE_BYTES: *value = f->ws_bytes; return CF_OK;
        case CF_OPT_ROUND2_SEGMENTED_MIN_KEYS: *value = f->round2_min; return CF_OK;
        case CF_OPT_REGION_MIN_KEYS: *value = f->rg_min_keys; return CF_OK;
        case CF_OPT_STAGING: *value = f->staging; return CF_OK;
        case CF_OPT_REGION_BYTES: *value = f->rg_bytes ? f->rg_bytes : kRgRegionBytes; return CF_OK;
        case CF_OPT_REGION_COUNT: *value = f->rgeom.nreg; return CF_OK;
        case CF_OPT_LOOKUP_KPT: *value = f->lookup_kpt; return CF_OK;
        case CF_OPT_PROBE_WIDTH: *value = f->probe_width; return CF_OK;
        case CF_OPT_PERSISTENT: *value = f->persistent; return CF_OK;
        case CF_OPT_ROUND1_CAP: *value = f->round1_cap; return CF_OK;
        case CF_OPT_CHAIN_HISTOGRAM: *value = f->chain_hist; return CF_OK;
        default: return fail(CF_ERR_INVALID, "unknown option %d", option);
    }
}

int cf_store_table(cf_filter* f, void* dst, uint64_t bytes, void* stream) {
    if (int s = check_filter(f)) return s;
    if (!dst) return fail(CF_ERR_INVALID, "dst is NULL");
    if (bytes != f->table_bytes)
        return fail(CF_ERR_INVALID, "buffer is %llu bytes, table is %llu", static_cast<unsigned long long>(bytes),
                    static_cast<unsigned long long>(f->table_bytes));
    DeviceGuard g(f->device);
    if (int st = follow_staged(f, stream)) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    CF_CUDA(cudaMemcpyAsync(dst, f->d_table, bytes, cudaMemcpyDefault, s), "table store");
    CF_CUDA(cudaStreamSynchronize(s), "stream synchronize");
    return CF_OK;
}

int cf_hash_candidates(const cf_config* cfg, uint64_t num_buckets, const void* h_keys, uint64_t n, uint64_t* i1,
                       uint64_t* i2, uint32_t* fp) {
    if (!cfg) return fail(CF_ERR_INVALID, "config is NULL");
    const uint32_t pol = cfg->alt_policy;
    if (pol > CF_ALT_OFFSET) return fail(CF_ERR_INVALID, "alt_policy must be CF_ALT_XOR, CF_ALT_ADDSUB or CF_ALT_OFFSET");
    if (num_buckets == 0 || (pol == CF_ALT_XOR && (num_buckets & (num_buckets - 1))))
        return fail(CF_ERR_INVALID, "num_buckets must be a power of two for the XOR policy, > 0 otherwise");
    if (pol == CF_ALT_ADDSUB && num_buckets % 2 != 0)
        return fail(CF_ERR_INVALID, "num_buckets must be even for the AddSub policy");
    if (n && !h_keys) return fail(CF_ERR_INVALID, "keys is NULL with n > 0");
    const uint32_t kb = cfg->key_bytes, bits = cfg->bits_per_tag;
    if ((kb != 4 && kb != 8) || (bits != 8 && bits != 16 && bits != 32))
        return fail(CF_ERR_INVALID, "key_bytes must be 4/8 and bits_per_tag 8/16/32");
    host_candidates(pol, kb, bits, num_buckets - 1, h_keys, n, i1, i2, fp);
    return CF_OK;
}

int cf_hash64(uint32_t value_bytes, const void* h_values, uint64_t n, uint64_t* out) {
    if (value_bytes != 1 && value_bytes != 2 && value_bytes != 4 && value_bytes != 8)
        return fail(CF_ERR_INVALID, "value_bytes must be 1, 2, 4 or 8");
    if (n && (!h_values || !out)) return fail(CF_ERR_INVALID, "values or out is NULL with n > 0");
    const uint8_t* p = static_cast<const uint8_t*>(h_values);
    for (uint64_t i = 0; i < n; ++i) {
        uint64_t v = 0;
        std::memcpy(&v, p + i * value_bytes, value_bytes);
        out[i] = value_bytes == 8   ? xxh64_u64(v)
                 : value_bytes == 4 ? xxh64_u32(static_cast<uint32_t>(v))
                 : value_bytes == 2 ? xxh64_u16(static_cast<uint32_t>(v))
                                    : xxh64_u8(static_cast<uint32_t>(v));
    }
    return CF_OK;
}

int cf_alt_buckets(const cf_config* cfg, uint64_t num_buckets, const uint64_t* buckets, const uint32_t* tags,
                   uint64_t n, uint64_t* out) {
    if (!cfg) return fail(CF_ERR_INVALID, "config is NULL");
    const uint32_t pol = cfg->alt_policy;
    if (pol > CF_ALT_OFFSET) return fail(CF_ERR_INVALID, "alt_policy must be CF_ALT_XOR, CF_ALT_ADDSUB or CF_ALT_OFFSET");
    if (num_buckets == 0 || (pol == CF_ALT_XOR && (num_buckets & (num_buckets - 1))))
        return fail(CF_ERR_INVALID, "num_buckets must be a power of two for the XOR policy, > 0 otherwise");
    if (pol == CF_ALT_ADDSUB && num_buckets % 2 != 0)
        return fail(CF_ERR_INVALID, "num_buckets must be even for the AddSub policy");
    if (n && (!buckets || !tags || !out)) return fail(CF_ERR_INVALID, "buckets, tags or out is NULL with n > 0");
    const uint32_t bits = cfg->bits_per_tag;
    if (bits != 8 && bits != 16 && bits != 32) return fail(CF_ERR_INVALID, "bits_per_tag must be 8, 16 or 32");
    const uint64_t nbm = num_buckets - 1;
    for (uint64_t i = 0; i < n; ++i) {
        const uint32_t t = bits == 32 ? tags[i] : (tags[i] & ((1u << bits) - 1u));
        uint64_t a;
#define CF_ALT_CASE(B)                                                                   \
    if (pol == CF_ALT_ADDSUB) a = alt_bucket<Cfg<8, B, 16, 8, ALT_ADDSUB>>(buckets[i], t, nbm); \
    else if (pol == CF_ALT_OFFSET) a = alt_bucket<Cfg<8, B, 16, 8, ALT_OFFSET>>(buckets[i], t, nbm); \
    else a = alt_bucket<Cfg<8, B, 16, 8>>(buckets[i], t, nbm);
        if (bits == 8) {
            CF_ALT_CASE(8)
        } else if (bits == 16) {
            CF_ALT_CASE(16)
        } else {
            CF_ALT_CASE(32)
        }
#undef CF_ALT_CASE
        out[i] = a;
    }
    return CF_OK;
}

int cf_probe_count(cf_filter* f, const void* d_keys, uint64_t n, uint64_t* primary_hits, void* stream) {
    if (int s = check_batch(f, d_keys, n)) return s;
    if (!primary_hits) return fail(CF_ERR_INVALID, "primary_hits is NULL");
    DeviceGuard g(f->device);
    if (int st = follow_staged(f, stream)) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    unsigned long long* d_res = nullptr;
    CF_CUDA(cudaMalloc(&d_res, sizeof(unsigned long long)), "scratch allocation");
    unsigned long long v = 0;
    cudaError_t e = cudaMemsetAsync(d_res, 0, sizeof(v), s);
    if (e == cudaSuccess) e = f->ops->probe(dev(f), d_keys, n, d_res, launch_aux(f, stream));
    if (e == cudaSuccess) e = cudaMemcpyAsync(&v, d_res, sizeof(v), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(d_res);
    CF_CUDA(e, "probe count");
    *primary_hits = v;
    return CF_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Sorted insert without allocation (cf_insert_sorted_noalloc).
//
// cf_insert_sorted grows a cudaMalloc'd workspace on demand and may free and
// re-allocate it.  Some callers cannot allow that: a cudaMalloc or cudaFree
// can synchronize the whole device (stalling the other streams of a serving
// process), and some hosts hand the library a device whose memory is already
// fully reserved by another allocator.  For them the segment-staged insert
// runs here on a fixed scratch area that is part of the library's own device
// image: a file-scope __device__ array, present on every GPU on which this
// library's code is loaded, until the process exits.  Nothing is allocated per
// call.  Like cf_insert_sorted, the call synchronizes its stream before it
// returns (it reads the per-round key counts back to the host).

namespace {

constexpr uint64_t kNoAllocMaxKeys = CF_NOALLOC_MAX_KEYS;
constexpr uint64_t kNoAllocMaxSegments = 1ull << 18;  // tables up to 16 GiB (64 KiB segments)
constexpr int kNoAllocMaxGrid = 2048;                  // radix-pass CTAs

constexpr uint64_t na_al(uint64_t x) { return (x + 255) & ~255ull; }
// Layout: two entry buffers, two payload buffers, the result bitmap (two bits
// per key, as the workspace allocator sizes it), the radix histogram, the
// segment starts and the list counters.
constexpr uint64_t kNaEnt = na_al(kNoAllocMaxKeys * 8);
constexpr uint64_t kNaPay = na_al(kNoAllocMaxKeys * 4);
constexpr uint64_t kNaBitmap = na_al((2 * kNoAllocMaxKeys + 31) / 32 * 4);
constexpr uint64_t kNaHist = na_al(static_cast<uint64_t>(kRadix) * kNoAllocMaxGrid * kRsHistSub * 4);
constexpr uint64_t kNaStart = na_al((kNoAllocMaxSegments + 1) * 4);
constexpr uint64_t kNaCnt = 256;
constexpr uint64_t kNoAllocScratchBytes = 2 * kNaEnt + 2 * kNaPay + kNaBitmap + kNaHist + kNaStart + kNaCnt;

// The scratch.  In host code this name is only a handle: the device address
// comes from cudaGetSymbolAddress (noalloc_scratch).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Device address of the scratch on the current device.  Looked up on every
// call (the lookup allocates nothing), so an address never outlives the
// context it came from, e.g. across a cudaDeviceReset.
int noalloc_scratch(void** out) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "scratch address lookup");
    *out = p;
    return CF_OK;
}

}  // namespace

extern "C" {

uint64_t cf_noalloc_scratch_bytes(void) { return kNoAllocScratchBytes; }

int cf_insert_sorted_noalloc(cf_filter* f, const void* d_keys, uint64_t n, uint8_t* d_out, void* stream,
                             uint64_t* occupied_out) {
    if (int s = check_batch(f, d_keys, n)) return s;
    if (n > kNoAllocMaxKeys)
        return fail(CF_ERR_INVALID, "%llu keys exceed the %llu-key limit of cf_insert_sorted_noalloc; split the batch",
                    static_cast<unsigned long long>(n), static_cast<unsigned long long>(kNoAllocMaxKeys));
    if (!f->seg_ok)
        return fail(CF_ERR_UNSUPPORTED, "bucket index and tag do not fit one 64-bit entry for this table");
    if (f->geom.nseg > kNoAllocMaxSegments)
        return fail(CF_ERR_UNSUPPORTED, "table of %llu segments exceeds the %llu-segment limit of the fixed scratch",
                    static_cast<unsigned long long>(f->geom.nseg), static_cast<unsigned long long>(kNoAllocMaxSegments));
    DeviceGuard g(f->device);
    f->known_empty = false;
    void* base = nullptr;
    if (int s = noalloc_scratch(&base)) return s;
    SegWork w{};
    CF_CUDA(rs_scatter_grid<0>(f->sms, &w.rs_grid[0]), "radix launch setup");
    CF_CUDA(rs_scatter_grid<1>(f->sms, &w.rs_grid[1]), "radix launch setup");
    CF_CUDA(rs_scatter_grid<2>(f->sms, &w.rs_grid[2]), "radix launch setup");
    for (int i = 0; i < 3; ++i)
        if (w.rs_grid[i] > kNoAllocMaxGrid) return fail(CF_ERR_UNSUPPORTED, "radix grid %d too large", w.rs_grid[i]);
    uint8_t* p = static_cast<uint8_t*>(base);
    w.ent[0] = reinterpret_cast<uint64_t*>(p);
    w.ent[1] = reinterpret_cast<uint64_t*>(p + kNaEnt);
    p += 2 * kNaEnt;
    w.pay[0] = reinterpret_cast<uint32_t*>(p);
    w.pay[1] = reinterpret_cast<uint32_t*>(p + kNaPay);
    p += 2 * kNaPay;
    w.bitmap = reinterpret_cast<uint32_t*>(p);
    p += kNaBitmap;
    w.hist = reinterpret_cast<uint32_t*>(p);
    p += kNaHist;
    w.start = reinterpret_cast<uint32_t*>(p);
    p += kNaStart;
    w.cnt = reinterpret_cast<unsigned long long*>(p);
    w.full = nullptr;  // no known-full bitmap in the fixed scratch: eviction probes every candidate
    w.full_words = 0;
    w.h_cnt = f->h_cnt;
    w.cap = kNoAllocMaxKeys;
    w.sms = f->sms;
    w.rg_grid = f->sms * 4;
    w.round2_segmented_min = f->round2_min ? f->round2_min : auto_threshold(f, SEG_INSERT);
    w.round1_cap = f->round1_cap;
    return staged_batch(f, stream, true, occupied_out, [&]() -> int {
        // the segment pass clears the list counters, the result bitmap and the
        // segment starts itself; the other buffers are written before read
        if (n)
            CF_CUDA(f->ops->seg_chunk(dev(f), f->geom, w, SEG_INSERT, d_keys, n, d_out, static_cast<cudaStream_t>(stream),
                                      f->cfg.eviction_policy == CF_EVICT_BFS ? 1u : 0u, f->cfg.max_evictions),
                    "segment-staged batch");
        return CF_OK;
    });
}

}  // extern "C"
