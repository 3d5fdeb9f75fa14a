// pj_global.cuh -- joins whose build side's hash table stays in L2: one
// table in the workspace, built and probed without partitioning.
//
// The partitioned path writes and reads every tuple once before the first
// lookup and takes a dozen launches; up to a few million build rows the
// whole table fits the 126 MB L2, where random 32-byte reads run at 270 G/s
// (64 MB of table; 170 G/s at 96 MB, 74 G/s at 256 MB).
//
// Unique build keys: open addressing in 32-byte buckets, so a lookup is one
// sector.  A row goes to the first free slot from its home bucket on, and a
// bucket with an empty slot ends a lookup.  A row whose key is in the table
// already is dropped: under the unique flag a probe row matches one build
// row at most.
//   4-byte keys: four slots {murmur(key), row + 1} (0: empty); the hash is the
//     key (MurmurHash3 of 4 bytes is a bijection), so the slot decides.
//   8-byte keys: eight slots of 10 hash bits and a 22-bit row; an equal
//     fingerprint compares the build key (read from its column).  Half the
//     size of {hash, row} slots, and 32-bit compare-and-swaps insert 93 G
//     rows/s where 64-bit ones insert 61 G/s.
//
// Repeated build keys: rows grouped by bucket (count, allocate, place),
// 8-byte entries {murmur(key), row} and each bucket's range; a lookup walks
// its bucket, long ones with the whole warp.
//
// Reference counterpart: hash_join (hash_join_kernels.cuh:24-200), which
// builds such a table per partition in shared memory.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "pj_device.cuh"

namespace pj {

constexpr int GT_THREADS = 256;
constexpr int GT_U = 2;                     // probe rows of a thread in flight together
constexpr int GT_TILE = GT_THREADS * GT_U;  // probe rows of one step of a CTA
constexpr int GT_STEPS = 4;                 // steps of a CTA (one where the probe side does not fill the GPU)
constexpr uint32_t GT_MAX_BUCKETS = 1u << 13;  // buckets an insert or a lookup tries
constexpr uint32_t GT_LONG = 32;            // repeated keys: ranges beyond this are walked by the warp
constexpr int GT_ROW_BITS = 22;             // 8-byte keys: row bits of a slot
constexpr int64_t GT_MAX_BUILD = int64_t(1) << GT_ROW_BITS;  // build rows of a table
constexpr int GT_STAGE = 2048;              // repeated keys: pairs a CTA stages for whole-run stores

struct GlobalOut {
    int32_t* out_build;  // nullptr: count only
    int32_t* out_probe;
    int64_t capacity;
    unsigned long long* count;
    uint32_t* status;
};

__device__ __forceinline__ uint32_t gt_bucket(uint32_t h, uint32_t nb) { return __umulhi(h, nb); }

// One bucket: a 32-byte request.
__device__ __forceinline__ void gt_load_bucket(const uint32_t* __restrict__ table, uint32_t b, uint32_t (&w)[8])
{
    asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                 : "l"(table + static_cast<size_t>(b) * 8));
}

// Slots of a key width.
template <typename K> struct GtSlots;

template <> struct GtSlots<int32_t> {
    static constexpr uint32_t N = 4;
    static constexpr bool EXACT = true;
    using Word = unsigned long long;
    __device__ __forceinline__ static Word make(uint32_t h, uint32_t row)
    {
        return (static_cast<Word>(h) << 32) | (row + 1u);
    }
    __device__ __forceinline__ static bool same_tag(Word a, Word b) { return (a >> 32) == (b >> 32); }
    __device__ __forceinline__ static uint32_t row_of(Word w) { return static_cast<uint32_t>(w) - 1u; }
    // the row of a slot with the hash's tag (the last one), or -1
    __device__ __forceinline__ static int32_t candidate(const uint32_t (&w)[8], uint32_t h, bool& full)
    {
        int32_t r = -1;
        full = true;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const bool used = w[2 * s] != 0u;
            if (used && w[2 * s + 1] == h) r = static_cast<int32_t>(w[2 * s] - 1u);
            full = full && used;
        }
        return r;
    }
};

template <> struct GtSlots<int64_t> {
    static constexpr uint32_t N = 8;
    static constexpr bool EXACT = false;
    using Word = uint32_t;
    __device__ __forceinline__ static uint32_t tag(uint32_t h)
    {
        const uint32_t t = h & ((1u << (32 - GT_ROW_BITS)) - 1u);
        return t ? t : 1u;  // a used slot is never 0
    }
    __device__ __forceinline__ static Word make(uint32_t h, uint32_t row) { return (tag(h) << GT_ROW_BITS) | row; }
    __device__ __forceinline__ static bool same_tag(Word a, Word b) { return (a ^ b) >> GT_ROW_BITS == 0u; }
    __device__ __forceinline__ static uint32_t row_of(Word w) { return w & ((1u << GT_ROW_BITS) - 1u); }
    __device__ __forceinline__ static int32_t candidate(const uint32_t (&w)[8], uint32_t h, bool& full)
    {
        const uint32_t want = tag(h);
        int32_t r = -1;
        full = true;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            if (w[s] >> GT_ROW_BITS == want) r = static_cast<int32_t>(row_of(w[s]));
            full = full && w[s] != 0u;
        }
        return r;
    }
};

// Inserts build row `row` with hash h.  Home slots differ by hash bits, so
// most inserts take one compare-and-swap.
template <typename K>
__device__ __forceinline__ void gt_insert(const K* __restrict__ keys, uint32_t* table, uint32_t nb, K key,
                                          uint32_t row, uint32_t* status)
{
    using S = GtSlots<K>;
    const uint32_t h = hash_key(key);
    const typename S::Word e = S::make(h, row);
    uint32_t b = gt_bucket(h, nb);
    for (uint32_t t = 0; t < GT_MAX_BUCKETS; ++t) {
        // another row has given up: this build has failed
        if ((t & 63u) == 63u && (*static_cast<volatile uint32_t*>(status) & ST_OVERFLOW)) return;
        auto* slot = reinterpret_cast<typename S::Word*>(table + static_cast<size_t>(b) * 8);
#pragma unroll 1
        for (uint32_t j = 0; j < S::N; ++j) {
            const typename S::Word old = atomicCAS(slot + ((h + j) & (S::N - 1u)), typename S::Word(0), e);
            if (old == 0) return;
            if (S::same_tag(old, e) && (S::EXACT || keys[S::row_of(old)] == key)) return;  // repeated key
        }
        if (++b == nb) b = 0;
    }
    raise_status(status, ST_OVERFLOW);
}

// Build: one row a thread (many independent compare-and-swap chains), and
// the output count's reset.
template <typename K>
__global__ void __launch_bounds__(GT_THREADS) gt_build_kernel(const K* __restrict__ keys, uint32_t n, uint32_t* table,
                                                              uint32_t nb, unsigned long long* count,
                                                              uint32_t* status)
{
    const uint32_t i = blockIdx.x * GT_THREADS + threadIdx.x;
    if (i == 0) *count = 0;
    if (i < n) gt_insert<K>(keys, table, nb, keys[i], i, status);
}

// This thread's two probe keys: rows 2t, 2t + 1 of the tile, one load
// streamed past L1 and marked evict-first in L2 (the table should stay).
// vec: the column starts on a 16-byte boundary (batches take any).
template <typename K>
__device__ __forceinline__ void gt_load_pair(const K* __restrict__ keys, bool vec, uint32_t n, uint32_t row0,
                                             K (&k)[GT_U])
{
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    if (vec && row0 + 1 < n) {
        if constexpr (sizeof(K) == 4) {
            uint32_t x, y;
            asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.u32 {%0, %1}, [%2], %3;"
                         : "=r"(x), "=r"(y)
                         : "l"(keys + row0), "l"(pol));
            k[0] = static_cast<K>(x);
            k[1] = static_cast<K>(y);
        } else {
            uint64_t x, y;
            asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v2.u64 {%0, %1}, [%2], %3;"
                         : "=l"(x), "=l"(y)
                         : "l"(keys + row0), "l"(pol));
            k[0] = static_cast<K>(x);
            k[1] = static_cast<K>(y);
        }
    } else {
        k[0] = row0 < n ? keys[row0] : K(0);
        k[1] = row0 + 1 < n ? keys[row0 + 1] : K(0);
    }
}

// The whole search for one key, bucket by bucket, every slot with its tag
// compared: the rare case after a full home bucket or a fingerprint of
// another key.
template <typename K>
__device__ __forceinline__ int32_t gt_search(const K* __restrict__ bkeys, const uint32_t* __restrict__ table, uint32_t nb,
                                          K key, uint32_t h)
{
    using S = GtSlots<K>;
    uint32_t b = gt_bucket(h, nb);
#pragma unroll 1
    for (uint32_t t = 0; t < GT_MAX_BUCKETS; ++t) {
        uint32_t w[8];
        gt_load_bucket(table, b, w);
        bool full;
        const int32_t r = S::candidate(w, h, full);
        if (r >= 0) {
            if constexpr (S::EXACT) {
                return r;
            } else {
#pragma unroll
                for (int s = 0; s < 8; ++s)
                    if (S::same_tag(w[s], S::make(h, 0)) && bkeys[S::row_of(w[s])] == key)
                        return static_cast<int32_t>(S::row_of(w[s]));
            }
        }
        if (!full) return -1;
        if (++b == nb) b = 0;
    }
    return -1;
}

// Positions of a CTA's matches in the output: n of this thread, dense over
// the block; one global atomic per CTA (one per warp serialised on the
// counter).  Returns the position of the thread's first match; *block_first
// and *block_total (optional) are the CTA's.
__device__ __forceinline__ unsigned long long gt_reserve(unsigned long long n, unsigned long long* s_warp,
                                                         unsigned long long* count)
{
    constexpr int NW = GT_THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long all = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            const unsigned long long x = s_warp[w];
            s_warp[w] = all;
            all += x;
        }
        s_warp[NW + 1] = all;
        s_warp[NW] = all ? atomicAdd(count, all) : 0ull;
    }
    __syncthreads();
    return s_warp[NW] + s_warp[warp] + incl - n;
}

__device__ __forceinline__ void gt_store_pair(const GlobalOut& o, unsigned long long pos, int32_t b, uint32_t q)
{
    if (pos < static_cast<unsigned long long>(o.capacity)) {
        __stcs(o.out_build + pos, b);
        __stcs(o.out_probe + pos, static_cast<int32_t>(q));
    } else {
        raise_status(o.status, ST_CAPACITY);
    }
}

// Probe of the unique table, STEPS tiles of GT_TILE rows per CTA.  Bound by
// the latency of its chain (key, bucket, for 8-byte keys the build key, then
// the output reservation): two rows a thread at a time keep the registers
// low, and all steps share one reservation -- with one per 512 rows every
// third stall was its barrier (3 M x 10 M 8-byte keys: 112 us).
template <typename K, int STEPS>
__device__ __forceinline__ void gt_probe_block(const K* __restrict__ pkeys, bool vec, uint32_t n,
                                               const K* __restrict__ bkeys, const uint32_t* __restrict__ table,
                                               uint32_t nb, const GlobalOut& o, uint32_t block_row)
{
    using S = GtSlots<K>;
    __shared__ unsigned long long s_warp[GT_THREADS / 32 + 2];
    const uint32_t row0 = block_row + threadIdx.x * GT_U;
    int32_t m[STEPS][GT_U];
    uint32_t again = 0;  // bit j * GT_U + u: that row needs the whole search
    K k[GT_U], nk[GT_U];
    gt_load_pair<K>(pkeys, vec, n, row0, nk);
#pragma unroll
    for (int j = 0; j < STEPS; ++j) {
        const uint32_t r0 = row0 + j * GT_TILE;
        uint32_t h[GT_U];
        bool unsure[GT_U];
        uint32_t w[GT_U][8];
#pragma unroll
        for (int u = 0; u < GT_U; ++u) {
            k[u] = nk[u];
            h[u] = hash_key(k[u]);
            gt_load_bucket(table, gt_bucket(h[u], nb), w[u]);
        }
        if (j + 1 < STEPS) gt_load_pair<K>(pkeys, vec, n, r0 + GT_TILE, nk);
#pragma unroll
        for (int u = 0; u < GT_U; ++u) {
            bool full;
            m[j][u] = S::candidate(w[u], h[u], full);
            unsure[u] = m[j][u] < 0 && full;
        }
        if constexpr (!S::EXACT) {
            K c[GT_U];
#pragma unroll
            for (int u = 0; u < GT_U; ++u) c[u] = m[j][u] >= 0 ? __ldg(bkeys + m[j][u]) : k[u];
#pragma unroll
            for (int u = 0; u < GT_U; ++u) unsure[u] = unsure[u] || c[u] != k[u];
        }
#pragma unroll
        for (int u = 0; u < GT_U; ++u) {
            if (r0 + u >= n) m[j][u] = -1;
            else if (unsure[u]) again |= 1u << (j * GT_U + u);
        }
    }
    for (; again; again &= again - 1u) {
        const int i = __ffs(again) - 1;
        const K key = pkeys[row0 + (i / GT_U) * GT_TILE + i % GT_U];
        const int32_t r = gt_search<K>(bkeys, table, nb, key, hash_key(key));
#pragma unroll
        for (int j = 0; j < STEPS; ++j)
#pragma unroll
            for (int u = 0; u < GT_U; ++u)
                if (i == j * GT_U + u) m[j][u] = r;
    }
    // positions inside the warp by step and row of the pair: every store
    // instruction writes one run
    const uint32_t lt = (1u << (threadIdx.x & 31)) - 1u;
    uint32_t off[STEPS][GT_U], total = 0;
#pragma unroll
    for (int j = 0; j < STEPS; ++j)
#pragma unroll
        for (int u = 0; u < GT_U; ++u) {
            const uint32_t bal = __ballot_sync(0xffffffffu, m[j][u] >= 0);
            off[j][u] = total + __popc(bal & lt);
            total += __popc(bal);
        }
    // lane 31 speaks for the warp: its position is the warp's base
    const unsigned long long at = gt_reserve((threadIdx.x & 31) == 31 ? total : 0u, s_warp, o.count);
    const unsigned long long base = __shfl_sync(0xffffffffu, at, 31);
    if (o.out_build == nullptr) return;
#pragma unroll
    for (int j = 0; j < STEPS; ++j)
#pragma unroll
        for (int u = 0; u < GT_U; ++u)
            if (m[j][u] >= 0) gt_store_pair(o, base + off[j][u], m[j][u], row0 + j * GT_TILE + u);
}

template <typename K, int STEPS>
__global__ void __launch_bounds__(GT_THREADS, STEPS == 1 ? 2048 / GT_THREADS : 1536 / GT_THREADS)
    gt_probe_kernel(const K* __restrict__ pkeys, uint32_t n, const K* __restrict__ bkeys,
                    const uint32_t* __restrict__ table, uint32_t nb, GlobalOut o)
{
    gt_probe_block<K, STEPS>(pkeys, true, n, bkeys, table, nb, o, blockIdx.x * (STEPS * GT_TILE));
}

// ---- batches -----------------------------------------------------------------
// Many joins, a group at a time: the tables of a group lie side by side in one
// region that stays in L2, one launch builds them and one probes them.  Every
// CTA takes one item {join, first row} of a table made when the batch was
// prepared.
struct GtJob {
    const void* build;
    const void* probe;
    int32_t* out_build;  // nullptr: count only
    int32_t* out_probe;
    int64_t capacity;
    unsigned long long* count;
    uint32_t n_build, n_probe;
    uint32_t nb;            // buckets
    uint32_t first_bucket;  // in the group's region
    uint32_t vec;           // the probe column starts on 16 bytes
    uint32_t pad;
};
struct GtItem {
    uint32_t job;
    uint32_t row0;
};
constexpr uint32_t GT_BUILD_ITEM = 4 * GT_THREADS;      // build rows of an item (GT_THREADS in a small batch)
constexpr uint32_t GT_PROBE_ITEM = GT_STEPS * GT_TILE;  // probe rows of an item (GT_TILE in a small batch)

template <typename K>
__global__ void __launch_bounds__(GT_THREADS) gt_batch_build_kernel(const GtJob* __restrict__ jobs,
                                                                    const GtItem* __restrict__ items,
                                                                    uint32_t item_rows, uint32_t* region,
                                                                    uint32_t* status)
{
    const GtItem it = items[blockIdx.x];
    const GtJob* __restrict__ J = jobs + it.job;
    const K* keys = static_cast<const K*>(J->build);
    uint32_t* table = region + static_cast<size_t>(J->first_bucket) * 8;
    const uint32_t n = J->n_build, nb = J->nb;
    if (it.row0 == 0 && threadIdx.x == 0) *J->count = 0;
#pragma unroll 1
    for (uint32_t i = it.row0 + threadIdx.x; i < n && i < it.row0 + item_rows; i += GT_THREADS)
        gt_insert<K>(keys, table, nb, keys[i], i, status);
}

template <typename K, int STEPS>
__global__ void __launch_bounds__(GT_THREADS, STEPS == 1 ? 2048 / GT_THREADS : 1536 / GT_THREADS)
    gt_batch_probe_kernel(const GtJob* __restrict__ jobs, const GtItem* __restrict__ items,
                          const uint32_t* __restrict__ region, uint32_t* status)
{
    const GtItem it = items[blockIdx.x];
    const GtJob* __restrict__ J = jobs + it.job;
    const GlobalOut o{J->out_build, J->out_probe, J->capacity, J->count, status};
    gt_probe_block<K, STEPS>(static_cast<const K*>(J->probe), J->vec != 0, J->n_probe,
                                static_cast<const K*>(J->build), region + static_cast<size_t>(J->first_bucket) * 8,
                                J->nb, o, it.row0);
}

// ---- repeated build keys ---------------------------------------------------

template <typename K>
__global__ void __launch_bounds__(GT_THREADS) gt_count_kernel(const K* __restrict__ keys, uint32_t n,
                                                              uint32_t* counts, uint32_t nb,
                                                              unsigned long long* count)
{
    const uint32_t i = blockIdx.x * GT_THREADS + threadIdx.x;
    if (i == 0) *count = 0;
    if (i < n) atomicAdd(&counts[gt_bucket(hash_key(keys[i]), nb)], 1u);
}

// Entry ranges of the buckets, range[b] = {start, start}: the buckets of a
// CTA lie one after another, the CTAs in whatever order they come (one
// atomic each instead of a scan over all of them).
constexpr int GT_ALLOC = 8;  // buckets per thread
static __global__ void __launch_bounds__(GT_THREADS) gt_alloc_kernel(const uint32_t* __restrict__ counts, uint32_t nb,
                                                              uint2* __restrict__ range, unsigned long long* cursor)
{
    __shared__ unsigned long long s_warp[GT_THREADS / 32 + 2];
    const uint32_t b0 = (blockIdx.x * GT_THREADS + threadIdx.x) * GT_ALLOC;
    uint32_t c[GT_ALLOC], sum = 0;
#pragma unroll
    for (int j = 0; j < GT_ALLOC; ++j) {
        c[j] = b0 + j < nb ? counts[b0 + j] : 0u;
        sum += c[j];
    }
    uint32_t at = static_cast<uint32_t>(gt_reserve(sum, s_warp, cursor));
#pragma unroll
    for (int j = 0; j < GT_ALLOC; ++j) {
        if (b0 + j < nb) range[b0 + j] = make_uint2(at, at);
        at += c[j];
    }
}

// range[b].y moves from the bucket's start to its end
template <typename K>
__global__ void __launch_bounds__(GT_THREADS) gt_place_kernel(const K* __restrict__ keys, uint32_t n, uint2* range,
                                                              uint32_t nb, uint2* __restrict__ entries)
{
    const uint32_t i = blockIdx.x * GT_THREADS + threadIdx.x;
    if (i >= n) return;
    const uint32_t h = hash_key(keys[i]);
    entries[atomicAdd(&range[gt_bucket(h, nb)].y, 1u)] = make_uint2(h, i);
}

// Probe of the grouped rows: a counting walk, then a writing walk at the
// positions it gave (the entries are in L1 by then).  A CTA's pairs pass
// through shared memory so that they leave as whole runs: single pairs
// stored by their finders were L2-request bound (4 M probe rows, 9.6 M
// pairs: 170 us).
template <typename K>
__global__ void __launch_bounds__(GT_THREADS) gt_probe_multi_kernel(const K* __restrict__ pkeys, uint32_t n,
                                                                    const K* __restrict__ bkeys,
                                                                    const uint2* __restrict__ range, uint32_t nb,
                                                                    const uint2* __restrict__ entries, GlobalOut o)
{
    __shared__ unsigned long long s_warp[GT_THREADS / 32 + 2];
    __shared__ uint2 s_pair[GT_STAGE];
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t row0 = blockIdx.x * GT_TILE + threadIdx.x * GT_U;
    K k[GT_U];
    uint32_t h[GT_U], lo[GT_U], hi[GT_U], c[GT_U];
    gt_load_pair<K>(pkeys, true, n, row0, k);
#pragma unroll
    for (int u = 0; u < GT_U; ++u) {
        h[u] = hash_key(k[u]);
        uint2 r = make_uint2(0u, 0u);
        if (row0 + u < n) r = __ldg(range + gt_bucket(h[u], nb));
        lo[u] = r.x;
        hi[u] = r.y;
    }
    auto equal = [&](const uint2& e, uint32_t hh, K kk) -> bool {
        return e.x == hh && (sizeof(K) == 4 || bkeys[e.y] == kk);
    };
    unsigned long long mine = 0;
#pragma unroll
    for (int u = 0; u < GT_U; ++u) {
        c[u] = 0;
        const bool is_long = hi[u] - lo[u] > GT_LONG;
        if (!is_long)
            for (uint32_t i = lo[u]; i < hi[u]; ++i) c[u] += equal(__ldg(entries + i), h[u], k[u]) ? 1u : 0u;
        for (uint32_t todo = __ballot_sync(0xffffffffu, is_long); todo; todo &= todo - 1u) {
            const int owner = __ffs(todo) - 1;
            const uint32_t a = __shfl_sync(0xffffffffu, lo[u], owner), z = __shfl_sync(0xffffffffu, hi[u], owner);
            const uint32_t hh = __shfl_sync(0xffffffffu, h[u], owner);
            const K kk = __shfl_sync(0xffffffffu, k[u], owner);
            uint32_t found = 0;
            for (uint32_t i = a + lane; i < z; i += 32) found += equal(__ldg(entries + i), hh, kk) ? 1u : 0u;
            found = __reduce_add_sync(0xffffffffu, found);
            if (lane == owner) c[u] = found;
        }
        mine += c[u];
    }
    unsigned long long pos = gt_reserve(mine, s_warp, o.count);
    if (o.out_build == nullptr) return;
    const unsigned long long first = s_warp[GT_THREADS / 32], all = s_warp[GT_THREADS / 32 + 1];
    const bool staged = all <= GT_STAGE;
    auto put = [&](unsigned long long at, uint32_t b, uint32_t q) {
        if (staged) s_pair[at - first] = make_uint2(b, q);
        else gt_store_pair(o, at, static_cast<int32_t>(b), q);
    };
#pragma unroll
    for (int u = 0; u < GT_U; ++u) {
        const bool is_long = hi[u] - lo[u] > GT_LONG;
        if (!is_long && c[u] > 0)
            for (uint32_t i = lo[u]; i < hi[u]; ++i) {
                const uint2 e = __ldg(entries + i);
                if (equal(e, h[u], k[u])) put(pos++, e.y, row0 + u);
            }
        for (uint32_t todo = __ballot_sync(0xffffffffu, is_long && c[u] > 0); todo; todo &= todo - 1u) {
            const int owner = __ffs(todo) - 1;
            const uint32_t a = __shfl_sync(0xffffffffu, lo[u], owner), z = __shfl_sync(0xffffffffu, hi[u], owner);
            const uint32_t hh = __shfl_sync(0xffffffffu, h[u], owner);
            const uint32_t r = __shfl_sync(0xffffffffu, row0 + u, owner);
            const K kk = __shfl_sync(0xffffffffu, k[u], owner);
            unsigned long long at = __shfl_sync(0xffffffffu, pos, owner);
            for (uint32_t i0 = a; i0 < z; i0 += 32) {
                const uint32_t i = i0 + lane;
                uint2 e = make_uint2(0u, 0u);
                if (i < z) e = __ldg(entries + i);
                const bool hit = i < z && equal(e, hh, kk);
                const uint32_t bal = __ballot_sync(0xffffffffu, hit);
                if (hit) put(at + __popc(bal & lt), e.y, r);
                at += __popc(bal);
            }
            if (lane == owner) pos = at;
        }
    }
    if (!staged) return;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < static_cast<uint32_t>(all); i += GT_THREADS) {
        const uint2 p = s_pair[i];
        gt_store_pair(o, first + i, static_cast<int32_t>(p.x), p.y);
    }
}

}  // namespace pj
