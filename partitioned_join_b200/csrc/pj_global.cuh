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
// entries {murmur(key), row} or, of 8-byte keys, {key, row}, and each bucket's
// range; a lookup walks its bucket.  Long buckets are left to a second launch, which cuts them into
// slices over the whole GPU, whatever probe rows meet them.
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
constexpr uint32_t GT_LONG = 32;            // repeated keys: longer ranges are walked by the warp or cut into slices
constexpr int GT_WALK_U = 4;                // entries of a short range in flight a lane
constexpr int GT_SLICE_U = 2;               // entries of a slice's step in flight a lane
constexpr uint32_t GT_SLICE = 32 * GT_SLICE_U;  // entries of a slice's step
constexpr int GT_SLICES = 4;                // slices of a warp in flight together
constexpr uint32_t GT_ROUND = GT_THREADS / 32 * GT_SLICES;  // slices of a CTA's round
// From GT_WALK_PROBE probe rows on, whose tiles fill the GPU, the finder's warp
// walks ranges of up to GT_WALK entries (runs of 96 4-byte rows a key, 2^16
// probe rows: 93 us walked, 50 cut; 2^18: 100 and 126; 2^20: 263 and 421; of
// 600 rows 2^20: 1198 and 1900).  Entries that hold an 8-byte key are twice the
// size (2^20 probe rows, runs of 96: 384 and 499; 256: 820 and 892; 600, before
// whole runs were stored at once: 1943 and 1982); those that do not are cut, since
// a walk waits for a build key at every step (2^20 x 2^19 rows, runs of 40: 312 and
// 255; 256: 1287 and 878).
constexpr int64_t GT_WALK_PROBE = int64_t(1) << 18;
constexpr uint32_t GT_WALK_32 = 1024, GT_WALK_64 = 256;
constexpr unsigned GT_LONG_CTAS = 4;        // CTAs per SM of the launch for them
constexpr int GT_ROW_BITS = 22;             // 8-byte keys: row bits of a slot
constexpr int64_t GT_MAX_BUILD = int64_t(1) << GT_ROW_BITS;  // build rows of a table
constexpr uint32_t GT_STAGE = 256;          // repeated keys: pairs a warp stages for whole-run stores

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

// A kernel of the chain below: the next one may be put in place, and this one
// goes on when the one before has ended and its writes are visible.  (What
// that one wrote is read by plain loads: a non-coherent load wants memory that
// nobody writes while its kernel is there, and one put in place ahead is there
// by then; gt_probe_multi_kernel, which is not, reads entries by such loads.)
__device__ __forceinline__ void gt_wait_before()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ uint2 gt_load(const uint2* p)
{
    uint2 v;
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

// One sector of entries: those at p and after it.
__device__ __forceinline__ void gt_load_sector(const uint2* p, uint2 (&e)[4])
{
    uint32_t w[8];
    gt_load_bucket(reinterpret_cast<const uint32_t*>(p), 0, w);
#pragma unroll
    for (int v = 0; v < 4; ++v) e[v] = make_uint2(w[2 * v], w[2 * v + 1]);
}
__device__ __forceinline__ void gt_load_sector(const uint4* p, uint4 (&e)[2])
{
    uint32_t w[8];
    gt_load_bucket(reinterpret_cast<const uint32_t*>(p), 0, w);
#pragma unroll
    for (int v = 0; v < 2; ++v) e[v] = make_uint4(w[4 * v], w[4 * v + 1], w[4 * v + 2], w[4 * v + 3]);
}

__device__ __forceinline__ uint4 gt_load(const uint4* p)
{
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// ---- repeated build keys ---------------------------------------------------

// One build row among those of its bucket.  Narrow: {hash, row}; an equal hash
// of an 8-byte key is compared with the build key, read from its column.  Wide
// (8-byte keys): {key, row}, which saves a random sector a pair where the probe
// side is no smaller than the build side (2^20 x 2^24 rows, four a key: 802 ->
// 681 us by itself).
template <typename K, bool WIDE> struct GtEntry {
    using T = uint2;
    static constexpr uint32_t SECTOR = 4;  // entries of 32 bytes
    __device__ __forceinline__ static T make(uint32_t h, K, uint32_t row) { return make_uint2(h, row); }
    __device__ __forceinline__ static T none(uint32_t h, K) { return make_uint2(~h, 0u); }  // equal to no such key
    __device__ __forceinline__ static uint32_t row(const T& e) { return e.y; }
    __device__ __forceinline__ static bool equal(const T& e, uint32_t h, K key, const K* __restrict__ bkeys)
    {
        return e.x == h && (sizeof(K) == 4 || bkeys[e.y] == key);
    }
};
template <> struct GtEntry<int64_t, true> {
    using T = uint4;
    static constexpr uint32_t SECTOR = 2;
    __device__ __forceinline__ static T make(uint32_t, int64_t key, uint32_t row)
    {
        return make_uint4(static_cast<uint32_t>(key), static_cast<uint32_t>(key >> 32), row, 0u);
    }
    __device__ __forceinline__ static T none(uint32_t, int64_t key) { return make(0u, ~key, 0u); }
    __device__ __forceinline__ static uint32_t row(const T& e) { return e.z; }
    __device__ __forceinline__ static bool equal(const T& e, uint32_t, int64_t key, const int64_t* __restrict__)
    {
        return e.x == static_cast<uint32_t>(key) && e.y == static_cast<uint32_t>(key >> 32);
    }
};

template <typename K>
__global__ void __launch_bounds__(GT_THREADS) gt_count_kernel(const K* __restrict__ keys, uint32_t n,
                                                              uint32_t* counts, uint32_t nb,
                                                              unsigned long long* count)
{
    gt_wait_before();
    const uint32_t i = blockIdx.x * GT_THREADS + threadIdx.x;
    if (i == 0) *count = 0;
    if (i < n) atomicAdd(&counts[gt_bucket(hash_key(keys[i]), nb)], 1u);
}

// Entry ranges of the buckets, range[b] = {start, start}: the buckets of a
// CTA lie one after another, the CTAs in whatever order they come (one
// atomic each instead of a scan over all of them).
constexpr int GT_ALLOC = 8;  // buckets per thread
static __global__ void __launch_bounds__(GT_THREADS) gt_alloc_kernel(const uint32_t* counts, uint32_t nb,
                                                              uint2* range, unsigned long long* cursor)
{
    __shared__ unsigned long long s_warp[GT_THREADS / 32 + 2];
    gt_wait_before();
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
template <typename K, bool WIDE>
__global__ void __launch_bounds__(GT_THREADS) gt_place_kernel(const K* __restrict__ keys, uint32_t n, uint2* range,
                                                              uint32_t nb,
                                                              typename GtEntry<K, WIDE>::T* __restrict__ entries)
{
    gt_wait_before();
    const uint32_t i = blockIdx.x * GT_THREADS + threadIdx.x;
    if (i >= n) return;
    const K key = keys[i];
    const uint32_t h = hash_key(key);
    entries[atomicAdd(&range[gt_bucket(h, nb)].y, 1u)] = GtEntry<K, WIDE>::make(h, key, i);
}

// Count, allocate and place by one CTA, the buckets' counts in shared memory,
// and what a memset would clear (head): four launches' work in one for builds
// of up to GT_GROUP rows, whose joins wait for launches.
constexpr int GT_GROUP_THREADS = 1024;
constexpr int64_t GT_GROUP = 4096;
template <typename K, bool WIDE>
__global__ void __launch_bounds__(GT_GROUP_THREADS) gt_group_kernel(const K* __restrict__ keys, uint32_t n,
                                                                    uint32_t nb, uint32_t* head, int head_words,
                                                                    uint2* __restrict__ range,
                                                                    typename GtEntry<K, WIDE>::T* __restrict__ entries,
                                                                    unsigned long long* count)
{
    constexpr int U = 4;  // rows of a thread in flight
    constexpr uint32_t T = GT_GROUP_THREADS;
    __shared__ uint32_t s_at[GT_GROUP];  // counts, then places
    __shared__ uint32_t s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t b = threadIdx.x; b < nb; b += T) s_at[b] = 0u;
    for (int i = threadIdx.x; i < head_words; i += T) head[i] = 0u;
    if (threadIdx.x == 0) *count = 0;
    auto each = [&](auto&& f) {
        for (uint32_t i0 = threadIdx.x; i0 < n; i0 += U * T) {
            K k[U];
#pragma unroll
            for (int u = 0; u < U; ++u) k[u] = i0 + u * T < n ? keys[i0 + u * T] : K(0);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (i0 + u * T < n) f(i0 + u * T, k[u], hash_key(k[u]));
        }
    };
    __syncthreads();
    each([&](uint32_t, K, uint32_t h) { atomicAdd(&s_at[gt_bucket(h, nb)], 1u); });
    __syncthreads();
    // (an odd run: the lanes walk 32 banks)
    const uint32_t run = ((nb + T - 1) / T) | 1u, b0 = threadIdx.x * run, b1 = min(b0 + run, nb);
    uint32_t sum = 0;
    for (uint32_t b = b0; b < b1; ++b) sum += s_at[b];
    uint32_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t at = incl - sum + __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[lane] : 0u);
    for (uint32_t b = b0; b < b1; ++b) {
        const uint32_t c = s_at[b];
        s_at[b] = at;
        range[b] = make_uint2(at, at + c);
        at += c;
    }
    __syncthreads();
    each([&](uint32_t i, K key, uint32_t h) {
        entries[atomicAdd(&s_at[gt_bucket(h, nb)], 1u)] = GtEntry<K, WIDE>::make(h, key, i);
    });
}

// Probe rows that meet a long range, for gt_probe_long_kernel: one word per
// warp of gt_probe_multi_kernel (64 probe rows) that has such rows, and a
// cursor over words and rounds of GT_ROUND slices.
struct GtLong {
    unsigned long long* cursor;  // words << round_bits | rounds
    unsigned long long* list;    // unit << round_bits | rounds of the words before it
    int32_t round_bits;
    uint32_t slice;              // entries of a slice: a multiple of GT_SLICE
    uint32_t walk;               // longer ranges are cut
    __device__ __forceinline__ uint32_t slices(uint32_t entries) const
    {
        return entries > walk ? (entries + slice - 1) / slice : 0u;
    }
};

// Probe of the grouped rows, bound by the latency of its loads (key, range,
// entries).  A range is read in whole sectors, both rows of a lane together:
// entry by entry a lane came back to its L1 line several times, and the lines of
// 1300 lanes evict each other before it does (2^20 x 2^24 rows, 16 a key: 2.07 ->
// 1.48 ms; a larger stage, which leaves less L1, 2.35).  A warp's pairs pass
// through shared memory, so that they leave in runs of 256 however many a row
// has; with 2048 staged a CTA, what did not fit was stored by its finders (the
// same join 5.46 ms; four rows a key 585 -> 339 us).  Wide entries need 64
// registers: five CTAs an SM would spill them (2^20 x 2^24, 4 a key: 466 -> 554).
template <typename K, bool WIDE>
__global__ void __launch_bounds__(GT_THREADS, WIDE ? 4 : 5)
    gt_probe_multi_kernel(const K* __restrict__ pkeys, uint32_t n, const K* __restrict__ bkeys, const uint2* range,
                          uint32_t nb, const typename GtEntry<K, WIDE>::T* entries, GtLong later, GlobalOut o)
{
    __shared__ unsigned long long s_warp[GT_THREADS / 32 + 2];
    __shared__ uint2 s_pair[GT_THREADS / 32][GT_STAGE];
    using E = GtEntry<K, WIDE>;
    gt_wait_before();
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t row0 = blockIdx.x * GT_TILE + threadIdx.x * GT_U;
    K k[GT_U];
    uint32_t h[GT_U], lo[GT_U], hi[GT_U];
    uint2* stage = s_pair[threadIdx.x >> 5];
    gt_load_pair<K>(pkeys, true, n, row0, k);
    uint32_t slices = 0;
#pragma unroll
    for (int u = 0; u < GT_U; ++u) {
        h[u] = hash_key(k[u]);
        uint2 r = make_uint2(0u, 0u);
        if (row0 + u < n) r = gt_load(range + gt_bucket(h[u], nb));
        const uint32_t s = later.slices(r.y - r.x);
        slices += s;
        lo[u] = r.x;
        hi[u] = s ? r.x : r.y;
    }
    slices = __reduce_add_sync(0xffffffffu, slices);
    if (slices && lane == 0) {
        const unsigned long long rounds = (slices + GT_ROUND - 1) / GT_ROUND;
        const unsigned long long at = atomicAdd(later.cursor, (1ull << later.round_bits) + rounds);
        const unsigned long long unit = row0 / (32 * GT_U);
        later.list[at >> later.round_bits] = (unit << later.round_bits) | (at & ((1ull << later.round_bits) - 1ull));
    }
    // The walk of the short ranges, sector by sector: the pairs go to the warp's
    // stage while it has room, a bit of hit[u] stands for one that did not fit.
    constexpr uint32_t S = E::SECTOR;
    const bool write = o.out_build != nullptr;
    uint32_t staged = 0, at0[GT_U], hit[GT_U], span[GT_U], longest = 0;
#pragma unroll
    for (int u = 0; u < GT_U; ++u) {
        at0[u] = lo[u] & ~(S - 1u);
        span[u] = hi[u] == lo[u] || hi[u] - at0[u] > GT_LONG ? 0u : hi[u] - at0[u];
        longest = max(longest, span[u]);
        hit[u] = 0;
    }
    longest = __reduce_max_sync(0xffffffffu, longest);
    for (uint32_t i = 0; i < longest; i += GT_WALK_U) {
        typename E::T e[GT_U][GT_WALK_U / S][S];
        bool eq[GT_U][GT_WALK_U];
#pragma unroll
        for (int u = 0; u < GT_U; ++u)
#pragma unroll
            for (uint32_t v = 0; v < GT_WALK_U; v += S)
                if (i + v < span[u]) gt_load_sector(entries + at0[u] + i + v, e[u][v / S]);
#pragma unroll
        for (int u = 0; u < GT_U; ++u)
#pragma unroll
            for (uint32_t v = 0; v < GT_WALK_U; ++v)
                eq[u][v] = i + v < span[u] && at0[u] + i + v >= lo[u] && E::equal(e[u][v / S][v % S], h[u], k[u], bkeys);
#pragma unroll
        for (int u = 0; u < GT_U; ++u)
#pragma unroll
            for (uint32_t v = 0; v < GT_WALK_U; ++v) {
                const uint32_t bal = __ballot_sync(0xffffffffu, eq[u][v]), n_eq = __popc(bal);
                if (!write) {
                    staged += n_eq;
                } else if (staged + n_eq <= GT_STAGE) {
                    if (eq[u][v]) stage[staged + __popc(bal & lt)] = make_uint2(E::row(e[u][v / S][v % S]), row0 + u);
                    staged += n_eq;
                } else if (eq[u][v]) {
                    hit[u] |= 1u << (i + v);
                }
            }
    }
    // the longer ones, counted by the whole warp
    uint32_t more = 0;
#pragma unroll
    for (int u = 0; u < GT_U; ++u) {
        more += __popc(hit[u]);
        uint32_t found = 0;  // this lane's row of them
        for (uint32_t todo = __ballot_sync(0xffffffffu, hi[u] - at0[u] > GT_LONG && hi[u] != lo[u]); todo; todo &= todo - 1u) {
            const int owner = __ffs(todo) - 1;
            const uint32_t a = __shfl_sync(0xffffffffu, lo[u], owner), z = __shfl_sync(0xffffffffu, hi[u], owner);
            const uint32_t hh = __shfl_sync(0xffffffffu, h[u], owner);
            const K kk = __shfl_sync(0xffffffffu, k[u], owner);
            uint32_t n_eq = 0;
            for (uint32_t i = a + lane; i < z; i += 64) {
                const typename E::T e0 = gt_load(entries + i);
                const typename E::T e1 = i + 32 < z ? gt_load(entries + i + 32) : E::none(hh, kk);
                n_eq += (E::equal(e0, hh, kk, bkeys) ? 1u : 0u) + (E::equal(e1, hh, kk, bkeys) ? 1u : 0u);
            }
            n_eq = __reduce_add_sync(0xffffffffu, n_eq);
            if (lane == owner) found = n_eq;
        }
        if (found == 0) hi[u] = lo[u];  // (no second walk)
        more += found;
    }
    more = __reduce_add_sync(0xffffffffu, more);
    // lane 31 speaks for the warp: its position is the warp's base
    const unsigned long long at = gt_reserve(lane == 31 ? staged + more : 0u, s_warp, o.count);
    unsigned long long pos = __shfl_sync(0xffffffffu, at, 31);
    if (!write) return;
    auto leave = [&]() {
        __syncwarp();
        for (uint32_t i = lane; i < staged; i += 32) {
            const uint2 x = stage[i];
            gt_store_pair(o, pos + i, static_cast<int32_t>(x.x), x.y);
        }
        pos += staged;
        staged = 0;
        __syncwarp();
    };
    leave();
    if (more == 0) return;
    auto put = [&](bool has, uint32_t b, uint32_t q) {
        const uint32_t bal = __ballot_sync(0xffffffffu, has);
        if (bal == 0xffffffffu) {  // a run by itself (2^20 x 2^22 rows, 64 a key: 849 -> 683 us)
            gt_store_pair(o, pos + lane, static_cast<int32_t>(b), q);
            pos += 32;
            return;
        }
        if (has) stage[staged + __popc(bal & lt)] = make_uint2(b, q);
        staged += __popc(bal);
        if (staged > GT_STAGE - 32) leave();
    };
    while (__any_sync(0xffffffffu, (hit[0] | hit[1]) != 0u)) {
        const int u = hit[0] ? 0 : 1;
        const uint32_t m = u == 0 ? hit[0] : hit[1];
        uint32_t b = 0;
        if (m) b = E::row(gt_load(entries + (u == 0 ? at0[0] : at0[1]) + __ffs(m) - 1));
        put(m != 0u, b, row0 + u);
        if (u == 0) hit[0] = m & (m - 1u);
        else hit[1] = m & (m - 1u);
    }
#pragma unroll
    for (int u = 0; u < GT_U; ++u) {
        for (uint32_t todo = __ballot_sync(0xffffffffu, hi[u] - at0[u] > GT_LONG && hi[u] != lo[u]); todo; todo &= todo - 1u) {
            const int owner = __ffs(todo) - 1;
            const uint32_t a = __shfl_sync(0xffffffffu, lo[u], owner), z = __shfl_sync(0xffffffffu, hi[u], owner);
            const uint32_t hh = __shfl_sync(0xffffffffu, h[u], owner);
            const uint32_t q = __shfl_sync(0xffffffffu, row0 + u, owner);
            const K kk = __shfl_sync(0xffffffffu, k[u], owner);
            for (uint32_t i0 = a; i0 < z; i0 += 64) {
                const uint32_t i = i0 + lane;
                const typename E::T e0 = i < z ? gt_load(entries + i) : E::none(hh, kk);
                const typename E::T e1 = i + 32 < z ? gt_load(entries + i + 32) : E::none(hh, kk);
                put(E::equal(e0, hh, kk, bkeys), E::row(e0), q);
                if (i0 + 32 < z) put(E::equal(e1, hh, kk, bkeys), E::row(e1), q);
            }
        }
    }
    leave();
}

// The probe rows that gt_probe_multi_kernel left: the rounds of all words, in
// equal shares over the CTAs.  A warp takes four (probe row, slice of its
// range) a round; their entries stay in registers from the comparison to the
// store, so a range is walked once, and the pairs of a round leave in whole
// runs at a position reserved by one atomic.  (Walked by one warp a row,
// 64 probe rows of a key with 2^20 build rows took 1.27 s.)
template <typename K, bool WIDE>
__global__ void __launch_bounds__(GT_THREADS) gt_probe_long_kernel(const K* __restrict__ pkeys, uint32_t n,
                                                                   const K* __restrict__ bkeys,
                                                                   const uint2* range, uint32_t nb,
                                                                   const typename GtEntry<K, WIDE>::T* entries, GtLong later,
                                                                   GlobalOut o)
{
    using E = GtEntry<K, WIDE>;
    constexpr uint32_t ROWS = 32 * GT_U;  // probe rows of a word
    static_assert(ROWS == 64, "two rows a lane");
    constexpr int NW = GT_THREADS / 32;
    __shared__ unsigned long long s_warp[2][NW + 2];
    __shared__ K s_key[ROWS];
    __shared__ uint32_t s_hash[ROWS], s_lo[ROWS], s_hi[ROWS], s_first[ROWS];  // s_first: slices of the rows before
    __shared__ uint32_t s_half;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    gt_wait_before();
    const unsigned long long mask = (1ull << later.round_bits) - 1ull, all = *later.cursor;
    const unsigned long long rounds = all & mask;
    const uint32_t words = static_cast<uint32_t>(all >> later.round_bits);
    unsigned long long r = rounds / gridDim.x * blockIdx.x + min(rounds % gridDim.x, static_cast<unsigned long long>(blockIdx.x));
    const unsigned long long end = r + rounds / gridDim.x + (blockIdx.x < rounds % gridDim.x ? 1 : 0);
    if (r == end) return;
    // the word of the first round: the last one that starts at it or before
    uint32_t w = 0;
    for (uint32_t count = words; count > 1u;) {
        const uint32_t half = count / 2u;
        if ((later.list[w + half] & mask) <= r) {
            w += half;
            count -= half;
        } else {
            count = half;
        }
    }
    int buffer = 0;
    while (r < end) {
        const unsigned long long word = later.list[w], word_first = word & mask;
        const unsigned long long word_end = w + 1u < words ? later.list[w + 1u] & mask : rounds;
        const uint32_t row0 = static_cast<uint32_t>(word >> later.round_bits) * ROWS;
        __syncthreads();  // (every warp has left the word before)
        uint32_t mine = 0, incl = 0;
        if (threadIdx.x < ROWS) {
            const uint32_t row = row0 + threadIdx.x;
            K key = 0;
            uint32_t h = 0;
            uint2 x = make_uint2(0u, 0u);
            if (row < n) {
                key = pkeys[row];
                h = hash_key(key);
                x = gt_load(range + gt_bucket(h, nb));
            }
            incl = mine = later.slices(x.y - x.x);
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += y;
            }
            if (threadIdx.x == 31) s_half = incl;
            s_key[threadIdx.x] = key;
            s_hash[threadIdx.x] = h;
            s_lo[threadIdx.x] = x.x;
            s_hi[threadIdx.x] = x.y;
        }
        __syncthreads();
        if (threadIdx.x < ROWS) s_first[threadIdx.x] = incl - mine + (warp > 0 ? s_half : 0u);
        __syncthreads();
        const unsigned long long stop = word_end < end ? word_end : end;
        for (; r < stop; ++r) {
            const uint32_t first = (static_cast<uint32_t>(r - word_first) * NW + warp) * GT_SLICES;
            int row[GT_SLICES];
            uint32_t lo[GT_SLICES], hi[GT_SLICES];
#pragma unroll
            for (int t = 0; t < GT_SLICES; ++t) {
                // the last row whose slices start at the slice or before (rows without slices start where the next does)
                const int j = __popc(__ballot_sync(0xffffffffu, s_first[lane] <= first + t)) +
                              __popc(__ballot_sync(0xffffffffu, s_first[lane + 32] <= first + t)) - 1;
                const uint32_t part = first + t - s_first[j], from = s_lo[j], to = s_hi[j];
                row[t] = j;
                lo[t] = from + part * later.slice;
                // (past the word's last slice: nothing)
                hi[t] = part < later.slices(to - from) ? min(lo[t] + later.slice, to) : 0u;
            }
            for (uint32_t step = 0; step < later.slice; step += GT_SLICE, buffer ^= 1) {
                typename E::T e[GT_SLICES][GT_SLICE_U];
#pragma unroll
                for (int t = 0; t < GT_SLICES; ++t)
#pragma unroll
                    for (int v = 0; v < GT_SLICE_U; ++v) {
                        const uint32_t i = lo[t] + step + v * 32 + lane;
                        e[t][v] = i < hi[t] ? gt_load(entries + i) : E::none(s_hash[row[t]], s_key[row[t]]);
                    }
                uint32_t off[GT_SLICES][GT_SLICE_U], hits = 0, total = 0;
#pragma unroll
                for (int t = 0; t < GT_SLICES; ++t)
#pragma unroll
                    for (int v = 0; v < GT_SLICE_U; ++v) {
                        const bool hit = E::equal(e[t][v], s_hash[row[t]], s_key[row[t]], bkeys);
                        const uint32_t bal = __ballot_sync(0xffffffffu, hit);
                        off[t][v] = total + __popc(bal & lt);
                        total += __popc(bal);
                        hits |= hit ? 1u << (t * GT_SLICE_U + v) : 0u;
                    }
                // lane 31 speaks for the warp: its position is the warp's base
                const unsigned long long at = gt_reserve(lane == 31 ? total : 0u, s_warp[buffer], o.count);
                const unsigned long long base = __shfl_sync(0xffffffffu, at, 31);
                if (o.out_build == nullptr) continue;
#pragma unroll
                for (int t = 0; t < GT_SLICES; ++t)
#pragma unroll
                    for (int v = 0; v < GT_SLICE_U; ++v)
                        if (hits >> (t * GT_SLICE_U + v) & 1u)
                            gt_store_pair(o, base + off[t][v], static_cast<int32_t>(E::row(e[t][v])), row0 + row[t]);
            }
        }
        ++w;
    }
}

}  // namespace pj
