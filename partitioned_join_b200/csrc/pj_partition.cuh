// pj_partition.cuh -- radix histogram, decoupled look-back scan and
// write-combining scatter.
//
// Layout of one partitioned column.  The input is cut into n_items equal
// chunks ("items", one per resident scatter CTA), and the items into groups of
// ipg.  Item i = (g, j) has one counter per partition at (g * P + p) * ipg + j;
// off is the exclusive scan of these counts, each rounded up to W tuples, and
// the item's tuples of partition p form the segment of that index.  So
// partition p is one contiguous range per group,
// [off[(g * P + p) * ipg], off[(g * P + p + 1) * ipg]), every segment starts on
// a W-tuple boundary, and the padding tuples of a segment carry row = -1.
// One group (ipg = n_items) makes partitions contiguous.  Large columns take
// several: a scatter CTA then writes within its group's part of the buffer,
// a few hundred MB that its address translation covers -- spread over all
// 4.3 GB, plain sector stores took 2.5 ms instead of 1.8.
//
// Tuples.  4-byte keys are stored as {murmur(key), row}: MurmurHash3_x86_32
// of a 4-byte key is a bijection of 32-bit values (every step -- odd
// multiplies, rotations, xor/add of constants, the fmix32 xor-shifts -- is
// invertible), so equal hashes mean equal keys and the join never hashes
// again.  8-byte keys are stored as {key_lo, key_hi, murmur(key), row}.
//
// Reference counterparts: histogram_pass_one (partition_kernels.cuh:141-194),
// the ExclusiveSum + copy of partitioned_join.cuh:86-88, partition_pass_one
// (partition_kernels.cuh:197-326).  The reference stages an 8 192-key tile in
// shared memory and flushes each partition's run with 32 threads; here each
// CTA keeps a W-tuple write-combining buffer per partition and writes only
// whole, aligned W-tuple groups (32-byte sectors), so the fan-out of one pass
// reaches 4 096.
//
// With the heavy-key path (pj_heavy.cuh) the probe side's histogram skips
// heavy keys and its scatter writes their output pairs directly.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "pj_device.cuh"
#include "pj_heavy.cuh"
#include "pj_types.cuh"

namespace pj {

// Index of item `item`'s first counter (partition 0) with the items in groups
// of ipg: partition p's is p * ipg further.
__device__ __forceinline__ int64_t seg_base(int item, int ipg, int P)
{
    return static_cast<int64_t>(item / ipg) * P * ipg + item % ipg;
}

template <typename K>
__device__ __forceinline__ uint32_t key_digit(const DigitFn& f, K key)
{
    return digit_of(f, key, f.mode == 1 ? hash_key(key) : 0u);
}

// Elements of a 16-byte vector.
template <typename K> struct Vec16 { static constexpr int N = 16 / sizeof(K); };

template <typename K>
__device__ __forceinline__ void load_vec16(const K* p, K (&out)[Vec16<K>::N])
{
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
    if constexpr (sizeof(K) == 4) {
        out[0] = static_cast<K>(v.x); out[1] = static_cast<K>(v.y);
        out[2] = static_cast<K>(v.z); out[3] = static_cast<K>(v.w);
    } else {
        out[0] = static_cast<K>((static_cast<uint64_t>(v.y) << 32) | v.x);
        out[1] = static_cast<K>((static_cast<uint64_t>(v.w) << 32) | v.z);
    }
}

// Byte offset of the heavy table in the scatter's shared memory: after P
// buffers of capw words, P fill counts and P cursors, rounded up to 16 bytes.
__host__ __device__ constexpr size_t heavy_table_offset(int P, int capw)
{
    return (static_cast<size_t>(P) * capw * 4 + static_cast<size_t>(P) * 8 + 15) & ~static_cast<size_t>(15);
}

// Output of heavy probe keys (heavy-key path).  The probe histogram counts,
// per item, the heavy probe rows that have a build row; item i's pairs then
// go to [sum of the counts of items < i, ...) -- exact positions, no global
// atomics -- and the join's output starts after all of them.
struct HeavyOut {
    const int32_t* heavy_row;          // build row of each heavy key (-1: none)
    unsigned long long* item_count;    // per scatter item: heavy pairs (zeroed by the caller)
    int32_t* out_build;                // nullptr: count only
    int32_t* out_probe;
    int64_t capacity;
};

// ---------------------------------------------------------------------------
// Histogram.  Grid = n_items * hsplit CTAs; CTA c counts the keys of the
// (c % hsplit)-th slice of item c / hsplit's chunk in shared memory and adds
// them into counts_T[p*n_items + item] (zeroed by the caller) and totals[p].
constexpr int HIST_THREADS = 512;
constexpr int HIST_UNROLL = 4;  // 16-byte vectors in flight per thread

template <typename K, bool HASHD, bool HEAVY>
__global__ void __launch_bounds__(HIST_THREADS) hist_keys_kernel(const K* __restrict__ keys, int64_t n,
                                                                 int64_t chunk, int32_t n_items, int32_t hsplit,
                                                                 DigitFn f, int32_t P, int32_t ipg,
                                                                 uint32_t* __restrict__ counts_T,
                                                                 int32_t* __restrict__ totals,
                                                                 typename HeavyArg<HEAVY>::type hs, HeavyOut ho)
{
    constexpr int VN = Vec16<K>::N;
    extern __shared__ __align__(16) uint32_t cnt[];
    const int item = blockIdx.x / hsplit, part = blockIdx.x % hsplit;
    for (int p = threadIdx.x; p < P; p += HIST_THREADS) cnt[p] = 0;
    HeavyTable heavy;
    uint32_t heavy_hits = 0;
    if constexpr (HEAVY) {
        heavy.bind(reinterpret_cast<uint8_t*>(cnt + ((P + 3) & ~3)));
        heavy.build<K>(hs, ho.heavy_row);  // ends with a barrier
    }
    __syncthreads();
    int64_t lo = static_cast<int64_t>(item) * chunk;
    int64_t hi = lo + chunk < n ? lo + chunk : n;
    if (lo > hi) lo = hi;
    // this CTA's slice of the item, 16-element aligned
    const int64_t per = (((hi - lo) + hsplit - 1) / hsplit + 15) & ~int64_t(15);
    int64_t s_lo = lo + part * per;
    int64_t s_hi = s_lo + per < hi ? s_lo + per : hi;
    if (s_lo > s_hi) s_lo = s_hi;
    // digit of key k, or -1 for a heavy probe key (not partitioned)
    auto digit = [&](K k) -> int {
        if constexpr (HEAVY) {
            const HeavyHit e = heavy.find(k);
            if (e.idx >= 0) {
                heavy_hits += e.row >= 0 ? 1u : 0u;
                return -1;
            }
        }
        uint32_t h = 0;
        if constexpr (HASHD) h = hash_key(k);
        return static_cast<int>(HASHD ? ((h >> f.shift) & f.mask)
                                      : (static_cast<uint32_t>(static_cast<uint64_t>(k) >> f.shift) & f.mask));
    };
    auto count = [&](K k) {
        const int d = digit(k);
        if (d >= 0) atomicAdd(&cnt[d], 1u);
    };
    constexpr int STEP = HIST_THREADS * VN * HIST_UNROLL;
    int64_t base = s_lo;
    // the next step's vectors load while this step's keys are counted
    K v[HIST_UNROLL][VN];
    auto load_step = [&](int64_t at) {
#pragma unroll
        for (int u = 0; u < HIST_UNROLL; ++u)
            load_vec16<K>(keys + at + (static_cast<int64_t>(u) * HIST_THREADS + threadIdx.x) * VN, v[u]);
    };
    if (base + STEP <= s_hi) load_step(base);
    for (; base + STEP <= s_hi; base += STEP) {
        K c[HIST_UNROLL][VN];
#pragma unroll
        for (int u = 0; u < HIST_UNROLL; ++u)
#pragma unroll
            for (int e = 0; e < VN; ++e) c[u][e] = v[u][e];
        if (base + 2 * STEP <= s_hi) load_step(base + STEP);
#pragma unroll
        for (int u = 0; u < HIST_UNROLL; ++u)
#pragma unroll
            for (int e = 0; e < VN; ++e) count(c[u][e]);
    }
    for (int64_t i = base + threadIdx.x; i < s_hi; i += HIST_THREADS) count(keys[i]);
    if constexpr (HEAVY) {
        heavy_hits = __reduce_add_sync(0xffffffffu, heavy_hits);
        if ((threadIdx.x & 31) == 0 && heavy_hits) atomicAdd(&ho.item_count[item], static_cast<unsigned long long>(heavy_hits));
    }
    __syncthreads();
    for (int p = threadIdx.x; p < P; p += HIST_THREADS) {
        const uint32_t c = cnt[p];
        if (c) {
            atomicAdd(&counts_T[seg_base(item, ipg, P) + static_cast<int64_t>(p) * ipg], c);
            if (totals != nullptr) atomicAdd(&totals[p], static_cast<int32_t>(c));
        }
    }
}

// Global digit histogram (no per-item split): the stage entry point
// pj_radix_histogram and the exact planner.
template <typename K>
__global__ void __launch_bounds__(512) global_hist_kernel(const K* __restrict__ keys, int64_t n, DigitFn f,
                                                          int32_t P, int32_t* __restrict__ hist)
{
    extern __shared__ __align__(16) uint32_t sh_hist[];
    for (int p = threadIdx.x; p < P; p += blockDim.x) sh_hist[p] = 0;
    __syncthreads();
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
        atomicAdd(&sh_hist[key_digit(f, keys[i])], 1u);
    __syncthreads();
    for (int p = threadIdx.x; p < P; p += blockDim.x)
        if (sh_hist[p]) atomicAdd(&hist[p], static_cast<int32_t>(sh_hist[p]));
}

// ---------------------------------------------------------------------------
// Single-pass exclusive scan with decoupled look-back (Merrill & Garland,
// "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016).
// out[i] = sum_{j<i} r(in[j]), out[m] = total, with r(x) = x rounded up to a
// multiple of round_to (a power of two).  Tiles are claimed through an atomic counter, so a
// tile's predecessors are always already running; the look-back spin is
// bounded all the same.  tile_state and tile_counter must be zero.
constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
constexpr uint64_t TS_AGG = 1ull << 62;
constexpr uint64_t TS_PREFIX = 2ull << 62;
constexpr uint64_t TS_VALUE = (1ull << 62) - 1;

__device__ __forceinline__ void st_release_u64(uint64_t* p, uint64_t v)
{
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ uint64_t ld_acquire_u64(const uint64_t* p)
{
    uint64_t v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// The look-back wait of a scan: how many polls a tile makes before it gives
// up (ST_TIMEOUT), and a tile that never publishes (-1: none).  Joins use
// {-1, SPIN_LIMIT}; pj_diag_scan_timeout withholds a tile to show that a
// wait which never ends returns an error instead of hanging.
struct ScanWait {
    int64_t withhold_tile;
    uint32_t spin_limit;
};

template <typename TIn>
__global__ void __launch_bounds__(SCAN_THREADS) lookback_scan_kernel(const TIn* __restrict__ in, int64_t m,
                                                                     uint32_t round_to, int64_t* __restrict__ out,
                                                                     uint64_t* __restrict__ tile_state,
                                                                     uint32_t* __restrict__ tile_counter,
                                                                     uint32_t* __restrict__ status, ScanWait wait)
{
    __shared__ uint32_t s_tile;
    __shared__ int64_t s_warp[SCAN_THREADS / 32];
    __shared__ int64_t s_excl;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_counter, 1u);
    __syncthreads();
    const int64_t tile = s_tile;
    const int64_t ntiles = (m + SCAN_TILE - 1) / SCAN_TILE;
    const int64_t base = tile * SCAN_TILE + static_cast<int64_t>(threadIdx.x) * SCAN_ITEMS;

    int64_t v[SCAN_ITEMS];
    int64_t sum = 0;
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) {
        const int64_t idx = base + j;
        int64_t x = idx < m ? static_cast<int64_t>(in[idx]) : 0;
        x = (x + round_to - 1) & ~static_cast<int64_t>(round_to - 1);
        v[j] = x;
        sum += x;
    }
    int64_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int64_t w = lane < SCAN_THREADS / 32 ? s_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < SCAN_THREADS / 32) s_warp[lane] = w;  // inclusive warp totals
    }
    __syncthreads();
    const int64_t block_total = s_warp[SCAN_THREADS / 32 - 1];
    const int64_t thread_excl = incl - sum + (warp > 0 ? s_warp[warp - 1] : 0);

    // Warp 0 looks back 32 tiles at a time: lane l at tile `at - l`.  The
    // aggregates up to the nearest published prefix are this tile's offset.
    // (One thread stepping back tile by tile took most of the kernel: 2^18
    // counters 12 us, 606 K counters 20 us.)
    if (warp == 0) {
        int64_t excl = 0;
        if (tile == wait.withhold_tile) {
            // publishes nothing: its successors' waits run out
        } else if (tile == 0) {
            if (lane == 0) st_release_u64(&tile_state[0], TS_PREFIX | static_cast<uint64_t>(block_total));
        } else {
            if (lane == 0) st_release_u64(&tile_state[tile], TS_AGG | static_cast<uint64_t>(block_total));
            uint32_t spins = 0;
            for (int64_t at = tile - 1;;) {
                const uint64_t s = at >= lane ? ld_acquire_u64(&tile_state[at - lane]) : TS_PREFIX;
                const uint32_t published = __ballot_sync(0xffffffffu, (s & ~TS_VALUE) != 0);
                const uint32_t prefixes = __ballot_sync(0xffffffffu, (s & ~TS_VALUE) == TS_PREFIX);
                const uint32_t upto = prefixes ? (prefixes & -prefixes) * 2u - 1u : 0xffffffffu;  // lanes that count
                if ((published & upto) != upto) {
                    if (++spins > wait.spin_limit) {
                        if (lane == 0) raise_status(status, ST_TIMEOUT);
                        break;
                    }
                    __nanosleep(32);
                    continue;
                }
                int64_t v32 = (upto >> lane) & 1u ? static_cast<int64_t>(s & TS_VALUE) : 0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v32 += __shfl_xor_sync(0xffffffffu, v32, o);
                excl += v32;
                if (prefixes) break;
                at -= 32;
            }
            if (lane == 0) st_release_u64(&tile_state[tile], TS_PREFIX | static_cast<uint64_t>(excl + block_total));
        }
        if (lane == 0) s_excl = excl;
    }
    __syncthreads();
    int64_t run = s_excl + thread_excl;
#pragma unroll
    for (int j = 0; j < SCAN_ITEMS; ++j) {
        const int64_t idx = base + j;
        if (idx < m) out[idx] = run;
        run += v[j];
    }
    if (tile == (ntiles > 0 ? ntiles - 1 : 0) && threadIdx.x == 0) out[m] = s_excl + block_total;
}

// ---------------------------------------------------------------------------
// Write-combining scatter.
//
// Each round every thread holds V tuples.  Phase A: a shared atomicAdd on
// the partition's fill counter gives each tuple its position s in the
// partition's stream; s < W goes into the W-slot buffer.  Phase B: the tuple
// that took position W-1 flushes the full buffer as one aligned group;
// tuples with W <= s < Q (Q = fill rounded down to W: groups completed
// entirely inside this round) are stored straight to global memory.
// Phase C: the remaining tuples (s >= Q) refill the emptied buffer and the
// flusher moves the partition cursor by Q.  Every tuple is placed in the
// round it is read, whatever the skew.
template <typename K, int W>
struct WcTraits {
    static constexpr int TW = TupleTraits<K>::WORDS;
    static constexpr int BW = W * TW;  // words per buffer
    static_assert((BW * 4) % 16 == 0, "a buffer must be whole 16-byte vectors");
};

template <typename K>
__device__ __forceinline__ void tuple_words(uint32_t (&w)[TupleTraits<K>::WORDS], K key, int32_t row);

template <>
__device__ __forceinline__ void tuple_words<int32_t>(uint32_t (&w)[2], int32_t key, int32_t row)
{
    w[0] = hash_key(key);  // stored hash: the join compares and places by it
    w[1] = static_cast<uint32_t>(row);
}

template <>
__device__ __forceinline__ void tuple_words<int64_t>(uint32_t (&w)[4], int64_t key, int32_t row)
{
    const uint64_t u = static_cast<uint64_t>(key);
    w[0] = static_cast<uint32_t>(u);
    w[1] = static_cast<uint32_t>(u >> 32);
    w[2] = hash_key(key);  // stored hash: digits, buckets and fingerprints come from it
    w[3] = static_cast<uint32_t>(row);
}

template <int TW>
__device__ __forceinline__ void store_words(uint32_t* dst, const uint32_t (&w)[TW])
{
    if constexpr (TW == 2) {
        *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
    } else if constexpr (TW == 4) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
#pragma unroll
        for (int i = 0; i < TW; ++i) dst[i] = w[i];
    }
}

// One 32-byte store per sector: sm_100's 256-bit st.global makes every
// flushed sector a single L2 write request (two 16-byte stores of one
// sector are two requests, which bounds the scatter at the L2 request rate).
__device__ __forceinline__ void st_global_v8(uint32_t* g, const uint4& a, const uint4& b)
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(g), "r"(a.x), "r"(a.y), "r"(a.z),
                 "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}

// The same with an L2 policy.
__device__ __forceinline__ void st_global_v8_keep(uint32_t* g, const uint4& a, const uint4& b, uint64_t pol)
{
    asm volatile("st.global.L2::cache_hint.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8}, %9;" ::"l"(g), "r"(a.x),
                 "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w), "l"(pol)
                 : "memory");
}

template <typename K, int W>
__device__ __forceinline__ void wc_flush(const uint32_t* sbuf, uint32_t* gdst)
{
    constexpr int BW = WcTraits<K, W>::BW;
    if constexpr ((BW * 4) % 32 == 0) {
#pragma unroll
        for (int q = 0; q < BW / 8; ++q)
            st_global_v8(gdst + 8 * q, reinterpret_cast<const uint4*>(sbuf)[2 * q],
                         reinterpret_cast<const uint4*>(sbuf)[2 * q + 1]);
    } else {
#pragma unroll
        for (int q = 0; q < BW / 4; ++q)
            reinterpret_cast<uint4*>(gdst)[q] = reinterpret_cast<const uint4*>(sbuf)[q];
    }
}



// Per-partition fill counts and output cursors of the write-combining
// scatter: two 4-byte arrays after the buffers.
struct WcState {
    int* fill;
    int* cur;
    __device__ static WcState at(uint32_t* after_buffers, int P)
    {
        int* f = reinterpret_cast<int*>(after_buffers);
        return WcState{f, f + P};
    }
    __device__ void init(int p, int cursor) const
    {
        fill[p] = 0;
        cur[p] = cursor;
    }
};

// One round of the write-combining scatter: every thread places its V
// tuples (words w, partition dv, ok = real) through the per-partition
// buffers of cap tuples (a multiple of the group size W).  Phase A: a shared
// atomic gives each tuple its slot in its partition's stream; slots below
// cap go to the buffer.  Phase B: the tuple in the last slot of each
// complete group inside the buffer flushes that group (one 32-byte store per
// sector); tuples of complete groups past the buffer go straight out.
// Phase C: the partial group after the last complete one moves to the
// buffer's front and the holder of the last complete slot advances the
// partition's cursor.  At every round's start a buffer holds fewer than W
// tuples.  Every thread of the CTA calls it (three barriers).
template <typename K, int W, int V>
__device__ __forceinline__ void wc_place(const uint32_t (&w)[V][TupleTraits<K>::WORDS], const uint32_t (&dv)[V],
                                         const bool (&ok)[V], uint32_t* buf, int cap, WcState fc,
                                         uint32_t* __restrict__ out, uint32_t out_cap, uint32_t* __restrict__ status)
{
    constexpr int TW = WcTraits<K, W>::TW;
    const int capw = cap * TW;
    int s[V], F[V], Q[V];
    // phase A
#pragma unroll
    for (int v = 0; v < V; ++v) {
        s[v] = ok[v] ? atomicAdd(&fc.fill[dv[v]], 1) : -1;
        if (ok[v] && s[v] < cap) store_words<TW>(buf + dv[v] * capw + s[v] * TW, w[v]);
    }
    __syncthreads();
    // phase B: only the tuples at or past the first group's last slot act
#pragma unroll
    for (int v = 0; v < V; ++v) {
        if (s[v] >= W - 1) {
            F[v] = fc.fill[dv[v]];
            Q[v] = F[v] & ~(W - 1);
            const uint32_t cur_p = static_cast<uint32_t>(fc.cur[dv[v]]);
            if (s[v] < cap) {
                if ((s[v] & (W - 1)) == W - 1) {
                    const int g0 = s[v] - (W - 1);  // first slot of the complete group
                    const uint32_t pos = cur_p + static_cast<uint32_t>(g0);
                    if (pos + static_cast<uint32_t>(W) <= out_cap)
                        wc_flush<K, W>(buf + dv[v] * capw + g0 * TW, out + static_cast<size_t>(pos) * TW);
                    else
                        raise_status(status, ST_INTERNAL);
                }
            } else if (s[v] < Q[v]) {
                const uint32_t pos = cur_p + static_cast<uint32_t>(s[v]);
                if (pos < out_cap)
                    store_words<TW>(out + static_cast<size_t>(pos) * TW, w[v]);
                else
                    raise_status(status, ST_INTERNAL);
            }
        }
    }
    __syncthreads();
    // phase C: a slot past the first group exists only where a group
    // completed (Q >= W), and then every slot from Q on was taken this round
#pragma unroll
    for (int v = 0; v < V; ++v) {
        if (s[v] >= W - 1 && Q[v] >= W) {
            if (s[v] >= Q[v]) store_words<TW>(buf + dv[v] * capw + (s[v] - Q[v]) * TW, w[v]);
            if (s[v] == Q[v] - 1) {
                fc.fill[dv[v]] = F[v] - Q[v];
                fc.cur[dv[v]] += Q[v];
            }
        }
    }
    __syncthreads();
}

// End of an item: pad every partial buffer to W tuples, write it, and check
// that each partition's cursor reached the end of its segment
// [offsets[p * n_items + item], offsets[p * n_items + item + 1]).
template <typename K, int W>
__device__ __forceinline__ void wc_finish(int P, uint32_t* buf, int cap, WcState fc, uint32_t* __restrict__ out,
                                          uint32_t out_cap,
                                          const int64_t* __restrict__ offsets, int32_t n_items, int32_t item,
                                          uint32_t* __restrict__ status)
{
    constexpr int TW = WcTraits<K, W>::TW;
    // final flush: pad every partial group (fewer than W tuples, at the
    // buffer's front) to W tuples and write it
    for (int p = threadIdx.x; p < P; p += blockDim.x) {
        const int fl = fc.fill[p];
        uint32_t cur_p = static_cast<uint32_t>(fc.cur[p]);
        if (fl > 0) {
            uint32_t* bq = buf + static_cast<size_t>(p) * cap * TW;
            for (int q = fl; q < W; ++q) {
                uint32_t pad[TW];
#pragma unroll
                for (int i = 0; i < TW; ++i) pad[i] = 0u;
                pad[TW - 1] = static_cast<uint32_t>(PAD_ROW);
                store_words<TW>(bq + q * TW, pad);
            }
            if (cur_p + static_cast<uint32_t>(W) <= out_cap)
                wc_flush<K, W>(bq, out + static_cast<size_t>(cur_p) * TW);
            else
                raise_status(status, ST_INTERNAL);
            cur_p += W;
        }
        if (cur_p != static_cast<uint32_t>(offsets[static_cast<int64_t>(p) * n_items + item + 1]))
            raise_status(status, ST_INTERNAL);
    }
}

// ---------------------------------------------------------------------------
// Write-combining placement without block barriers.
//
// Per partition the CTA keeps one unit of F tuples (a power of two, about
// 128 KB over all partitions) in shared memory, a fill word {parity, count},
// a front cursor and a back cursor into the partition's segment.  A tuple
// takes count c by a shared atomic on the fill word:
//   c < F      it goes to slot c, its row's top bit set to the unit's parity
//              (rows are below 2^31);
//   c >= F     the unit is full and not yet written: the tuple goes straight
//              to the back of the segment (back cursor, one atomic), so no
//              thread ever waits for a unit and the front stays aligned;
//   c == F - 1 the tuple's warp writes the unit: it notes {partition, parity}
//              in the warp's list, and after its round the warp writes the
//              listed units together, one 32-byte sector a lane.
// A lane that writes a sector re-reads it until every row shows the unit's
// parity: the other tuples of the unit took their slots before this one,
// and nothing stands between a taken slot and its store, so the wait is a few
// shared-memory latencies (bounded all the same).  Taking the sector into
// registers frees the unit: the fill word moves to the other parity and
// count 0 before the sector leaves.
//
// What makes this race-free: a tuple is stored and read by one scalar memory
// operation of its size (64 or 128 bits; a vector access would be several in
// no stated order), so parity and words are seen together; the fill word is
// only ever touched by atomics (a plain store beside atomicAdd could be lost);
// and the unit changes hands by them -- the release exchange that frees it,
// after a __syncwarp behind the last lane's read, and the acquire add that
// takes a slot -- so no read meets the next unit's tuple and no later read
// an older one's of the same parity.  The release waits for the warp's earlier
// sectors: 2^27 int32 keys over 4096 partitions 0.63 ms, 0.61 without it (a
// fence a round in its place 0.65; 2^28 int64 keys 2.17, 2.15 and 2.46 ms).
// The acquire and the scalar accesses cost nothing measurable.
//
// The block-wide form (three barriers per round of one vector a thread)
// waited on shared-memory latency and barriers with half the issue slots
// idle.  The count of a unit that stays full grows with every tuple that meets
// it, so a block barrier every WCU_EPOCH tuples, at which no unit is full,
// keeps it within its bits (a tuple is counted twice at most: as it comes and
// from the late list).
constexpr int WCU_LATE = 64;  // tuples a warp keeps to place later
constexpr uint32_t WCU_COUNT = (1u << 24) - 1u;  // count bits of a fill word; bit 24: parity
constexpr uint32_t WCU_EPOCH = 1u << 22;         // tuples of a CTA between barriers; a multiple of a round's

template <typename K>
struct WcUnits {
    static constexpr int TW = TupleTraits<K>::WORDS;
    static constexpr int CH = 8 / TW;  // tuples of a sector
    static constexpr int LOG_CH = CH == 4 ? 2 : 1;
    static constexpr int MAX_LOGF = LOG_CH + 5;  // a unit's sectors are written by one pass of a warp
    uint32_t* buf;
    uint32_t* fill;
    uint32_t* cur;
    uint32_t* back;
    uint16_t* list;  // this warp's: one entry per tuple of a round
    uint32_t* late;  // this warp's tuples that met a full unit (WCU_LATE)
    uint16_t* late_d;  // and their partitions
    int logF;
    uint64_t keep, done;  // L2 policies of sectors that leave their line open / complete it (0: none)

    // shared memory of P partitions, threads * v tuples a round
    __host__ __device__ static size_t bytes(int P, int logF, int threads, int v)
    {
        return (static_cast<size_t>(P) << logF) * TW * 4 + static_cast<size_t>(threads / 32) * WCU_LATE * (TW * 4 + 2) +
               static_cast<size_t>(P) * 12 + static_cast<size_t>(threads) * v * 2;
    }
    __device__ void bind(uint8_t* smem, int P, int lf, int v)
    {
        const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
        logF = lf;
        buf = reinterpret_cast<uint32_t*>(smem);
        // Many partitions: a line waits for its other sectors while the CTAs
        // fill P x 148 others, and is written to HBM in parts if it is evicted
        // meanwhile.  So its sectors are marked evict-last, the one that
        // completes it evict-first: 4096 partitions of 2^27 int32 keys 0.81 ->
        // 0.60 ms, of 2^28 int64 keys 2.94 -> 2.39 ms, 2048 of 2^26 int64 keys
        // 0.49 -> 0.43 ms (without the demotion 0.605, 2.45, 0.43).  At 2048
        // partitions of int32 keys, whose scatter waits on the SMs, the
        // policy operands cost 4 %.  (Before units were freed by a release exchange.)
        keep = done = 0;
        if (P >= (CH == 4 ? 4096 : 2048)) {
            asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(keep));
            asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(done));
        }
        uint32_t* after = buf + (static_cast<size_t>(P) << lf) * TW;
        late = after + warp * WCU_LATE * TW;
        fill = after + warps * WCU_LATE * TW;
        cur = fill + P;
        back = cur + P;
        uint16_t* half = reinterpret_cast<uint16_t*>(back + P);
        late_d = half + warp * WCU_LATE;
        list = half + warps * WCU_LATE + warp * 32 * v;
    }
};

// A tuple in shared memory, by one scalar store and one scalar load.
template <int TW>
__device__ __forceinline__ void sts_tuple(uint32_t* p, const uint32_t (&w)[TW], uint32_t row)
{
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
    if constexpr (TW == 2)
        asm volatile("{ .reg .b64 t; mov.b64 t, {%1, %2}; st.relaxed.cta.shared.b64 [%0], t; }" ::"r"(a), "r"(w[0]),
                     "r"(row)
                     : "memory");
    else
        asm volatile("{ .reg .b64 l, h; .reg .b128 t; mov.b64 l, {%1, %2}; mov.b64 h, {%3, %4}; mov.b128 t, {l, h}; "
                     "st.relaxed.cta.shared.b128 [%0], t; }" ::"r"(a),
                     "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(row)
                     : "memory");
}

// The 16 bytes at p: two 8-byte tuples, or one of 16 bytes.
template <int TW>
__device__ __forceinline__ uint4 lds_tuples(const uint32_t* p)
{
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p));
    uint4 v;
    if constexpr (TW == 2)
        asm volatile("{ .reg .b64 l, h; ld.relaxed.cta.shared.v2.b64 {l, h}, [%4]; mov.b64 {%0, %1}, l; "
                     "mov.b64 {%2, %3}, h; }"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "r"(a)
                     : "memory");
    else
        asm volatile("{ .reg .b64 l, h; .reg .b128 t; ld.relaxed.cta.shared.b128 t, [%4]; mov.b128 {l, h}, t; "
                     "mov.b64 {%0, %1}, l; mov.b64 {%2, %3}, h; }"
                     : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "r"(a)
                     : "memory");
    return v;
}

// A slot of a unit: the fill word before this tuple.
__device__ __forceinline__ uint32_t unit_take(uint32_t* fill)
{
    uint32_t old;
    asm volatile("atom.acquire.cta.shared.add.u32 %0, [%1], 1;"
                 : "=r"(old)
                 : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(fill)))
                 : "memory");
    return old;
}

// The unit is free again, with this fill word.
__device__ __forceinline__ void unit_free(uint32_t* fill, uint32_t word)
{
    asm volatile("{ .reg .b32 t; atom.release.cta.shared.exch.b32 t, [%0], %1; }" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(fill))),
                 "r"(word)
                 : "memory");
}

// Start of an item: empty units of parity 1 over slots of parity 0, cursors
// at the ends of the item's segments.  off(p) / off_end(p): the segment.
template <typename K, typename Off, typename OffEnd>
__device__ __forceinline__ void wcu_begin(const WcUnits<K>& u, int P, Off off, OffEnd off_end)
{
    const int words4 = static_cast<int>((static_cast<size_t>(P) << u.logF) * WcUnits<K>::TW / 4);
    for (int i = threadIdx.x; i < words4; i += blockDim.x) reinterpret_cast<uint4*>(u.buf)[i] = make_uint4(0u, 0u, 0u, 0u);
    for (int p = threadIdx.x; p < P; p += blockDim.x) {
        u.fill[p] = 1u << 24;
        u.cur[p] = static_cast<uint32_t>(off(p));
        u.back[p] = static_cast<uint32_t>(off_end(p));
    }
    __syncthreads();
}

// Places a warp's tuples: w[v] = words, dv[v] = partition, ok[v] = real.
// KEEP: tuples that meet a full unit go to the warp's late list (n_late of
// them so far) while it has room.
template <typename K, int V, bool KEEP>
__device__ __forceinline__ void wcu_put(const WcUnits<K>& u, uint32_t& n_late,
                                        const uint32_t (&w)[V][TupleTraits<K>::WORDS],
                                        const uint32_t (&dv)[V], const bool (&ok)[V], uint32_t* __restrict__ out,
                                        uint32_t out_cap, uint32_t* __restrict__ status)
{
    using U = WcUnits<K>;
    constexpr int TW = U::TW;
    const uint32_t F = 1u << u.logF;
    const int lane = threadIdx.x & 31;
    uint32_t old[V];
#pragma unroll
    for (int v = 0; v < V; ++v) old[v] = ok[v] ? unit_take(&u.fill[dv[v]]) : WCU_COUNT;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const uint32_t c = old[v] & WCU_COUNT;
        if (c < F)
            sts_tuple<TW>(u.buf + (static_cast<size_t>(dv[v]) << u.logF) * TW + c * TW, w[v],
                          w[v][TW - 1] | ((old[v] << 7) & 0x80000000u));
    }
    uint32_t n = 0;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const bool last = (old[v] & WCU_COUNT) == F - 1u;
        const uint32_t bal = __ballot_sync(0xffffffffu, last);
        if (last)
            u.list[n + __popc(bal & ((1u << lane) - 1u))] = static_cast<uint16_t>(dv[v] | ((old[v] >> 9) & 0x8000u));
        n += __popc(bal);
    }
    __syncwarp();
    const int log_c = u.logF - U::LOG_CH;  // sectors of a unit
    const uint32_t total = n << log_c;
    for (uint32_t i0 = 0; i0 < total; i0 += 32) {
        const uint32_t i = i0 + lane;
        const bool act = i < total;
        const uint32_t e = act ? u.list[i >> log_c] : 0u;
        const uint32_t p = e & 0x7fffu, c = i & ((1u << log_c) - 1u);
        const uint32_t parity = (e >> 15) << 31;
        const uint32_t* src = u.buf + (static_cast<size_t>(p) << u.logF) * TW + c * 8;
        uint4 a, b;
        uint32_t spins = 0;
        for (;;) {
            a = lds_tuples<TW>(src);
            b = lds_tuples<TW>(src + 4);
            uint32_t differ;
            if constexpr (TW == 2)
                differ = (a.y ^ parity) | (a.w ^ parity) | (b.y ^ parity) | (b.w ^ parity);
            else
                differ = (a.w ^ parity) | (b.w ^ parity);
            if (__all_sync(0xffffffffu, !act || static_cast<int32_t>(differ) >= 0)) break;
            if (++spins > SPIN_LIMIT) {
                if (lane == 0) raise_status(status, ST_TIMEOUT);
                break;
            }
        }
        __syncwarp();  // every lane has its sector
        uint32_t pos = 0;
        if (act && c == 0) {  // free the unit, then claim its place (units may leave in any order)
            unit_free(u.fill + p, (~e & 0x8000u) << 9);
            pos = atomicAdd(&u.cur[p], F);
        }
        pos = __shfl_sync(0xffffffffu, pos, static_cast<int>(lane - c)) + c * U::CH;
        if (act) {
            if constexpr (TW == 2) {
                a.y &= 0x7fffffffu;
                a.w &= 0x7fffffffu;
                b.y &= 0x7fffffffu;
            } else {
                a.w &= 0x7fffffffu;
            }
            b.w &= 0x7fffffffu;
            uint32_t* g = out + static_cast<size_t>(pos) * TW;
            if (pos + U::CH > out_cap) {
                raise_status(status, ST_INTERNAL);
            } else if ((static_cast<uint32_t>(reinterpret_cast<uintptr_t>(g)) & 31u) == 0) {
                if (u.keep) st_global_v8_keep(g, a, b, ((pos + U::CH) & (4 * U::CH - 1)) != 0 ? u.keep : u.done);
                else st_global_v8(g, a, b);
            } else if constexpr (TW == 2) {  // half-sector groups (W = 2), or a caller's buffer on 16 bytes
                reinterpret_cast<uint2*>(g)[0] = make_uint2(a.x, a.y);
                reinterpret_cast<uint2*>(g)[1] = make_uint2(a.z, a.w);
                reinterpret_cast<uint2*>(g)[2] = make_uint2(b.x, b.y);
                reinterpret_cast<uint2*>(g)[3] = make_uint2(b.z, b.w);
            } else {
                reinterpret_cast<uint4*>(g)[0] = a;
                reinterpret_cast<uint4*>(g)[1] = b;
            }
        }
    }
    // last, so that a store held up by memory holds up no slot or unit
#pragma unroll
    for (int v = 0; v < V; ++v) {
        bool direct = ok[v] && (old[v] & WCU_COUNT) >= F;
        if constexpr (KEEP) {
            // 8-byte keys: not those that the unit's next filling cannot hold
            // either (2^26 keys over 2048 partitions, Zipf 1.5: 667 -> 520 us; 4-byte units are larger, and uniform keys paid 2 %)
            const bool soon = direct && (TW == 2 || (old[v] & WCU_COUNT) < 2u * F);
            const uint32_t bal = __ballot_sync(0xffffffffu, soon);
            const uint32_t at = n_late + __popc(bal & ((1u << lane) - 1u));
            if (soon && at < WCU_LATE) {
                sts_tuple<TW>(u.late + at * TW, w[v], w[v][TW - 1]);
                u.late_d[at] = static_cast<uint16_t>(dv[v]);
                direct = false;
            }
            n_late = min(n_late + __popc(bal), static_cast<uint32_t>(WCU_LATE));
        }
        if (direct) {
            const uint32_t pos = atomicSub(&u.back[dv[v]], 1u) - 1u;
            if (pos < out_cap)
                store_words<TW>(out + static_cast<size_t>(pos) * TW, w[v]);
            else
                raise_status(status, ST_INTERNAL);
        }
    }
    __syncwarp();
}

// Places up to 32 of the warp's late tuples.
template <typename K>
__device__ __forceinline__ void wcu_late(const WcUnits<K>& u, uint32_t& n_late, uint32_t* __restrict__ out,
                                         uint32_t out_cap, uint32_t* __restrict__ status)
{
    constexpr int TW = WcUnits<K>::TW;
    const uint32_t first = n_late > 32u ? n_late - 32u : 0u;
    const uint32_t at = first + (threadIdx.x & 31);
    uint32_t w[1][TW], dv[1] = {0u};
    const bool ok[1] = {at < n_late};
#pragma unroll
    for (int i = 0; i < TW; ++i) w[0][i] = ok[0] ? u.late[at * TW + i] : 0u;
    if (ok[0]) dv[0] = u.late_d[at];
    __syncwarp();
    n_late = first;
    wcu_put<K, 1, false>(u, n_late, w, dv, ok, out, out_cap, status);
}

// One round of a warp: its tuples, then late ones once 32 have gathered.
template <typename K, int V>
__device__ __forceinline__ void wcu_place(const WcUnits<K>& u, uint32_t& n_late,
                                          const uint32_t (&w)[V][TupleTraits<K>::WORDS], const uint32_t (&dv)[V],
                                          const bool (&ok)[V], uint32_t* __restrict__ out, uint32_t out_cap,
                                          uint32_t* __restrict__ status)
{
    wcu_put<K, V, true>(u, n_late, w, dv, ok, out, out_cap, status);
    if (n_late >= 32u) wcu_late<K>(u, n_late, out, out_cap, status);
}

// A round of which few tuples are to be placed (most are heavy keys): they
// join the late list, and 32 at a time are placed together.  Placing them
// where they are costs a whole round's instructions for, at Zipf 1.5, every
// seventh lane (2^26 int64 probe rows, 105 heavy keys: 551 -> 453 us).
template <typename K, int V>
__device__ __forceinline__ void wcu_place_few(const WcUnits<K>& u, uint32_t& n_late,
                                              const uint32_t (&w)[V][TupleTraits<K>::WORDS], const uint32_t (&dv)[V],
                                              const bool (&ok)[V], uint32_t* __restrict__ out, uint32_t out_cap,
                                              uint32_t* __restrict__ status)
{
    constexpr int TW = WcUnits<K>::TW;
    uint32_t bal[V], total = 0;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        bal[v] = __ballot_sync(0xffffffffu, ok[v]);
        total += __popc(bal[v]);
    }
    if (total > 20u * V) {
        wcu_place<K, V>(u, n_late, w, dv, ok, out, out_cap, status);
        return;
    }
    const uint32_t lt = (1u << (threadIdx.x & 31)) - 1u;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        if (n_late + __popc(bal[v]) > WCU_LATE) wcu_late<K>(u, n_late, out, out_cap, status);
        const uint32_t at = n_late + __popc(bal[v] & lt);
        if (ok[v]) {
            sts_tuple<TW>(u.late + at * TW, w[v], w[v][TW - 1]);
            u.late_d[at] = static_cast<uint16_t>(dv[v]);
        }
        n_late += __popc(bal[v]);
        __syncwarp();
    }
}

// End of an item: every unit's remaining tuples at its front cursor, padding
// (at most W - 1 tuples) between them and the back cursor.
template <typename K>
__device__ __forceinline__ void wcu_finish(const WcUnits<K>& u, uint32_t& n_late, int P, uint32_t W,
                                           uint32_t* __restrict__ out, uint32_t out_cap,
                                           uint32_t* __restrict__ status)
{
    constexpr int TW = WcUnits<K>::TW;
    while (n_late > 0u) wcu_late<K>(u, n_late, out, out_cap, status);
    __syncthreads();
    const uint32_t F = 1u << u.logF, span = 2u * (F > W ? F : W);  // slots, then padding
    const uint32_t all = static_cast<uint32_t>(P) * span;          // P * span <= 2^17
    for (uint32_t i = threadIdx.x; i < all; i += blockDim.x) {
        const uint32_t p = i / span, s = i & (span - 1u);
        const uint32_t n = u.fill[p] & WCU_COUNT, at = u.cur[p], end = u.back[p];
        if (s == 0 && (n >= F || end - at - n >= W || end > out_cap)) raise_status(status, ST_INTERNAL);
        if (n < F && at + s < end && s < n + W && end <= out_cap) {
            uint32_t t[TW];
#pragma unroll
            for (int j = 0; j < TW; ++j) t[j] = 0u;
            if (s < n) {
#pragma unroll
                for (int j = 0; j < TW; ++j) t[j] = u.buf[(static_cast<size_t>(p) << u.logF) * TW + s * TW + j];
                t[TW - 1] &= 0x7fffffffu;
            } else {
                t[TW - 1] = static_cast<uint32_t>(PAD_ROW);
            }
            store_words<TW>(out + static_cast<size_t>(at + s) * TW, t);
        }
    }
    __syncthreads();
}

// The heavy ones among a thread's V probe keys leave the partitions (ok =
// false), and their pairs go to the output: after the pairs of earlier items
// (first) and of this item so far (*done, in shared memory).  Positions go by
// key index, then lane, so every store instruction writes one run (lane by
// lane, each lane's pairs together, the same scatter took 453 us, not 414).
// Whole warp.
template <typename K, int V>
__device__ __forceinline__ void heavy_take(const HeavyTable& heavy, const K (&key)[V], const uint32_t (&row)[V],
                                           bool (&ok)[V], unsigned long long first, uint32_t* done, const HeavyOut& ho,
                                           uint32_t* __restrict__ status)
{
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    int32_t hb[V];
    uint32_t off[V], total = 0;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        hb[v] = -1;
        if (ok[v]) {
            const HeavyHit e = heavy.find(key[v]);
            if (e.idx >= 0) {
                ok[v] = false;
                hb[v] = e.row;
            }
        }
        __syncwarp();
        const uint32_t bal = __ballot_sync(0xffffffffu, hb[v] >= 0);
        off[v] = total + __popc(bal & lt);
        total += __popc(bal);
    }
    if (total == 0) return;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(done, total);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (!ho.out_build) return;
    const long long pos = static_cast<long long>(first) + base;
    if (pos + total <= ho.capacity) {
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (hb[v] >= 0) {
                __stcs(ho.out_build + pos + off[v], hb[v]);
                __stcs(ho.out_probe + pos + off[v], static_cast<int32_t>(row[v]));
            }
    } else {
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (hb[v] >= 0) {
                if (pos + off[v] < ho.capacity) {
                    ho.out_build[pos + off[v]] = hb[v];
                    ho.out_probe[pos + off[v]] = static_cast<int32_t>(row[v]);
                } else {
                    raise_status(status, ST_CAPACITY);
                }
            }
    }
}

// Scatter of a raw key column (row = key index).  V keys per thread per
// round (whole 16-byte vectors), the next round's vectors loaded while the
// current one is placed; the warps of the CTA run on their own.
template <typename K, int THREADS, int V, bool HASHD, bool HEAVY>
__global__ void __launch_bounds__(THREADS, 1) scatter_keys_kernel(const K* __restrict__ keys, int64_t n,
                                                                  int64_t chunk, int32_t n_items, DigitFn f,
                                                                  int32_t P, int32_t logF, int32_t W, int32_t ipg,
                                                                  const int64_t* __restrict__ offsets,
                                                                  uint32_t* __restrict__ out, uint32_t out_cap,
                                                                  uint32_t* __restrict__ status,
                                                                  typename HeavyArg<HEAVY>::type hs, HeavyOut ho)
{
    constexpr int TW = TupleTraits<K>::WORDS;
    constexpr int VN = Vec16<K>::N;
    constexpr int NV = V / VN;  // vectors per thread per round
    static_assert(V % VN == 0, "V must be whole vectors");
    constexpr int ROUND = THREADS * V;
    static_assert(WCU_EPOCH % ROUND == 0 && 2 * WCU_EPOCH < WCU_COUNT, "a count stays within its bits");
    extern __shared__ __align__(128) uint8_t smem[];
    WcUnits<K> wc;
    wc.bind(smem, P, logF, V);
    uint32_t n_late = 0;
    HeavyTable heavy;
    if constexpr (HEAVY) {
        // after the units and the lists, on a 16-byte boundary (slots are
        // read as 16-byte words)
        heavy.bind(smem + ((WcUnits<K>::bytes(P, logF, THREADS, V) + 15) & ~size_t(15)));
        heavy.build<K>(hs, ho.heavy_row);  // ends with a barrier
    }

    __shared__ unsigned long long s_hbase;  // heavy pairs of the items before this one
    __shared__ uint32_t s_hcur;             // heavy pairs of this item so far
    for (int32_t item = blockIdx.x; item < n_items; item += gridDim.x) {
        if constexpr (HEAVY) {
            if (threadIdx.x < 32) {
                unsigned long long sum = 0;
                for (int j = threadIdx.x; j < item; j += 32) sum += ho.item_count[j];
                for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
                if (threadIdx.x == 0) {
                    s_hbase = sum;
                    s_hcur = 0;
                }
            }
        }
        const int64_t* seg = offsets + seg_base(item, ipg, P);  // partition p's segment: [seg[p * ipg], seg[p * ipg + 1])
        wcu_begin<K>(wc, P, [&](int p) { return seg[static_cast<int64_t>(p) * ipg]; },
                     [&](int p) { return seg[static_cast<int64_t>(p) * ipg + 1]; });
        int64_t lo = static_cast<int64_t>(item) * chunk;
        const int64_t hi = lo + chunk < n ? lo + chunk : n;
        if (lo > hi) lo = hi;
        const K* kp = keys + lo;
        const uint32_t len = static_cast<uint32_t>(hi - lo);
        const uint32_t row0 = static_cast<uint32_t>(lo);

        // element e of vector j of this thread in the round at offset b:
        //   b + (j * THREADS + threadIdx.x) * VN + e
        auto load_round = [&](uint32_t b, K (&dst)[NV][VN]) {
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const uint32_t at = b + (static_cast<uint32_t>(j) * THREADS + threadIdx.x) * VN;
                if (at + VN <= len) {
                    load_vec16<K>(kp + at, dst[j]);
                } else {
#pragma unroll
                    for (int e = 0; e < VN; ++e) dst[j][e] = at + e < len ? kp[at + e] : K(0);
                }
            }
        };
        K nxt[NV][VN];
        if (len > 0) load_round(0, nxt);
        for (uint32_t b = 0; b < len; b += ROUND) {
            K cur[NV][VN];
#pragma unroll
            for (int j = 0; j < NV; ++j)
#pragma unroll
                for (int e = 0; e < VN; ++e) cur[j][e] = nxt[j][e];
            if (b + ROUND < len) load_round(b + ROUND, nxt);
            const bool full = b + ROUND <= len;

            uint32_t w[V][TW];
            uint32_t dv[V];  // the tuple's partition
            bool ok[V];
#pragma unroll
            for (int j = 0; j < NV; ++j)
#pragma unroll
                for (int e = 0; e < VN; ++e) {
                    const int v = j * VN + e;
                    const uint32_t at = b + (static_cast<uint32_t>(j) * THREADS + threadIdx.x) * VN + e;
                    ok[v] = full || at < len;
                    const K k = cur[j][e];
                    tuple_words<K>(w[v], k, static_cast<int32_t>(row0 + at));
                    uint32_t d;
                    if constexpr (HASHD) {
                        const uint32_t h = sizeof(K) == 4 ? w[v][0] : w[v][TW - 2];
                        d = (h >> f.shift) & f.mask;
                    } else {
                        d = static_cast<uint32_t>(static_cast<uint64_t>(k) >> f.shift) & f.mask;
                    }
                    dv[v] = d;
                }
            if constexpr (HEAVY) {
                K key[V];
                uint32_t row[V];
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    key[v] = static_cast<K>(cur[v / VN][v % VN]);
                    row[v] = w[v][TW - 1];
                }
                heavy_take<K, V>(heavy, key, row, ok, s_hbase, &s_hcur, ho, status);
            }
            if constexpr (HEAVY) wcu_place_few<K, V>(wc, n_late, w, dv, ok, out, out_cap, status);
            else wcu_place<K, V>(wc, n_late, w, dv, ok, out, out_cap, status);
            if (((b + ROUND) & (WCU_EPOCH - 1u)) == 0) __syncthreads();
        }
        wcu_finish<K>(wc, n_late, P, static_cast<uint32_t>(W), out, out_cap, status);
    }
}

// The same scatter with wc_place, in rounds between block barriers: for
// fan-outs whose units and cursors do not fit shared memory (8192 partitions of
// half-sector groups), and for 4096 partitions of items with few tuples.  V
// keys per thread per round (whole 16-byte vectors), the next round's vectors
// loaded while the current one is processed.  Per partition the CTA keeps a
// buffer of cap tuples (whole groups of W), a fill count and an output cursor.
template <typename K, int THREADS, int V, int W, bool HASHD, bool HEAVY>
__global__ void __launch_bounds__(THREADS, 1) scatter_rounds_kernel(const K* __restrict__ keys, int64_t n,
                                                                  int64_t chunk, int32_t n_items, DigitFn f,
                                                                  int32_t P, int32_t cap,
                                                                  const int64_t* __restrict__ offsets,
                                                                  uint32_t* __restrict__ out, uint32_t out_cap,
                                                                  uint32_t* __restrict__ status,
                                                                  typename HeavyArg<HEAVY>::type hs, HeavyOut ho)
{
    constexpr int TW = WcTraits<K, W>::TW;
    constexpr int VN = Vec16<K>::N;
    constexpr int NV = V / VN;  // vectors per thread per round
    static_assert(V % VN == 0, "V must be whole vectors");
    constexpr int ROUND = THREADS * V;
    extern __shared__ __align__(128) uint8_t smem[];
    uint32_t* buf = reinterpret_cast<uint32_t*>(smem);
    const WcState fc = WcState::at(buf + static_cast<size_t>(P) * cap * TW, P);
    HeavyTable heavy;
    if constexpr (HEAVY) {
        // after the buffers and counters, on a 16-byte boundary (slots are
        // read as 16-byte words)
        heavy.bind(smem + heavy_table_offset(P, cap * TW));
        heavy.build<K>(hs, ho.heavy_row);  // ends with a barrier
    }

    __shared__ unsigned long long s_hbase;  // heavy pairs of the items before this one
    __shared__ uint32_t s_hcur;             // heavy pairs of this item so far
    for (int32_t item = blockIdx.x; item < n_items; item += gridDim.x) {
        for (int p = threadIdx.x; p < P; p += THREADS)
            fc.init(p, static_cast<int>(offsets[static_cast<int64_t>(p) * n_items + item]));
        if constexpr (HEAVY) {
            if (threadIdx.x < 32) {
                unsigned long long sum = 0;
                for (int j = threadIdx.x; j < item; j += 32) sum += ho.item_count[j];
                for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
                if (threadIdx.x == 0) {
                    s_hbase = sum;
                    s_hcur = 0;
                }
            }
        }
        __syncthreads();
        int64_t lo = static_cast<int64_t>(item) * chunk;
        const int64_t hi = lo + chunk < n ? lo + chunk : n;
        if (lo > hi) lo = hi;
        const K* kp = keys + lo;
        const uint32_t len = static_cast<uint32_t>(hi - lo);
        const uint32_t row0 = static_cast<uint32_t>(lo);

        // element e of vector j of this thread in the round at offset b:
        //   b + (j * THREADS + threadIdx.x) * VN + e
        auto load_round = [&](uint32_t b, K (&dst)[NV][VN]) {
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                const uint32_t at = b + (static_cast<uint32_t>(j) * THREADS + threadIdx.x) * VN;
                if (at + VN <= len) {
                    load_vec16<K>(kp + at, dst[j]);
                } else {
#pragma unroll
                    for (int e = 0; e < VN; ++e) dst[j][e] = at + e < len ? kp[at + e] : K(0);
                }
            }
        };
        K nxt[NV][VN], nxt2[NV][VN];
        if (len > 0) load_round(0, nxt);
        if (ROUND < len) load_round(ROUND, nxt2);
        for (uint32_t b = 0; b < len; b += ROUND) {
            K cur[NV][VN];
#pragma unroll
            for (int j = 0; j < NV; ++j)
#pragma unroll
                for (int e = 0; e < VN; ++e) {
                    cur[j][e] = nxt[j][e];
                    nxt[j][e] = nxt2[j][e];
                }
            if (b + 2 * ROUND < len) load_round(b + 2 * ROUND, nxt2);
            const bool full = b + ROUND <= len;

            uint32_t w[V][TW];
            uint32_t dv[V];  // the tuple's partition
            bool ok[V];
#pragma unroll
            for (int j = 0; j < NV; ++j)
#pragma unroll
                for (int e = 0; e < VN; ++e) {
                    const int v = j * VN + e;
                    const uint32_t at = b + (static_cast<uint32_t>(j) * THREADS + threadIdx.x) * VN + e;
                    ok[v] = full || at < len;
                    const K k = cur[j][e];
                    tuple_words<K>(w[v], k, static_cast<int32_t>(row0 + at));
                    uint32_t d;
                    if constexpr (HASHD) {
                        const uint32_t h = sizeof(K) == 4 ? w[v][0] : w[v][TW - 2];
                        d = (h >> f.shift) & f.mask;
                    } else {
                        d = static_cast<uint32_t>(static_cast<uint64_t>(k) >> f.shift) & f.mask;
                    }
                    dv[v] = d;
                }
            if constexpr (HEAVY) {
                K key[V];
                uint32_t row[V];
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    key[v] = static_cast<K>(cur[v / VN][v % VN]);
                    row[v] = w[v][TW - 1];
                }
                heavy_take<K, V>(heavy, key, row, ok, s_hbase, &s_hcur, ho, status);
            }
            wc_place<K, W, V>(w, dv, ok, buf, cap, fc, out, out_cap, status);
        }
        wc_finish<K, W>(P, buf, cap, fc, out, out_cap, offsets, n_items, item, status);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Second radix pass (two-pass plans): the tuples of each pass-one partition
// are partitioned again by the next hash bits -- the reference's
// histogram_pass_two / partition_pass_two (partition_kernels.cuh:329-563),
// reading pass-one tuples instead of rewriting the input columns.
// Item (p1, c) is the c-th of C slices of pass-one partition p1's tuples
// [in_off[p1 * in_items], in_off[(p1 + 1) * in_items]); its tuples of sub-
// partition p2 go to the segment [off[p2 * n_items + item], ...).  With
// item = p1 * C + c that index is (p2 * P1 + p1) * C + c, so the join sees
// partition q = p2 * P1 + p1 as one range over C segments.
struct Pass2Items {
    const int64_t* in_off;  // pass-one segment offsets
    int32_t in_items;       // pass-one items
    int32_t C;              // slices per pass-one partition
};

__device__ __forceinline__ void pass2_range(const Pass2Items& it, int item, int64_t& lo, int64_t& hi)
{
    const int p1 = item / it.C, c = item % it.C;
    const int64_t start = it.in_off[static_cast<int64_t>(p1) * it.in_items];
    const int64_t end = it.in_off[static_cast<int64_t>(p1 + 1) * it.in_items];
    const int64_t per = (((end - start) + it.C - 1) / it.C + 15) & ~int64_t(15);
    lo = start + c * per;
    hi = lo + per < end ? lo + per : end;
    if (lo > hi) lo = hi;
}

// tuple i's words and whether it is a real (not padding) tuple
template <typename K>
__device__ __forceinline__ bool load_tuple_words(const uint32_t* __restrict__ t, int64_t i,
                                                 uint32_t (&w)[TupleTraits<K>::WORDS])
{
    if constexpr (TupleTraits<K>::WORDS == 2) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(t) + i);
        w[0] = v.x;
        w[1] = v.y;
    } else {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(t) + i);
        w[0] = v.x;
        w[1] = v.y;
        w[2] = v.z;
        w[3] = v.w;
    }
    return static_cast<int32_t>(w[TupleTraits<K>::WORDS - 1]) != PAD_ROW;
}

// the stored hash of a tuple (word 0 for 4-byte keys, word 2 for 8-byte keys)
template <typename K>
__device__ __forceinline__ uint32_t tuple_hash(const uint32_t (&w)[TupleTraits<K>::WORDS])
{
    return TupleTraits<K>::WORDS == 2 ? w[0] : w[TupleTraits<K>::WORDS - 2];
}

// Pass-two histogram: counts_T[p2 * n_items + item] and totals[p2 * P1 + p1]
// (zeroed by the caller).  Grid = n_items * hsplit CTAs.
template <typename K>
__global__ void __launch_bounds__(HIST_THREADS) hist_tuples_kernel(const uint32_t* __restrict__ tuples, Pass2Items it,
                                                                   int32_t n_items, int32_t hsplit, DigitFn f,
                                                                   int32_t P2, int32_t P1,
                                                                   uint32_t* __restrict__ counts_T,
                                                                   int32_t* __restrict__ totals)
{
    constexpr int TW = TupleTraits<K>::WORDS;
    extern __shared__ __align__(16) uint32_t cnt[];
    const int item = blockIdx.x / hsplit, part = blockIdx.x % hsplit;
    for (int p = threadIdx.x; p < P2; p += HIST_THREADS) cnt[p] = 0;
    __syncthreads();
    int64_t lo, hi;
    pass2_range(it, item, lo, hi);
    const int64_t per = (((hi - lo) + hsplit - 1) / hsplit + 15) & ~int64_t(15);
    int64_t s_lo = lo + part * per;
    const int64_t s_hi = s_lo + per < hi ? s_lo + per : hi;
    if (s_lo > s_hi) s_lo = s_hi;
    for (int64_t i = s_lo + threadIdx.x; i < s_hi; i += HIST_THREADS) {
        uint32_t w[TW];
        if (load_tuple_words<K>(tuples, i, w)) atomicAdd(&cnt[(tuple_hash<K>(w) >> f.shift) & f.mask], 1u);
    }
    __syncthreads();
    const int p1 = item / it.C;
    for (int p = threadIdx.x; p < P2; p += HIST_THREADS) {
        const uint32_t c = cnt[p];
        if (c) {
            atomicAdd(&counts_T[static_cast<int64_t>(p) * n_items + item], c);
            atomicAdd(&totals[static_cast<int64_t>(p) * P1 + p1], static_cast<int32_t>(c));
        }
    }
}

// Pass-two scatter: the pass-one tuples of each item, placed by the next
// hash bits through the same write-combining units as the first pass.
// VT tuples per thread per round, the next round's loaded ahead.
template <typename K, int THREADS, int VT>
__global__ void __launch_bounds__(THREADS, 1) scatter_tuples_kernel(const uint32_t* __restrict__ in, Pass2Items it,
                                                                    int32_t n_items, DigitFn f, int32_t P,
                                                                    int32_t logF, int32_t W,
                                                                    const int64_t* __restrict__ offsets,
                                                                    uint32_t* __restrict__ out, uint32_t out_cap,
                                                                    uint32_t* __restrict__ status)
{
    constexpr int TW = TupleTraits<K>::WORDS;
    constexpr int ROUND = THREADS * VT;
    static_assert(WCU_EPOCH % ROUND == 0);
    extern __shared__ __align__(128) uint8_t smem[];
    WcUnits<K> wc;
    wc.bind(smem, P, logF, VT);
    uint32_t n_late = 0;
    for (int32_t item = blockIdx.x; item < n_items; item += gridDim.x) {
        const int64_t* seg = offsets + item;
        wcu_begin<K>(wc, P, [&](int p) { return seg[static_cast<int64_t>(p) * n_items]; },
                     [&](int p) { return seg[static_cast<int64_t>(p) * n_items + 1]; });
        int64_t lo, hi;
        pass2_range(it, item, lo, hi);
        uint32_t nw[VT][TW];
        bool nok[VT];
        auto load_round = [&](int64_t b) {
#pragma unroll
            for (int v = 0; v < VT; ++v) {
                const int64_t i = b + static_cast<int64_t>(v) * THREADS + threadIdx.x;
                nok[v] = i < hi && load_tuple_words<K>(in, i, nw[v]);
            }
        };
        if (lo < hi) load_round(lo);
        for (int64_t b = lo; b < hi; b += ROUND) {
            uint32_t w[VT][TW];
            uint32_t dv[VT];
            bool ok[VT];
#pragma unroll
            for (int v = 0; v < VT; ++v) {
                ok[v] = nok[v];
#pragma unroll
                for (int i = 0; i < TW; ++i) w[v][i] = nw[v][i];
                dv[v] = (tuple_hash<K>(w[v]) >> f.shift) & f.mask;
            }
            if (b + ROUND < hi) load_round(b + ROUND);
            wcu_place<K, VT>(wc, n_late, w, dv, ok, out, out_cap, status);
            if (((b + ROUND - lo) & (WCU_EPOCH - 1u)) == 0) __syncthreads();
        }
        wcu_finish<K>(wc, n_late, P, static_cast<uint32_t>(W), out, out_cap, status);
    }
}

// ---------------------------------------------------------------------------
// Batches of joins: histogram and scatter over the items (SegItem) of many
// join sides in one launch each.

// Histogram of the items (grid = items * hsplit, hsplit CTAs per item).
template <typename K>
__global__ void __launch_bounds__(HIST_THREADS) hist_seg_kernel(const SegItem* __restrict__ items, int32_t hsplit,
                                                                uint32_t* __restrict__ counts,
                                                                int32_t* __restrict__ totals)
{
    extern __shared__ __align__(16) uint32_t cnt[];
    const SegItem it = items[blockIdx.x / hsplit];
    const int part = blockIdx.x % hsplit;
    for (int p = threadIdx.x; p < it.P; p += HIST_THREADS) cnt[p] = 0;
    __syncthreads();
    const K* keys = static_cast<const K*>(it.keys);
    const int64_t per = (((it.hi - it.lo) + hsplit - 1) / hsplit + 15) & ~int64_t(15);
    int64_t s_lo = it.lo + part * per;
    const int64_t s_hi = s_lo + per < it.hi ? s_lo + per : it.hi;
    if (s_lo > s_hi) s_lo = s_hi;
    // SEG_UNROLL independent loads in flight per thread, then their counts
    constexpr int SEG_UNROLL = 8;
    int64_t i = s_lo + threadIdx.x;
    for (; i + (SEG_UNROLL - 1) * HIST_THREADS < s_hi; i += SEG_UNROLL * HIST_THREADS) {
        K k[SEG_UNROLL];
#pragma unroll
        for (int u = 0; u < SEG_UNROLL; ++u) k[u] = __ldg(keys + i + u * HIST_THREADS);
#pragma unroll
        for (int u = 0; u < SEG_UNROLL; ++u) atomicAdd(&cnt[(hash_key(k[u]) >> it.f.shift) & it.f.mask], 1u);
    }
    for (; i < s_hi; i += HIST_THREADS) atomicAdd(&cnt[(hash_key(keys[i]) >> it.f.shift) & it.f.mask], 1u);
    __syncthreads();
    for (int p = threadIdx.x; p < it.P; p += HIST_THREADS) {
        const uint32_t c = cnt[p];
        if (c) {
            atomicAdd(&counts[it.cnt_base + static_cast<int64_t>(p) * it.seg_items + it.item], c);
            atomicAdd(&totals[it.tot_base + p], static_cast<int32_t>(c));
        }
    }
}

// Write-combining scatter of the items (persistent grid; buffers sized for
// the largest partition count of the batch, Pmax; an item's SEG_CHUNK rows
// stay below WCU_EPOCH).
template <typename K, int THREADS, int VT>
__global__ void __launch_bounds__(THREADS, 1) scatter_seg_kernel(const SegItem* __restrict__ items, int32_t n_items,
                                                                 int32_t Pmax, int32_t logF, int32_t W,
                                                                 const int64_t* __restrict__ offsets,
                                                                 uint32_t* __restrict__ out, uint32_t out_cap,
                                                                 uint32_t* __restrict__ status)
{
    constexpr int TW = TupleTraits<K>::WORDS;
    constexpr int ROUND = THREADS * VT;
    extern __shared__ __align__(128) uint8_t smem[];
    WcUnits<K> wc;
    wc.bind(smem, Pmax, logF, VT);
    uint32_t n_late = 0;
    for (int32_t i = blockIdx.x; i < n_items; i += gridDim.x) {
        const SegItem it = items[i];
        const int64_t* off = offsets + it.cnt_base;
        wcu_begin<K>(wc, it.P, [&](int p) { return off[static_cast<int64_t>(p) * it.seg_items + it.item]; },
                     [&](int p) { return off[static_cast<int64_t>(p) * it.seg_items + it.item + 1]; });
        const K* keys = static_cast<const K*>(it.keys);
        K nk[VT];
        auto load_round = [&](int64_t b) {
#pragma unroll
            for (int v = 0; v < VT; ++v) {
                const int64_t r = b + static_cast<int64_t>(v) * THREADS + threadIdx.x;
                nk[v] = r < it.hi ? keys[r] : K(0);
            }
        };
        if (it.lo < it.hi) load_round(it.lo);
        for (int64_t b = it.lo; b < it.hi; b += ROUND) {
            uint32_t w[VT][TW];
            uint32_t dv[VT];
            bool ok[VT];
#pragma unroll
            for (int v = 0; v < VT; ++v) {
                const int64_t r = b + static_cast<int64_t>(v) * THREADS + threadIdx.x;
                ok[v] = r < it.hi;
                tuple_words<K>(w[v], nk[v], static_cast<int32_t>(r));
                dv[v] = (tuple_hash<K>(w[v]) >> it.f.shift) & it.f.mask;
            }
            if (b + ROUND < it.hi) load_round(b + ROUND);
            wcu_place<K, VT>(wc, n_late, w, dv, ok, out, out_cap, status);
        }
        wcu_finish<K>(wc, n_late, it.P, static_cast<uint32_t>(W), out, out_cap, status);
    }
}

}  // namespace pj
