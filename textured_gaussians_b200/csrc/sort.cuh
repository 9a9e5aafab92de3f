// Building blocks of the radix sorts: one onesweep pass over 4096-pair tiles, and a whole sort in one CTA.
#pragma once
#include "tg_common.cuh"

namespace tg {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;  // 4096 keys per CTA
constexpr int kRadix = 256;
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagInc = 2u << 30;
constexpr uint32_t kFlagMask = 3u << 30;
constexpr uint32_t kValueMask = kFlagAgg - 1u;
constexpr uint32_t kSpinLimit = 1u << 22;  // ~0.3 s of polling with 64 ns sleeps
// Predecessors whose status a look-back step reads at once.  The tiles of a launch's first wave publish their counts
// together, so tile k meets the first finished prefix after about k / (2 kWindow) steps of one memory latency
// each: read one at a time, the 560 tiles of a 2.3M-pair sort took 48 us a pass, most of it in this walk.
constexpr int kWindow = 16;

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t* p) { return *reinterpret_cast<const volatile uint32_t*>(p); }
__device__ __forceinline__ void st_volatile(uint32_t* p, uint32_t v) { *reinterpret_cast<volatile uint32_t*>(p) = v; }

// The lanes whose item is valid and has the calling lane's digit.
__device__ __forceinline__ unsigned digit_peers(uint32_t d, bool ok, int bits) {
    unsigned peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        if (b >= bits) break;  // uniform
        const bool set = (d >> b) & 1u;
        const unsigned m = __ballot_sync(0xffffffffu, set);
        peers &= set ? m : ~m;
    }
    return peers;
}

// Ranks the calling warp's item among its warp's earlier items of the same digit, counting in wh[256].
__device__ __forceinline__ uint32_t warp_rank(uint32_t d, bool ok, int bits, uint32_t* wh) {
    const int lane = threadIdx.x & 31;
    const unsigned peers = digit_peers(d, ok, bits);
    const int leader = (__ffs(peers) - 1) & 31;
    uint32_t before = 0;
    if (ok && lane == leader) {
        before = wh[d];
        wh[d] = before + __popc(peers);
    }
    __syncwarp();
    return __shfl_sync(0xffffffffu, before, leader) + __popc(peers & lanemask_lt());
}

// Sum of the digit's counts over all earlier tiles (status: [tiles][256], the calling thread's digit d).
__device__ __forceinline__ uint32_t look_back(const uint32_t* status, uint32_t tile, int d, uint32_t* error) {
    uint32_t prefix = 0;
    for (int64_t j = (int64_t)tile - 1; j >= 0; j -= kWindow) {
        uint32_t s[kWindow];
#pragma unroll
        for (int q = 0; q < kWindow; ++q)
            s[q] = j - q >= 0 ? ld_volatile(status + (size_t)(j - q) * kRadix + d) : kFlagInc;
#pragma unroll
        for (int q = 0; q < kWindow; ++q) {
            uint32_t iter = 0;
            while ((s[q] & kFlagMask) == 0u) {
                if (++iter > kSpinLimit) {  // gave up: record and stop waiting
                    atomicExch(error, 1u);
                    return prefix;
                }
                __nanosleep(64);
                s[q] = ld_volatile(status + (size_t)(j - q) * kRadix + d);
            }
            prefix += s[q] & kValueMask;
            if (s[q] & kFlagInc) return prefix;
        }
    }
    return prefix;
}

template <class Key>
constexpr size_t sort_pass_smem() {
    return (sizeof(Key) + sizeof(uint32_t)) * kSortTile + sizeof(uint32_t) * (kSortWarps * kRadix + 2 * kRadix);
}

// One pass of a stable LSD radix sort over digit bits [shift, shift + bits), bits <= 8: the CTA takes the next
// 4096-pair tile, ranks it, exchanges it through shared memory and writes each digit's run where the digit's earlier
// pairs end.  load(pos, key, value) / store(pos, key, value); hist: the pass's digit counts over all keys.
// After a look-back that gave up, some places of the output are not written, and the next pass finds digits there that
// hist has not counted: its places are held below n.
template <class Key, class Load, class Store>
__device__ __forceinline__ void sort_pass(Load load, Store store, int64_t n, int shift, int bits,
                                          const uint32_t* __restrict__ hist, uint32_t* status, uint32_t* tile_counter,
                                          uint32_t* error) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Key* s_keys = reinterpret_cast<Key*>(smem_raw);
    uint32_t* s_vals = reinterpret_cast<uint32_t*>(s_keys + kSortTile);
    uint32_t* s_whist = s_vals + kSortTile;             // [warps][256]
    uint32_t* s_start = s_whist + kSortWarps * kRadix;  // [256] first slot of each digit in the tile
    uint32_t* s_gbase = s_start + kRadix;               // [256] output position of slot j: s_gbase[digit] + j
    __shared__ uint32_t s_tile;
    __shared__ uint64_t s_scan[kSortWarps];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t digit_mask = (1u << bits) - 1u;
    if (tid == 0) s_tile = atomicAdd(tile_counter, 1u);
    for (int i = tid; i < kSortWarps * kRadix; i += kSortThreads) s_whist[i] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t base = (int64_t)tile * kSortTile;

    Key k[kSortItems];
    uint32_t v[kSortItems], rk[kSortItems / 2];  // ranks, two to a word
    const int64_t wbase = base + (int64_t)warp * (kSortItems * 32) + lane;
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        k[i] = 0;
        v[i] = 0;
        if (wbase + i * 32 < n) load(wbase + i * 32, k[i], v[i]);
    }
    uint32_t* wh = s_whist + warp * kRadix;
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        const uint32_t r = warp_rank((uint32_t)(k[i] >> shift) & digit_mask, wbase + i * 32 < n, bits, wh);
        rk[i >> 1] = (i & 1) ? (rk[i >> 1] | (r << 16)) : r;
    }
    __syncthreads();

    // per digit (thread = digit): exclusive scan over warps, tile total
    const int d = tid;
    uint32_t count = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t c = s_whist[w * kRadix + d];
        s_whist[w * kRadix + d] = count;
        count += c;
    }
    uint32_t* st = status + (size_t)tile * kRadix;
    st_volatile(st + d, (tile == 0 ? kFlagInc : kFlagAgg) | count);
    // one scan over the digits for both the tile's counts (low half) and all keys' (high half)
    const uint64_t own = ((uint64_t)hist[d] << 32) | count;
    uint64_t incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) s_scan[warp] = incl;
    __syncthreads();
    uint64_t excl = incl - own;
    for (int w = 0; w < warp; ++w) excl += s_scan[w];
    const uint32_t start = (uint32_t)excl;
    s_start[d] = start;
    __syncthreads();
    // the exchange first: the keys' registers are free before the look-back's window needs them
#pragma unroll
    for (int i = 0; i < kSortItems; ++i) {
        if (wbase + i * 32 < n) {
            const uint32_t dg = (uint32_t)(k[i] >> shift) & digit_mask;
            const uint32_t p = s_start[dg] + wh[dg] + ((i & 1) ? rk[i >> 1] >> 16 : rk[i >> 1] & 0xffffu);
            s_keys[p] = k[i];
            s_vals[p] = v[i];
        }
    }
    const uint32_t prefix = tile > 0 ? look_back(status, tile, d, error) : 0u;
    if (tile > 0) st_volatile(st + d, kFlagInc | (prefix + count));
    s_gbase[d] = (uint32_t)(excl >> 32) + prefix - start;
    __syncthreads();
    const int64_t rem = n - base;
    const int tile_n = rem < kSortTile ? (int)rem : kSortTile;
    for (int j = tid; j < tile_n; j += kSortThreads) {
        const Key key = s_keys[j];
        const uint32_t pos = s_gbase[(uint32_t)(key >> shift) & digit_mask] + (uint32_t)j;
        store((int64_t)min(pos, (uint32_t)n - 1u), key, s_vals[j]);  // (a branch here: 57 -> 65 us for the last list pass)
    }
}

// A whole stable sort of n <= kSmallSort (32-bit key, index) pairs on key bits [0, end_bit) by one CTA of 1024
// threads.  Returns with the sorted keys and indices in shared memory (s_keys / s_idx below); one launch, where the
// onesweep passes take two launches and a memset plus one launch per 8 bits, each of about 7 us at such sizes.
// load(i, counts) gives the key and whether the pair's place matters: a digit in which no two such keys differ (a
// depth's sign and exponent, a list length's upper bits) needs no pass, about 8 us at 10,000 pairs.
constexpr int kSmallThreads = 1024;
constexpr int kSmallItems = 16;
constexpr int kSmallSort = kSmallThreads * kSmallItems;
constexpr size_t kSmallSmem = sizeof(uint32_t) * (2 * kSmallSort + kRadix) + sizeof(uint16_t) * 32 * kRadix;

template <class Load>
__device__ __forceinline__ void sort_small(Load load, int n, int end_bit, uint32_t*& s_keys, uint32_t*& s_idx) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    s_keys = reinterpret_cast<uint32_t*>(smem_raw);
    s_idx = s_keys + kSmallSort;
    uint32_t* s_start = s_idx + kSmallSort;                           // [256]
    uint16_t* s_whist = reinterpret_cast<uint16_t*>(s_start + kRadix);  // [32 warps][256]
    __shared__ uint32_t s_scan[kRadix / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int items = (n + kSmallThreads - 1) / kSmallThreads;  // per thread; warp w owns a run of 32 * items
    const int wbase = warp * 32 * items + lane;
    __shared__ uint32_t s_ones, s_zeros;
    if (tid == 0) s_ones = s_zeros = 0u;
    __syncthreads();
    uint32_t ones = 0u, zeros = 0u;
    for (int i = tid; i < n; i += kSmallThreads) {
        bool counts = true;
        const uint32_t k = load(i, counts);
        s_keys[i] = k;
        s_idx[i] = (uint32_t)i;
        if (counts) {
            ones |= k;
            zeros |= ~k;
        }
    }
    ones = __reduce_or_sync(0xffffffffu, ones);
    zeros = __reduce_or_sync(0xffffffffu, zeros);
    if (lane == 0) {
        atomicOr(&s_ones, ones);
        atomicOr(&s_zeros, zeros);
    }
    __syncthreads();
    const uint32_t differ = s_ones & s_zeros;
    uint16_t* wh = s_whist + warp * kRadix;
    const int passes = (end_bit + 7) / 8;
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p, bits = min(8, end_bit - shift);
        const uint32_t digit_mask = (1u << bits) - 1u;
        if (((differ >> shift) & digit_mask) == 0u) continue;  // (uniform)
        for (int i = tid; i < 32 * kRadix / 2; i += kSmallThreads) reinterpret_cast<uint32_t*>(s_whist)[i] = 0u;
        __syncthreads();
        uint32_t k[kSmallItems], v[kSmallItems], rk[kSmallItems / 2];
#pragma unroll
        for (int i = 0; i < kSmallItems; ++i) {
            if (i >= items) break;  // uniform
            const bool ok = wbase + i * 32 < n;
            k[i] = ok ? s_keys[wbase + i * 32] : 0u;
            v[i] = ok ? s_idx[wbase + i * 32] : 0u;
            const uint32_t dg = (k[i] >> shift) & digit_mask;
            const unsigned peers = digit_peers(dg, ok, bits);
            const int leader = (__ffs(peers) - 1) & 31;
            uint32_t before = 0;
            if (ok && lane == leader) {
                before = wh[dg];
                wh[dg] = (uint16_t)(before + __popc(peers));
            }
            __syncwarp();
            const uint32_t r = __shfl_sync(0xffffffffu, before, leader) + __popc(peers & lanemask_lt());
            rk[i >> 1] = (i & 1) ? (rk[i >> 1] | (r << 16)) : r;
        }
        __syncthreads();
        uint32_t count = 0, incl = 0;
        if (tid < kRadix) {  // exclusive scan of each digit over the warps, then of the digits
            for (int w = 0; w < 32; ++w) {
                const uint32_t c = s_whist[w * kRadix + tid];
                s_whist[w * kRadix + tid] = (uint16_t)count;
                count += c;
            }
            incl = count;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += u;
            }
            if (lane == 31) s_scan[warp] = incl;
        }
        __syncthreads();
        if (tid < kRadix) {
            uint32_t excl = incl - count;
            for (int w = 0; w < warp; ++w) excl += s_scan[w];
            s_start[tid] = excl;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kSmallItems; ++i) {
            if (i >= items) break;
            if (wbase + i * 32 < n) {
                const uint32_t dg = (k[i] >> shift) & digit_mask;
                const uint32_t q = s_start[dg] + wh[dg] + ((i & 1) ? rk[i >> 1] >> 16 : rk[i >> 1] & 0xffffu);
                s_keys[q] = k[i];
                s_idx[q] = v[i];
            }
        }
        __syncthreads();
    }
    __syncthreads();
}

}  // namespace tg
