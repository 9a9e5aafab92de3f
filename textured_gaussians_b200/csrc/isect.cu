// Tile intersection, prefix sum, onesweep radix sort and tile offsets for sm_100a.
//
// Semantics follow textured_gaussians/cuda/csrc/isect_tiles.cu of the
// reference:  per projected Gaussian the tile AABB [floor((x-r)/ts),
// ceil((x+r)/ts)) clamped to the grid (:60-70), keys
// cam << (32+tile_bits) | tile << 32 | sign-extended float bits of depth
// (:90-101), a stable sort on key bits [0, 32+tile_bits+cam_bits) (:262-299)
// and per-tile run offsets (:309-355).
//
// The sort is a hand-written LSD onesweep radix sort (8-bit digits): one
// read of the keys builds the digit histograms of every pass, then each pass
// is a single kernel whose CTAs take 4096-key tiles in launch order, rank the
// keys with warp ballots, publish their digit counts and resolve their
// global digit offsets by decoupled look-back over earlier tiles (sort.cuh).
// Every look-back wait is bounded; a wait that gives up raises an error flag in
// the sort's workspace, which tg_sort_status, tg_isect_sorted_status and
// tg_tile_order_status turn into TG_ERR_TIMEOUT.
//
// Sorted intersection lists (the renderer's path) do not sort the 64-bit keys.
// An entry's intersections share its depth, so the entries are sorted by depth
// once, their intersections written in that order, and only the (camera, tile)
// half of the keys is left to sort -- stably, which gives the same order as
// sorting the whole keys, ties included.  Against seven passes of 24 bytes a pair
// over the intersections (1M splats x four 1600x1200 views, 30M of them, 4M
// entries) that is four passes of 16 bytes an entry and three of 16-20 bytes a pair.
#include "scan.cuh"
#include "sort.cuh"

namespace tg {

// ------------------------------------------------------------------ tile boxes
__device__ __forceinline__ void tile_box(float mx, float my, int32_t radius, int tile_size, uint32_t tw, uint32_t th,
                                         uint32_t& x0, uint32_t& y0, uint32_t& x1, uint32_t& y1) {
    const float ts = (float)tile_size;
    const float tr = __fdiv_rn((float)radius, ts);
    const float tx = __fdiv_rn(mx, ts), ty = __fdiv_rn(my, ts);
    // float -> u32 conversions saturate (negative -> 0), as in the reference
    x0 = min((uint32_t)floorf(tx - tr), tw);
    y0 = min((uint32_t)floorf(ty - tr), th);
    x1 = min((uint32_t)ceilf(tx + tr), tw);
    y1 = min((uint32_t)ceilf(ty + tr), th);
}

// Camera of element e and its tile grid; false if the camera id is out of range.
__device__ __forceinline__ bool camera_grid(const tg_isect_args& a, int64_t e, uint32_t& tw, uint32_t& th) {
    const int64_t cid = a.camera_ids ? a.camera_ids[e] : e / a.N;
    if (cid < 0 || cid >= a.n_cameras) return false;
    if (a.views) {
        tw = (uint32_t)a.views[cid].tile_width;
        th = (uint32_t)a.views[cid].tile_height;
    } else {
        tw = (uint32_t)a.tile_width;
        th = (uint32_t)a.tile_height;
    }
    return true;
}

// Phase 1: tile counts per element and per-chunk sums.
__global__ void __launch_bounds__(kScanThreads) isect_count_kernel(tg_isect_args a, int64_t* chunk_sums) {
    __shared__ int64_t s_warp[kScanThreads / 32];
    const int64_t base = (int64_t)blockIdx.x * kScanChunk;
    int64_t local = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const int64_t e = base + (int64_t)i * kScanThreads + threadIdx.x;
        if (e >= a.n_elems) break;
        int32_t cnt = 0;
        const int32_t r = a.radii[e];
        uint32_t tw, th;
        if (r > 0 && camera_grid(a, e, tw, th)) {
            const float2 m = reinterpret_cast<const float2*>(a.means2d)[e];
            uint32_t x0, y0, x1, y1;
            tile_box(m.x, m.y, r, a.tile_size, tw, th, x0, y0, x1, y1);
            cnt = (int32_t)((y1 - y0) * (x1 - x0));
        }
        a.tiles_per_gauss[e] = cnt;
        local += cnt;
    }
    int64_t total;
    block_excl_scan(local, s_warp, total);
    if (threadIdx.x == 0) chunk_sums[blockIdx.x] = total;
}

// Phase 2: exclusive scan of the chunk sums in one CTA; writes the grand total.
__global__ void __launch_bounds__(kScanThreads) scan_chunk_sums_kernel(int64_t* chunk_sums, int64_t n_chunks,
                                                                       int64_t* n_total) {
    __shared__ int64_t s_warp[kScanThreads / 32];
    int64_t carry = 0;
    for (int64_t b = 0; b < n_chunks; b += kScanThreads) {
        const int64_t i = b + threadIdx.x;
        const int64_t v = i < n_chunks ? chunk_sums[i] : 0;
        int64_t total;
        const int64_t ex = block_excl_scan(v, s_warp, total);
        if (i < n_chunks) chunk_sums[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) *n_total = carry;
}

cudaError_t launch_scan_chunk_sums(int64_t* chunk_sums, int64_t n_chunks, int64_t* n_total, cudaStream_t s) {
    scan_chunk_sums_kernel<<<1, kScanThreads, 0, s>>>(chunk_sums, n_chunks, n_total);
    note_launches(1);
    return cudaGetLastError();
}

// Phase 3: inclusive prefix of tiles_per_gauss within each chunk plus the chunk offset.
__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(const int32_t* counts, int64_t n,
                                                                  const int64_t* chunk_offsets, int64_t* cum) {
    __shared__ int64_t s_warp[kScanThreads / 32];
    const int64_t base = (int64_t)blockIdx.x * kScanChunk;
    // blocked arrangement: thread t owns items [t*16, t*16+16) of the chunk
    int32_t v[kScanItems];
    int64_t local = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const int64_t e = base + (int64_t)threadIdx.x * kScanItems + i;
        v[i] = e < n ? counts[e] : 0;
        local += v[i];
    }
    int64_t total;
    int64_t run = chunk_offsets[blockIdx.x] + block_excl_scan(local, s_warp, total);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const int64_t e = base + (int64_t)threadIdx.x * kScanItems + i;
        run += v[i];
        if (e < n) cum[e] = run;
    }
}

__global__ void __launch_bounds__(256) isect_emit_kernel(tg_isect_args a, int tile_n_bits) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= a.n_elems) return;
    const int32_t r = a.radii[e];
    uint32_t tw, th;
    if (r <= 0 || !camera_grid(a, e, tw, th)) return;
    const float2 m = reinterpret_cast<const float2*>(a.means2d)[e];
    uint32_t x0, y0, x1, y1;
    tile_box(m.x, m.y, r, a.tile_size, tw, th, x0, y0, x1, y1);
    const int64_t cid = a.camera_ids ? a.camera_ids[e] : e / a.N;
    const int64_t cid_enc = cid << (32 + tile_n_bits);
    const int64_t depth_enc = (int64_t)__float_as_int(a.depths[e]);  // sign-extended like the reference
    int64_t cur = e == 0 ? 0 : a.cum_tiles[e - 1];
    // capacity mode: only the first `capacity` entries exist
    const int64_t limit = a.overflow ? a.capacity : INT64_MAX;
    if (a.overflow && a.cum_tiles[e] > limit) atomicOr(a.overflow, 1u);
    for (uint32_t y = y0; y < y1; ++y)
        for (uint32_t x = x0; x < x1; ++x) {
            if (cur >= limit) return;
            const int64_t tile_id = (int64_t)y * tw + x;
            a.isect_ids[cur] = cid_enc | (tile_id << 32) | depth_enc;
            a.flatten_ids[cur] = (int32_t)e;
            ++cur;
        }
}

// Capacity mode: keys past the valid count sort after every real key.
__global__ void __launch_bounds__(256) isect_pad_kernel(int64_t* keys, int32_t* vals, const int64_t* n_dev,
                                                        int64_t capacity, int64_t pad_key) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= capacity || i < *n_dev) return;
    keys[i] = pad_key;
    vals[i] = 0;
}

// offsets[t] = lower_bound over sorted keys of (camera, tile) index t.
__global__ void __launch_bounds__(256) offset_encode_kernel(const int64_t* keys, int64_t n, int64_t n_ids,
                                                            int n_tiles, int tile_n_bits, uint64_t key_mask,
                                                            int32_t* offsets) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_ids) return;
    int64_t lo = 0, hi = n;
    const uint64_t tmask = (1ull << tile_n_bits) - 1ull;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        const uint64_t h = ((uint64_t)__ldg(keys + mid) & key_mask) >> 32;
        const int64_t id = (int64_t)(h >> tile_n_bits) * n_tiles + (int64_t)(h & tmask);
        if (id < t) lo = mid + 1; else hi = mid;
    }
    offsets[t] = (int32_t)lo;
}

// Batching form: flat tile t of view c = tile_view[t] is the key prefix
// (c << tile_bits) | (t - tile_base_c); offsets[t] = its lower bound.
__global__ void __launch_bounds__(256) offset_encode_views_kernel(const int64_t* keys, int64_t n, int64_t n_tiles,
                                                                  int C, const tg_view* views,
                                                                  const int32_t* tile_view, int tile_n_bits,
                                                                  uint64_t key_mask, int32_t* offsets) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_tiles) return;
    const int c = tile_view[t];
    uint64_t target = ~0ull;  // an out-of-range view sorts after every key
    if (c >= 0 && c < C) target = ((uint64_t)c << tile_n_bits) | (uint64_t)(t - views[c].tile_base);
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        const uint64_t h = ((uint64_t)__ldg(keys + mid) & key_mask) >> 32;
        if (h < target) lo = mid + 1; else hi = mid;
    }
    offsets[t] = (int32_t)lo;
}

// ------------------------------------------------------------------ onesweep radix sort
constexpr int kMaxPasses = 8;

struct SortWorkspace {
    uint32_t* hist;          // [kMaxPasses][256] digit counts
    uint32_t* tile_counter;  // [kMaxPasses]
    uint32_t* error;         // [1]
    uint32_t* status;        // [passes][n_tiles][256]
    size_t bytes;
};


inline SortWorkspace carve_sort_workspace(void* base, int64_t n, int passes) {
    SortWorkspace w;
    const int64_t n_tiles = (n + kSortTile - 1) / kSortTile;
    char* p = static_cast<char*>(base);
    size_t off = 0;
    w.hist = reinterpret_cast<uint32_t*>(p + off); off += align256(sizeof(uint32_t) * kMaxPasses * kRadix);
    w.tile_counter = reinterpret_cast<uint32_t*>(p + off); off += align256(sizeof(uint32_t) * kMaxPasses);
    w.error = reinterpret_cast<uint32_t*>(p + off); off += align256(sizeof(uint32_t));
    w.status = reinterpret_cast<uint32_t*>(p + off); off += align256(sizeof(uint32_t) * (size_t)passes * n_tiles * kRadix);
    w.bytes = off;
    return w;
}

__global__ void __launch_bounds__(kSortThreads) sort_histogram_kernel(const uint64_t* keys, int64_t n, int passes,
                                                                      int end_bit, uint32_t* hist) {
    __shared__ uint32_t s_hist[kMaxPasses * kRadix];
    for (int i = threadIdx.x; i < passes * kRadix; i += kSortThreads) s_hist[i] = 0;
    __syncthreads();
    const uint64_t mask = end_bit >= 64 ? ~0ull : ((1ull << end_bit) - 1ull);
    for (int64_t i = (int64_t)blockIdx.x * kSortThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kSortThreads) {
        const uint64_t k = keys[i] & mask;
        for (int p = 0; p < passes; ++p) atomicAdd(&s_hist[p * kRadix + ((k >> (8 * p)) & 0xffu)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * kRadix; i += kSortThreads)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

template <class Key>
__global__ void __launch_bounds__(kSortThreads, 3) sort_pass_kernel(const Key* __restrict__ keys_in,
                                                                 const uint32_t* __restrict__ vals_in,
                                                                 Key* __restrict__ keys_out,
                                                                 uint32_t* __restrict__ vals_out, int64_t n, int shift,
                                                                 int bits, const uint32_t* hist, uint32_t* status,
                                                                 uint32_t* tile_counter, uint32_t* error) {
    sort_pass<Key>(
        [&](int64_t i, Key& k, uint32_t& v) {
            k = keys_in[i];
            v = vals_in[i];
        },
        [&](int64_t i, Key k, uint32_t v) {
            keys_out[i] = k;
            vals_out[i] = v;
        },
        n, shift, bits, hist, status, tile_counter, error);
}

size_t sort_workspace_bytes(int64_t n, int end_bit) {
    const int passes = (end_bit + 7) / 8;
    return carve_sort_workspace(nullptr, n, passes).bytes;
}

// Returns TG_OK / TG_ERR_*; *result_in_alt tells where the sorted data ends.
int sort_pairs(int64_t* keys, int32_t* vals, int64_t* keys_alt, int32_t* vals_alt, int64_t n, int end_bit,
               void* workspace, size_t ws_bytes, int32_t* result_in_alt, cudaStream_t s, cudaError_t& cerr) {
    cerr = cudaSuccess;
    *result_in_alt = 0;
    if (n <= 1 || end_bit <= 0) return TG_OK;
    const int passes = (end_bit + 7) / 8;
    if (passes > kMaxPasses) return TG_ERR_INVALID_ARG;
    SortWorkspace w = carve_sort_workspace(workspace, n, passes);
    if (ws_bytes < w.bytes) return TG_ERR_WORKSPACE;
    const int64_t n_tiles = (n + kSortTile - 1) / kSortTile;
    if ((cerr = cudaMemsetAsync(workspace, 0, w.bytes, s)) != cudaSuccess) return TG_ERR_CUDA;
    const int hist_blocks = (int)std::min<int64_t>(n_tiles, (int64_t)kNumSMs * 4);
    sort_histogram_kernel<<<hist_blocks, kSortThreads, 0, s>>>(reinterpret_cast<const uint64_t*>(keys), n, passes,
                                                               end_bit, w.hist);
    note_launches(1);
    if ((cerr = cudaGetLastError()) != cudaSuccess) return TG_ERR_CUDA;
    // a per-device function attribute: set on every call (cheap, allowed during stream capture)
    constexpr size_t smem = sort_pass_smem<uint64_t>();
    if ((cerr = cudaFuncSetAttribute(sort_pass_kernel<uint64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem)) != cudaSuccess)
        return TG_ERR_CUDA;
    uint64_t* kin = reinterpret_cast<uint64_t*>(keys);
    uint32_t* vin = reinterpret_cast<uint32_t*>(vals);
    uint64_t* kout = reinterpret_cast<uint64_t*>(keys_alt);
    uint32_t* vout = reinterpret_cast<uint32_t*>(vals_alt);
    for (int p = 0; p < passes; ++p) {
        const int shift = 8 * p;
        sort_pass_kernel<uint64_t><<<(unsigned)n_tiles, kSortThreads, smem, s>>>(
            kin, vin, kout, vout, n, shift, std::min(8, end_bit - shift), w.hist + p * kRadix,
            w.status + (size_t)p * n_tiles * kRadix, w.tile_counter + p, w.error);
        if ((cerr = cudaGetLastError()) != cudaSuccess) return TG_ERR_CUDA;
        note_launches(1);
        std::swap(kin, kout);
        std::swap(vin, vout);
    }
    *result_in_alt = passes & 1;
    return TG_OK;
}

__global__ void set_u32_kernel(uint32_t* p, uint32_t v) { *p = v; }

// Diagnostic: one pass over two tiles (8192 pairs, 8 key bits) run by a single
// CTA whose tile counter is preset to 1, so its look-back waits on tile 0,
// which never publishes.  The bounded wait gives up after kSpinLimit polls and
// raises the error flag; a partial prefix only lowers scatter positions, so
// every write stays inside the output buffers.
int sort_lookback_selftest(int64_t* keys, int32_t* vals, int64_t* keys_alt, int32_t* vals_alt, void* workspace,
                           size_t ws_bytes, cudaStream_t s, cudaError_t& cerr) {
    cerr = cudaSuccess;
    constexpr int64_t n = 2 * kSortTile;
    SortWorkspace w = carve_sort_workspace(workspace, n, 1);
    if (ws_bytes < w.bytes) return TG_ERR_WORKSPACE;
    if ((cerr = cudaMemsetAsync(workspace, 0, w.bytes, s)) != cudaSuccess) return TG_ERR_CUDA;
    set_u32_kernel<<<1, 1, 0, s>>>(w.tile_counter, 1u);  // the single CTA takes tile 1
    sort_histogram_kernel<<<2, kSortThreads, 0, s>>>(reinterpret_cast<const uint64_t*>(keys), n, 1, 8, w.hist);
    constexpr size_t smem = sort_pass_smem<uint64_t>();
    if ((cerr = cudaFuncSetAttribute(sort_pass_kernel<uint64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem)) != cudaSuccess)
        return TG_ERR_CUDA;
    sort_pass_kernel<uint64_t><<<1, kSortThreads, smem, s>>>(
        reinterpret_cast<const uint64_t*>(keys), reinterpret_cast<const uint32_t*>(vals),
        reinterpret_cast<uint64_t*>(keys_alt), reinterpret_cast<uint32_t*>(vals_alt), n, 0, 8, w.hist, w.status,
        w.tile_counter, w.error);
    note_launches(3);
    if ((cerr = cudaGetLastError()) != cudaSuccess) return TG_ERR_CUDA;
    uint32_t h = 0;
    if ((cerr = cudaStreamSynchronize(s)) != cudaSuccess) return TG_ERR_CUDA;
    if ((cerr = cudaMemcpy(&h, w.error, sizeof(h), cudaMemcpyDeviceToHost)) != cudaSuccess) return TG_ERR_CUDA;
    return h ? TG_ERR_TIMEOUT : TG_OK;
}

// error flag location inside a carved workspace (for the host to read back)
uint32_t* sort_error_flag(void* workspace, int64_t n, int end_bit) {
    return carve_sort_workspace(workspace, n, (end_bit + 7) / 8).error;
}

size_t scan_workspace_bytes(int64_t n_elems) {
    const int64_t chunks = (n_elems + kScanChunk - 1) / kScanChunk;
    return align256(sizeof(int64_t) * (size_t)std::max<int64_t>(chunks, 1));
}

cudaError_t launch_isect_count(const tg_isect_args& a, cudaStream_t s) {
    const int64_t chunks = (a.n_elems + kScanChunk - 1) / kScanChunk;
    if (a.n_elems == 0) return cudaMemsetAsync(a.n_isects, 0, sizeof(int64_t), s);
    int64_t* sums = static_cast<int64_t*>(a.scan_workspace);
    isect_count_kernel<<<(unsigned)chunks, kScanThreads, 0, s>>>(a, sums);
    scan_chunk_sums_kernel<<<1, kScanThreads, 0, s>>>(sums, chunks, a.n_isects);
    scan_apply_kernel<<<(unsigned)chunks, kScanThreads, 0, s>>>(a.tiles_per_gauss, a.n_elems, sums, a.cum_tiles);
    note_launches(3);
    return cudaGetLastError();
}

cudaError_t launch_isect_emit(const tg_isect_args& a, int tile_n_bits, int end_bit, cudaStream_t s) {
    if (a.n_elems > 0) {
        isect_emit_kernel<<<(unsigned)((a.n_elems + 255) / 256), 256, 0, s>>>(a, tile_n_bits);
        note_launches(1);
    }
    if (a.overflow && a.capacity > 0) {
        const int64_t pad = end_bit >= 63 ? INT64_MAX : (int64_t)((1ull << end_bit) - 1ull);
        isect_pad_kernel<<<(unsigned)((a.capacity + 255) / 256), 256, 0, s>>>(a.isect_ids, a.flatten_ids, a.n_isects,
                                                                              a.capacity, pad);
        note_launches(1);
    }
    return cudaGetLastError();
}

cudaError_t launch_offset_encode_views(const int64_t* keys, int64_t n, int C, int64_t n_tiles, const tg_view* views,
                                       const int32_t* tile_view, int tile_n_bits, int end_bit, int32_t* offsets,
                                       cudaStream_t s) {
    if (n_tiles == 0) return cudaSuccess;
    const uint64_t key_mask = end_bit >= 64 ? ~0ull : ((1ull << end_bit) - 1ull);
    offset_encode_views_kernel<<<(unsigned)((n_tiles + 255) / 256), 256, 0, s>>>(keys, n, n_tiles, C, views, tile_view,
                                                                                tile_n_bits, key_mask, offsets);
    note_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_offset_encode(const int64_t* keys, int64_t n, int C, int tw, int th, int tile_n_bits,
                                 int end_bit, int32_t* offsets, cudaStream_t s) {
    const int64_t n_ids = (int64_t)C * tw * th;
    if (n_ids == 0) return cudaSuccess;
    const uint64_t mask = end_bit >= 64 ? ~0ull : ((1ull << end_bit) - 1ull);
    offset_encode_kernel<<<(unsigned)((n_ids + 255) / 256), 256, 0, s>>>(keys, n, n_ids, tw * th, tile_n_bits, mask,
                                                                       offsets);
    note_launches(1);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ sorted intersection lists
constexpr int kOrderChunk = 1024;  // depth-ordered entries per emission CTA
constexpr int kDepthPasses = 4;

// Scratch of the entry stage.
struct OrderWorkspace {
    uint32_t* hist;     // [4][256] depth digits  (zeroed, with all up to `status` inclusive)
    uint32_t* counter;  // [4] tiles taken, then the error flag
    uint32_t* status;   // [4][tiles][256]
    uint32_t *keys[2], *ids[2];  // ping-pong; the depth order ends in ids[1]
    int64_t* chunks;    // [chunks] intersections before each chunk of the depth order
    size_t zeroed, bytes;
};
inline OrderWorkspace carve_order_workspace(void* base, int64_t E) {
    OrderWorkspace w;
    char* p = static_cast<char*>(base);
    size_t off = 0;
    auto take = [&](size_t n) {
        char* q = p + off;
        off += align256(n);
        return q;
    };
    const int64_t tiles = E > kSmallSort ? (E + kSortTile - 1) / kSortTile : 0;  // the small sort needs no status
    w.hist = reinterpret_cast<uint32_t*>(take(4 * kDepthPasses * kRadix));
    w.counter = reinterpret_cast<uint32_t*>(take(4 * (kDepthPasses + 1)));
    w.status = reinterpret_cast<uint32_t*>(take(4 * (size_t)kDepthPasses * tiles * kRadix));
    w.zeroed = off;
    for (int i = 0; i < 2; ++i) w.keys[i] = reinterpret_cast<uint32_t*>(take(4 * (size_t)(tiles ? E : 0)));
    for (int i = 0; i < 2; ++i) w.ids[i] = reinterpret_cast<uint32_t*>(take(4 * (size_t)(tiles || i ? E : 0)));
    w.chunks = reinterpret_cast<int64_t*>(take(8 * ((E + kOrderChunk - 1) / kOrderChunk)));
    w.bytes = off;
    return w;
}
size_t isect_order_workspace_bytes(int64_t E) { return carve_order_workspace(nullptr, E).bytes; }

// Adds one to s[d] for every lane with ok, one add per warp where all its digits agree (a depth's exponent digits).
__device__ __forceinline__ void count_digit(uint32_t* s, uint32_t d, bool ok) {
    const unsigned m = __ballot_sync(0xffffffffu, ok);
    if (m == 0u) return;
    const uint32_t d0 = __shfl_sync(0xffffffffu, d, __ffs(m) - 1);
    if (__all_sync(0xffffffffu, !ok || d == d0)) {
        if ((threadIdx.x & 31) == 0) atomicAdd(s + d0, (uint32_t)__popc(m));
    } else if (ok) {
        atomicAdd(s + d, 1u);
    }
}

// Tile counts of the entries, their sum (added to the zeroed *n_isects), and the digit counts of their depths.  The
// host waits for the sum alone: the entries' sort comes after its read, so a small call does not wait for it (35 us
// of a 376 us frame, now 348; a plain training step of 150,000 splats 1774 -> 1687 us), and a large one is the same
// (1,000,000 entries: 311 us).  Eight CTAs an SM: at 36 registers the 977 CTAs of a million entries need a second
// wave (18.9 -> 25.1 us).
__global__ void __launch_bounds__(256, 8) order_count_kernel(tg_isect_args a, uint32_t* hist) {
    __shared__ uint32_t s_hist[kDepthPasses * kRadix];
    __shared__ int64_t s_warp[256 / 32];
    int64_t local = 0;
    if (hist != nullptr) {
        for (int i = threadIdx.x; i < kDepthPasses * kRadix; i += 256) s_hist[i] = 0;
        __syncthreads();
    }
    const int64_t first = (int64_t)blockIdx.x * kOrderChunk;
#pragma unroll 1
    for (int i = 0; i < kOrderChunk; i += 256) {
        const int64_t e = first + i + threadIdx.x;
        const bool in = e < a.n_elems;
        if (in) {
            int32_t cnt = 0;
            const int32_t r = a.radii[e];
            uint32_t tw, th;
            if (r > 0 && camera_grid(a, e, tw, th)) {
                const float2 m = reinterpret_cast<const float2*>(a.means2d)[e];
                uint32_t x0, y0, x1, y1;
                tile_box(m.x, m.y, r, a.tile_size, tw, th, x0, y0, x1, y1);
                cnt = (int32_t)((y1 - y0) * (x1 - x0));
            }
            a.tiles_per_gauss[e] = cnt;
            local += cnt;
        }
        if (hist != nullptr) {
            const uint32_t k = in ? __float_as_uint(a.depths[e]) : 0u;
#pragma unroll
            for (int p = 0; p < kDepthPasses; ++p) count_digit(s_hist + p * kRadix, (k >> (8 * p)) & 0xffu, in);
        }
    }
    int64_t sum;
    block_excl_scan(local, s_warp, sum);
    if (threadIdx.x == 0 && sum != 0)
        atomicAdd(reinterpret_cast<unsigned long long*>(a.n_isects), (unsigned long long)sum);
    if (hist == nullptr) return;
    for (int i = threadIdx.x; i < kDepthPasses * kRadix; i += 256)  // (the scan above is a barrier)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

// Pass p of the entries' depth sort; the first reads the depths themselves.
__global__ void __launch_bounds__(kSortThreads, 4) order_pass_kernel(const float* __restrict__ depths,
                                                                  const uint32_t* __restrict__ keys_in,
                                                                  const uint32_t* __restrict__ ids_in,
                                                                  uint32_t* __restrict__ keys_out,
                                                                  uint32_t* __restrict__ ids_out, int64_t n, int pass,
                                                                  const uint32_t* hist, uint32_t* status,
                                                                  uint32_t* counter, uint32_t* error) {
    sort_pass<uint32_t>(
        [&](int64_t i, uint32_t& k, uint32_t& v) {
            k = pass == 0 ? __float_as_uint(depths[i]) : keys_in[i];
            v = pass == 0 ? (uint32_t)i : ids_in[i];
        },
        [&](int64_t i, uint32_t k, uint32_t v) {
            if (pass != kDepthPasses - 1) keys_out[i] = k;  // (only the order is kept of the last)
            ids_out[i] = v;
        },
        n, 8 * pass, 8, hist, status, counter, error);
}

// The whole entry order and its chunk offsets by one CTA, for n <= kSmallSort (entries without tiles anywhere).
__global__ void __launch_bounds__(kSmallThreads) order_small_kernel(const float* __restrict__ depths,
                                                                    const int32_t* __restrict__ counts, int n,
                                                                    uint32_t* __restrict__ ids, int64_t* chunks) {
    static_assert(kSmallThreads == kOrderChunk && kSmallItems <= 32, "item i of all threads is chunk i");
    __shared__ int64_t s_part[kSmallItems][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, items = (n + kSmallThreads - 1) / kSmallThreads;
    uint32_t *s_keys, *s_idx;
    sort_small(
        [&](int i, bool& matters) {
            matters = counts[i] > 0;
            return __float_as_uint(depths[i]);
        },
        n, 32, s_keys, s_idx);
    for (int c = 0; c < items; ++c) {
        const int i = c * kSmallThreads + threadIdx.x;
        int64_t v = 0;
        if (i < n) {
            const uint32_t id = s_idx[i];
            ids[i] = id;
            v = counts[id];
        }
        v = warp_incl_scan(v);
        if (lane == 31) s_part[c][warp] = v;
    }
    __syncthreads();
    if (warp != 0) return;
    int64_t v = 0;
    if (lane < items)
        for (int w = 0; w < 32; ++w) v += s_part[lane][w];
    const int64_t incl = warp_incl_scan(v);
    if (lane < items) chunks[lane] = incl - v;
}

// Intersections of each chunk of the depth order.  (Here and below an id that is no entry's is passed over: a sort whose
// look-back gave up leaves places unwritten.)
__global__ void __launch_bounds__(256) order_sums_kernel(const uint32_t* __restrict__ ids,
                                                         const int32_t* __restrict__ counts, int64_t n,
                                                         int64_t* chunks) {
    __shared__ int64_t s_warp[kScanThreads / 32];
    int64_t local = 0;
#pragma unroll
    for (int i = 0; i < kOrderChunk; i += 256) {
        const int64_t k = (int64_t)blockIdx.x * kOrderChunk + i + threadIdx.x;
        const uint32_t e = k < n ? ids[k] : 0xffffffffu;
        if (e < (uint32_t)n) local += counts[e];
    }
    int64_t total;
    block_excl_scan(local, s_warp, total);
    if (threadIdx.x == 0) chunks[blockIdx.x] = total;
}

// Exclusive scan of the chunk sums by one CTA of 1024 threads, four sums each.
__global__ void __launch_bounds__(1024) order_scan_kernel(int64_t* chunks, int64_t n_chunks) {
    __shared__ int64_t s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t carry = 0;
    for (int64_t b = 0; b < n_chunks; b += 4096) {
        const int64_t i0 = b + threadIdx.x * 4;
        int64_t v[4], sum = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = i0 + k < n_chunks ? chunks[i0 + k] : 0;
            sum += v[k];
        }
        int64_t incl = warp_incl_scan(sum);
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        if (warp == 0) s_warp[lane] = warp_incl_scan(s_warp[lane]);
        __syncthreads();
        int64_t run = carry + incl - sum + (warp > 0 ? s_warp[warp - 1] : 0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (i0 + k < n_chunks) chunks[i0 + k] = run;
            run += v[k];
        }
        carry += s_warp[31];
        __syncthreads();
    }
}

// Counts of the entries' tiles and their sum.
cudaError_t launch_isect_order(const tg_isect_args& a, void* workspace, cudaStream_t s) {
    const int64_t E = a.n_elems;
    cudaError_t e = cudaMemsetAsync(a.n_isects, 0, sizeof(int64_t), s);
    if (e != cudaSuccess || E == 0) return e;
    const OrderWorkspace w = carve_order_workspace(workspace, E);
    const int64_t chunks = (E + kOrderChunk - 1) / kOrderChunk;
    const bool small = E <= kSmallSort;
    if (!small && (e = cudaMemsetAsync(workspace, 0, w.zeroed, s)) != cudaSuccess) return e;
    order_count_kernel<<<(unsigned)chunks, 256, 0, s>>>(a, small ? nullptr : w.hist);
    note_launches(1);
    return cudaGetLastError();
}

// The entries by depth and the offsets of its chunks.  lost: nobody takes the first tile of the first pass.
cudaError_t launch_entry_sort(const tg_isect_args& a, const OrderWorkspace& w, bool lost, cudaStream_t s) {
    const int64_t E = a.n_elems, chunks = (E + kOrderChunk - 1) / kOrderChunk;
    cudaError_t e;
    if (E <= kSmallSort) {
        if ((e = cudaFuncSetAttribute(order_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kSmallSmem)) != cudaSuccess)
            return e;
        order_small_kernel<<<1, kSmallThreads, kSmallSmem, s>>>(a.depths, a.tiles_per_gauss, (int)E, w.ids[1],
                                                                w.chunks);
        note_launches(1);
    } else {
        constexpr size_t smem = sort_pass_smem<uint32_t>();
        if ((e = cudaFuncSetAttribute(order_pass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) !=
            cudaSuccess)
            return e;
        const int64_t tiles = (E + kSortTile - 1) / kSortTile;
        if (lost) set_u32_kernel<<<1, 1, 0, s>>>(w.counter, 1u);
        for (int p = 0; p < kDepthPasses; ++p)
            order_pass_kernel<<<(unsigned)(tiles - (lost && p == 0)), kSortThreads, smem, s>>>(
                a.depths, w.keys[(p + 1) & 1], w.ids[(p + 1) & 1], w.keys[p & 1], w.ids[p & 1], E, p,
                w.hist + p * kRadix, w.status + (size_t)p * tiles * kRadix, w.counter + p, w.counter + kDepthPasses);
        order_sums_kernel<<<(unsigned)chunks, 256, 0, s>>>(w.ids[1], a.tiles_per_gauss, E, w.chunks);
        order_scan_kernel<<<1, 1024, 0, s>>>(w.chunks, chunks);
        note_launches(kDepthPasses + 2);
    }
    return cudaGetLastError();
}

// Scratch of the list stage: pairs of (camera | tile) key and entry.
struct ListWorkspace {
    uint32_t* hist;     // [4][256]  (zeroed, with all up to `status` inclusive)
    uint32_t* counter;  // [4] tiles taken, then the error flag
    uint32_t* status;   // [passes][tiles][256]
    uint32_t *keys[2], *ids[2];
    size_t zeroed, bytes;
};
inline ListWorkspace carve_list_workspace(void* base, int64_t n, int passes) {
    ListWorkspace w;
    char* p = static_cast<char*>(base);
    size_t off = 0;
    auto take = [&](size_t k) {
        char* q = p + off;
        off += align256(k);
        return q;
    };
    const int64_t tiles = (n + kSortTile - 1) / kSortTile;
    w.hist = reinterpret_cast<uint32_t*>(take(4 * 4 * kRadix));
    w.counter = reinterpret_cast<uint32_t*>(take(4 * 5));
    w.status = reinterpret_cast<uint32_t*>(take(4 * (size_t)passes * tiles * kRadix));
    w.zeroed = off;
    for (int i = 0; i < 2; ++i) w.keys[i] = reinterpret_cast<uint32_t*>(take(4 * (size_t)n));
    for (int i = 0; i < 2; ++i) w.ids[i] = reinterpret_cast<uint32_t*>(take(4 * (size_t)n));
    w.bytes = off;
    return w;
}
// Passes over `key_bits` bits, each of the same number of bits (fewer digits: longer runs to write).
inline int list_passes(int key_bits) { return (key_bits + 7) / 8; }
inline int list_pass_bits(int key_bits) { return (key_bits + list_passes(key_bits) - 1) / list_passes(key_bits); }
size_t isect_lists_workspace_bytes(int64_t n, int key_bits) {
    return carve_list_workspace(nullptr, n, list_passes(key_bits)).bytes;
}

// Writes the intersections in depth order and counts their keys' digits.  A CTA expands 1024 entries: their tile
// boxes go to shared memory, and each thread fills four consecutive list places at a time (one search for the
// first, then stepping), so that the writes are whole vectors whatever the entries' sizes.  flatten_ids gets an entry
// in every place beforehand, so that whoever reads the lists of a sort that gave up stays within the entries.
__global__ void __launch_bounds__(256) isect_expand_kernel(tg_isect_args a, const uint32_t* __restrict__ order,
                                                           const int64_t* __restrict__ chunks, int64_t limit,
                                                           int tile_bits, int passes, int pass_bits,
                                                           uint32_t* __restrict__ keys, uint32_t* __restrict__ ids,
                                                           uint32_t* hist) {
    __shared__ uint32_t s_hist[4 * kRadix];
    __shared__ uint32_t s_off[kOrderChunk + 1];  // places before each entry
    __shared__ uint32_t s_id[kOrderChunk], s_first[kOrderChunk], s_width[kOrderChunk], s_row[kOrderChunk],
        s_high[kOrderChunk];  // s_high: the key's camera bits, or all ones (a negative depth's sign extension)
    __shared__ uint32_t s_warp[8];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < 4 * kRadix; i += 256) s_hist[i] = 0;
    const int64_t first = (int64_t)blockIdx.x * kOrderChunk;
    uint32_t cnt[4], sum = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // thread t owns entries 4t .. 4t+3 of the chunk
        const int64_t k = first + tid * 4 + i;
        const int slot = tid * 4 + i;
        cnt[i] = 0;
        if (k < a.n_elems) {
            const uint32_t e = order[k];
            const int32_t r = e < (uint32_t)a.n_elems ? a.radii[e] : 0;
            uint32_t tw, th;
            if (r > 0 && camera_grid(a, e, tw, th)) {
                const float2 m = reinterpret_cast<const float2*>(a.means2d)[e];
                uint32_t x0, y0, x1, y1;
                tile_box(m.x, m.y, r, a.tile_size, tw, th, x0, y0, x1, y1);
                cnt[i] = (y1 - y0) * (x1 - x0);
                const int64_t cid = a.camera_ids ? a.camera_ids[e] : (int64_t)e / a.N;
                s_id[slot] = e;
                s_first[slot] = y0 * tw + x0;
                s_width[slot] = x1 - x0;
                s_row[slot] = tw;
                s_high[slot] = (__float_as_uint(a.depths[e]) >> 31) ? 0xffffffffu : (uint32_t)(cid << tile_bits);
            }
        }
        sum += cnt[i];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t run = incl - sum;
    for (int w = 0; w < warp; ++w) run += s_warp[w];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        s_off[tid * 4 + i] = run;
        run += cnt[i];
    }
    if (tid == 255) s_off[kOrderChunk] = run;
    __syncthreads();
    const int64_t base = chunks[blockIdx.x];
    const int64_t end = min(base + (int64_t)s_off[kOrderChunk], limit);
    const uint32_t digit_mask = (1u << pass_bits) - 1u;
    const bool whole = (reinterpret_cast<uintptr_t>(a.flatten_ids) & 15) == 0;
    for (int64_t p4 = (base >> 2) + tid; p4 * 4 < end; p4 += 256) {  // four places from 4 * p4 on
        const int64_t lo = max(p4 * 4, base), hi = min(p4 * 4 + 4, end);
        uint32_t rel = (uint32_t)(lo - base);
        int slot = 0;  // last entry whose places start at or before rel
#pragma unroll
        for (int step = kOrderChunk / 2; step > 0; step >>= 1)
            if (s_off[slot + step] <= rel) slot += step;
        uint32_t k = rel - s_off[slot];
        uint32_t y = k / s_width[slot], x = k - y * s_width[slot];
        uint32_t key[4], id[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int64_t pos = p4 * 4 + q;
            if (pos < lo || pos >= hi) continue;
            key[q] = s_high[slot] | (s_first[slot] + y * s_row[slot] + x);
            id[q] = s_id[slot];
            for (int p = 0; p < passes; ++p)
                atomicAdd(&s_hist[p * kRadix + ((key[q] >> (p * pass_bits)) & digit_mask)], 1u);
            ++rel;
            if (++x == s_width[slot]) {
                x = 0;
                ++y;
            }
            if (pos + 1 < hi && rel == s_off[slot + 1]) {
                do ++slot; while (slot + 1 < kOrderChunk && s_off[slot + 1] == rel);  // (entries without places)
                x = y = 0;
            }
        }
        if (hi - lo == 4) {
            reinterpret_cast<uint4*>(keys)[p4] = make_uint4(key[0], key[1], key[2], key[3]);
            reinterpret_cast<uint4*>(ids)[p4] = make_uint4(id[0], id[1], id[2], id[3]);
        }
        if (hi - lo == 4 && whole) {
            reinterpret_cast<int4*>(a.flatten_ids)[p4] = make_int4(0, 0, 0, 0);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int64_t pos = p4 * 4 + q;
                if (pos >= lo && pos < hi) {
                    keys[pos] = key[q];
                    ids[pos] = id[q];
                    a.flatten_ids[pos] = 0;
                }
            }
        }
    }
    if (blockIdx.x == gridDim.x - 1) {  // an entry sort that gave up can leave fewer intersections than were counted
        const int64_t counted = a.overflow ? min(*a.n_isects, limit) : limit;
        for (int64_t pos = end + tid; pos < counted; pos += 256) {
            keys[pos] = ids[pos] = 0xffffffffu;
            a.flatten_ids[pos] = 0;
        }
    }
    __syncthreads();
    for (int i = tid; i < passes * kRadix; i += 256)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
    if (a.overflow && tid == 0 && base + (int64_t)s_off[kOrderChunk] > limit) atomicOr(a.overflow, 1u);
}

// Capacity mode: the places past the valid count get the largest key (they sort last) and no entry.
__global__ void __launch_bounds__(256) isect_expand_pad_kernel(const int64_t* n_dev, int64_t capacity, uint32_t pad_key,
                                                               int passes, int pass_bits, uint32_t* keys, uint32_t* ids,
                                                               int32_t* flatten_ids, uint32_t* hist) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, n = min(max(*n_dev, (int64_t)0), capacity);
    if (i == 0 && n < capacity)
        for (int p = 0; p < passes; ++p)
            atomicAdd(&hist[p * kRadix + ((pad_key >> (p * pass_bits)) & ((1u << pass_bits) - 1u))],
                      (uint32_t)(capacity - n));
    if (i < n || i >= capacity) return;
    keys[i] = pad_key;
    ids[i] = 0xffffffffu;
    flatten_ids[i] = 0;
}

// A capacity of zero intersections: any at all are too many.
__global__ void overflow_if_any_kernel(const int64_t* n_dev, uint32_t* overflow) {
    if (*n_dev > 0) atomicOr(overflow, 1u);
}

// One pass over the (camera, tile) keys; the last writes the 64-bit keys and the entries.
template <bool kLast>
__global__ void __launch_bounds__(kSortThreads, 4) list_pass_kernel(const uint32_t* __restrict__ keys_in,
                                                                 const uint32_t* __restrict__ ids_in,
                                                                 uint32_t* __restrict__ keys_out,
                                                                 uint32_t* __restrict__ ids_out,
                                                                 const float* __restrict__ depths, uint32_t n_elems,
                                                                 int64_t* __restrict__ isect_ids,
                                                                 int32_t* __restrict__ flatten_ids, int64_t n,
                                                                 int shift, int bits, const uint32_t* hist,
                                                                 uint32_t* status, uint32_t* counter, uint32_t* error) {
    sort_pass<uint32_t>(
        [&](int64_t i, uint32_t& k, uint32_t& v) {
            k = keys_in[i];
            v = ids_in[i];
        },
        [&](int64_t i, uint32_t k, uint32_t v) {
            if constexpr (kLast) {
                const bool pad = v >= n_elems;  // (padding has the id 0xffffffff)
                const uint32_t low = pad ? 0xffffffffu : __float_as_uint(__ldg(depths + v));
                isect_ids[i] = (int64_t)(((uint64_t)k << 32) | low);
                flatten_ids[i] = pad ? 0 : (int32_t)v;
            } else {
                keys_out[i] = k;
                ids_out[i] = v;
            }
        },
        n, shift, bits, hist, status, counter, error);
}

// lost: the sort whose first tile nobody takes, as in sort_lookback_selftest (1: the entries', 2: the lists', 0: none).
cudaError_t launch_isect_lists(const tg_isect_args& a, void* order_ws, int64_t n, int tile_bits, int key_bits, void* ws,
                               int lost, cudaStream_t s) {
    const int64_t E = a.n_elems;
    if (n == 0) {
        if (!a.overflow) return cudaSuccess;
        overflow_if_any_kernel<<<1, 1, 0, s>>>(a.n_isects, a.overflow);
        note_launches(1);
        return cudaGetLastError();
    }
    const int passes = list_passes(key_bits), pass_bits = list_pass_bits(key_bits);
    const OrderWorkspace o = carve_order_workspace(order_ws, E);
    const ListWorkspace w = carve_list_workspace(ws, n, passes);
    cudaError_t e = cudaMemsetAsync(ws, 0, w.zeroed, s);
    if (e != cudaSuccess) return e;
    if (E > 0) {
        if ((e = launch_entry_sort(a, o, lost == 1, s)) != cudaSuccess) return e;
        isect_expand_kernel<<<(unsigned)((E + kOrderChunk - 1) / kOrderChunk), 256, 0, s>>>(
            a, o.ids[1], o.chunks, n, tile_bits, passes, pass_bits, w.keys[0], w.ids[0], w.hist);
        note_launches(1);
    }
    if (a.overflow) {
        const uint32_t pad = key_bits >= 32 ? 0xffffffffu : (1u << key_bits) - 1u;
        isect_expand_pad_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a.n_isects, n, pad, passes, pass_bits,
                                                                           w.keys[0], w.ids[0], a.flatten_ids, w.hist);
        note_launches(1);
    }
    constexpr size_t smem = sort_pass_smem<uint32_t>();
    if ((e = cudaFuncSetAttribute(list_pass_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) !=
            cudaSuccess ||
        (e = cudaFuncSetAttribute(list_pass_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) !=
            cudaSuccess)
        return e;
    const int64_t tiles = (n + kSortTile - 1) / kSortTile;
    if (lost == 2) set_u32_kernel<<<1, 1, 0, s>>>(w.counter, 1u);
    for (int p = 0; p < passes; ++p) {
        const int shift = p * pass_bits, bits = std::min(pass_bits, key_bits - shift);
        const auto fn = p == passes - 1 ? list_pass_kernel<true> : list_pass_kernel<false>;
        fn<<<(unsigned)(tiles - (lost == 2 && p == 0)), kSortThreads, smem, s>>>(w.keys[p & 1], w.ids[p & 1], w.keys[(p + 1) & 1],
                                                       w.ids[(p + 1) & 1], a.depths, (uint32_t)E, a.isect_ids, a.flatten_ids, n,
                                                       shift, bits, w.hist + p * kRadix,
                                                       w.status + (size_t)p * tiles * kRadix, w.counter + p,
                                                       w.counter + 4);
    }
    note_launches(passes);
    return cudaGetLastError();
}

// Where the host finds whether a look-back of the call's sorts gave up (NULL: the size takes a sort without any).
const uint32_t* entry_sort_error(const void* order_ws, int64_t E) {
    return E > kSmallSort ? carve_order_workspace(const_cast<void*>(order_ws), E).counter + kDepthPasses : nullptr;
}
const uint32_t* list_sort_error(const void* list_ws, int64_t n, int key_bits) {
    return n > 0 ? carve_list_workspace(const_cast<void*>(list_ws), n, list_passes(key_bits)).counter + 4 : nullptr;
}
const uint32_t* tile_order_error(const void* ws, int64_t n_tiles) {
    return n_tiles > kSmallSort ? carve_list_workspace(const_cast<void*>(ws), n_tiles, 4).counter + 4 : nullptr;
}

// ------------------------------------------------------------------ tile order
// Tiles by descending list length (stable): keys bound - length, bound >= every length.
__device__ __forceinline__ uint32_t tile_key(const int32_t* __restrict__ offsets, int64_t t, int64_t n_tiles,
                                             int64_t n_isects, const int64_t* n_dev, uint32_t bound) {
    const int64_t end = t + 1 < n_tiles ? (int64_t)offsets[t + 1] : (n_dev ? *n_dev : n_isects);
    const int64_t c = end - (int64_t)offsets[t];
    return bound - (uint32_t)min(max(c, (int64_t)0), (int64_t)bound);
}

__global__ void __launch_bounds__(kSmallThreads) tile_order_small_kernel(const int32_t* offsets, int n_tiles,
                                                                         int64_t n_isects, const int64_t* n_dev,
                                                                         uint32_t bound, int end_bit, int32_t* order) {
    uint32_t *s_keys, *s_idx;
    sort_small([&](int i, bool&) { return tile_key(offsets, i, n_tiles, n_isects, n_dev, bound); }, n_tiles, end_bit,
               s_keys, s_idx);
    for (int i = threadIdx.x; i < n_tiles; i += kSmallThreads) order[i] = (int32_t)s_idx[i];
}

__global__ void __launch_bounds__(256) tile_order_count_kernel(const int32_t* offsets, int64_t n_tiles,
                                                               int64_t n_isects, const int64_t* n_dev, uint32_t bound,
                                                               int passes, uint32_t* hist) {
    __shared__ uint32_t s_hist[4 * kRadix];
    for (int i = threadIdx.x; i < 4 * kRadix; i += 256) s_hist[i] = 0;
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * 256;
    for (int64_t b = (int64_t)blockIdx.x * 256; b < n_tiles; b += stride) {  // uniform over the CTA
        const int64_t t = b + threadIdx.x;
        const bool in = t < n_tiles;
        const uint32_t k = in ? tile_key(offsets, t, n_tiles, n_isects, n_dev, bound) : 0u;
        for (int p = 0; p < passes; ++p) count_digit(s_hist + p * kRadix, (k >> (8 * p)) & 0xffu, in);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * kRadix; i += 256)
        if (s_hist[i]) atomicAdd(&hist[i], s_hist[i]);
}

__global__ void __launch_bounds__(kSortThreads, 4) tile_order_pass_kernel(
    const int32_t* __restrict__ offsets, int64_t n_isects, const int64_t* n_dev, uint32_t bound,
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ ids_in, uint32_t* __restrict__ keys_out,
    uint32_t* __restrict__ ids_out, int64_t n, int pass, int bits, const uint32_t* hist, uint32_t* status,
    uint32_t* counter, uint32_t* error) {
    sort_pass<uint32_t>(
        [&](int64_t i, uint32_t& k, uint32_t& v) {
            k = pass == 0 ? tile_key(offsets, i, n, n_isects, n_dev, bound) : keys_in[i];
            v = pass == 0 ? (uint32_t)i : ids_in[i];
        },
        [&](int64_t i, uint32_t k, uint32_t v) {
            keys_out[i] = k;
            ids_out[i] = v;
        },
        n, 8 * pass, bits, hist, status, counter, error);
}

// Above kSmallSort tiles: the list stage's scratch serves (its pairs are of the same kind).
size_t tile_order_workspace_bytes(int64_t n_tiles) {
    return n_tiles <= kSmallSort ? 256 : carve_list_workspace(nullptr, n_tiles, 4).bytes;
}

// lost: nobody takes the first tile of the first pass, as in sort_lookback_selftest.
cudaError_t launch_tile_order(const int32_t* offsets, int64_t n_tiles, int64_t n_isects, const int64_t* n_dev,
                              int32_t* order, void* ws, bool lost, cudaStream_t s) {
    if (n_tiles == 0) return cudaSuccess;
    const uint32_t bound = (uint32_t)std::min<int64_t>(std::max<int64_t>(n_isects, 1), 0x7fffffff);
    int end_bit = 0;
    for (uint32_t b = bound; b; b >>= 1) ++end_bit;
    cudaError_t e;
    if (n_tiles <= kSmallSort) {
        if ((e = cudaFuncSetAttribute(tile_order_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kSmallSmem)) != cudaSuccess)
            return e;
        tile_order_small_kernel<<<1, kSmallThreads, kSmallSmem, s>>>(offsets, (int)n_tiles, n_isects, n_dev, bound,
                                                                     end_bit, order);
        note_launches(1);
        return cudaGetLastError();
    }
    const int passes = (end_bit + 7) / 8;
    const ListWorkspace w = carve_list_workspace(ws, n_tiles, 4);
    if ((e = cudaMemsetAsync(ws, 0, w.zeroed, s)) != cudaSuccess) return e;
    const int64_t tiles = (n_tiles + kSortTile - 1) / kSortTile;
    tile_order_count_kernel<<<(unsigned)std::min<int64_t>((n_tiles + 1023) / 1024, kNumSMs * 4), 256, 0, s>>>(
        offsets, n_tiles, n_isects, n_dev, bound, passes, w.hist);
    constexpr size_t smem = sort_pass_smem<uint32_t>();
    if ((e = cudaFuncSetAttribute(tile_order_pass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) !=
        cudaSuccess)
        return e;
    if (lost) set_u32_kernel<<<1, 1, 0, s>>>(w.counter, 1u);
    for (int p = 0; p < passes; ++p) {
        uint32_t* out = p == passes - 1 ? reinterpret_cast<uint32_t*>(order) : w.ids[(p + 1) & 1];
        tile_order_pass_kernel<<<(unsigned)(tiles - (lost && p == 0)), kSortThreads, smem, s>>>(
            offsets, n_isects, n_dev, bound, w.keys[p & 1], w.ids[p & 1], w.keys[(p + 1) & 1], out, n_tiles, p,
            std::min(8, end_bit - 8 * p), w.hist + p * kRadix, w.status + (size_t)p * tiles * kRadix, w.counter + p,
            w.counter + 4);
    }
    note_launches(1 + passes);
    return cudaGetLastError();
}

}  // namespace tg
