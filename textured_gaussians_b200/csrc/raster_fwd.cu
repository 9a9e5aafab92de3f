// Textured / plain 2DGS compositor, forward, for sm_100a.
//
// A square is an 8x8 or 16x16 tile, or a quarter of a 32x32 one.  One CTA per square, one thread per pixel, walks the
// tile's depth-sorted splats front to back in batches of `batch_depth` (tile_size^2 by default) staged in shared
// memory: 80 contiguous bytes a splat, packed once per call where the lists repeat the entries often enough
// (tg_raster_fwd_args.entry_records).  A warp is four groups of 4x2 pixels; staging leaves each group a bit list of
// the batch's splats whose bounds meet it (group_mask), and the four groups walk their own lists, so one warp
// iteration works on four splats.  A warp per 8x4 block and a box test took 1.13 iterations a listed splat on the
// 1M-splat mixture, the groups take 0.49 (four 1600x1200 views: forward 9.2 -> 6.7 ms).  What bounds it: issue (58-78 %
// of the cycles from 100,000 splats on, 44-50 % of the warps resident at 64 registers) and the reads it waits for between.
// Each pixel samples its splat's RGBA texture with one 16-byte (FP32), 8-byte (BF16/FP16) or 4-byte (FP8) load per
// bilinear tap and reuses the four taps for the alpha scale and every colour channel.  Lists end early for saturated
// pixels, and a square at the next batch boundary once all are.  The contribution statistics are reduced per group,
// then summed in shared memory before one global atomic per (splat, square).  With contrib_masks every pixel's
// composited splats are left as bits for the adjoint.
//
// Semantics: textured_gaussians/cuda/csrc/rasterize_to_pixels_textured_
// gaussians_2dgs_fwd.cu:73-445 and rasterize_to_pixels_2dgs_fwd.cu (plain),
// with the texture / statistics row of element e taken as e % N (dense) or
// gaussian_ids[e] (packed) instead of the reference's out-of-range e.
#include "raster_common.cuh"

namespace tg {

// Resident CTAs per SM the register allocation targets.
#ifndef TG_FWD_MIN_CTAS
#define TG_FWD_MIN_CTAS 4
#endif

// Staged splats: an EntryRecord each (with a fifth colour channel apart), the texture scale (FP8 only), the
// contribution statistics and the groups' list words.  The record's five vectors lie together, not in an array each:
// a pair's reads share one address (untextured forward of 150,000 splats at 800x800: 330 -> 302 us, textured 1 %).
template <int D, class Tex>
struct FwdSmem {
    static constexpr bool kScale = Tex::kFormat == TG_TEX_FP8_E4M3;
    float4* rec;  // [bs][5] EntryRecords: one address a splat, and an odd number of vectors apart (no bank conflicts)
    float *col5, *scale;
    uint32_t *csum, *ccnt, *words;
    float4* extra;  // what follows (anisotropic_bilinear's step)
    __device__ __forceinline__ FwdSmem(float4* base, int bs, int side) {
        rec = base;
        csum = reinterpret_cast<uint32_t*>(rec + 5 * bs);
        ccnt = csum + bs;
        words = ccnt + bs;
        scale = reinterpret_cast<float*>(words + (side * side / kGroupLanes) * (bs / 32));
        col5 = scale + (kScale ? bs : 0);
        extra = reinterpret_cast<float4*>(col5 + (D == 5 ? bs : 0));
    }
    static size_t bytes(int bs, int side) {
        return (size_t)bs * (5 * sizeof(float4) + 8 + (kScale ? 4 : 0) + (D == 5 ? 4 : 0)) +
               (size_t)(side * side / kGroupLanes) * (bs / 32) * 4;
    }
};

// The threads that composite one square: a whole CTA, or 64 of its threads with a barrier of their own.
struct WholeCta {
    __device__ __forceinline__ int tid() const { return threadIdx.x; }
    __device__ __forceinline__ int size() const { return blockDim.x; }
    __device__ __forceinline__ void sync() const { __syncthreads(); }
    __device__ __forceinline__ int count(bool p) const { return __syncthreads_count(p); }
};
struct QuarterCta {
    __device__ __forceinline__ int tid() const { return threadIdx.x & 63; }
    __device__ __forceinline__ int size() const { return 64; }
    __device__ __forceinline__ int barrier() const { return 1 + (threadIdx.x >> 6); }
    __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, 64;" ::"r"(barrier()) : "memory"); }
    __device__ __forceinline__ int count(bool p) const {
        int n;
        asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %1, 0;\n bar.red.popc.u32 %0, %2, 64, p;\n}"
                     : "=r"(n)
                     : "r"((int)p), "r"(barrier())
                     : "memory");
        return n;
    }
};

// One square (sub-square `sub` of tile work item `item`) of the forward; every early return is uniform over its
// threads.  smem4: its part of the CTA's shared memory.
template <int D, class Tex, class Filt, class Crew>
__device__ __forceinline__ void fwd_square(const tg_raster_fwd_args& a, const int bs, const int64_t item, const int sub,
                                           const int side, float4* smem4, const Crew crew) {
    constexpr bool kTextured = Tex::kFormat != TG_TEX_NONE;
    constexpr unsigned kFull = 0xffffffffu;
    const int nt = crew.size();  // one thread per pixel of the square; bs = splats staged per batch
    const int ts = a.tile_size;
    const FwdSmem<D, Tex> S(smem4, bs, side);
    const int tr = crew.tid(), lane = tr & 31;
    float4* s_aniso = Filt::kAniso ? S.extra + (tr >> 5) * kAnisoWarpF4 : nullptr;

    const TileWork tc = tile_work(a, item);
    if (!tc.valid) return;
    const int per_row = ts / side;
    const int X0 = tc.tx * ts + (sub % per_row) * side, Y0 = tc.ty * ts + (sub / per_row) * side;
    const PixelSlot ps = pixel_slot(tr, side);
    const int j = X0 + ps.x, i = Y0 + ps.y;
    const int64_t pix = pixel_index(tc, i, j);
    const bool inside = pix >= 0;
    const float px = (float)j + 0.5f, py = (float)i + 0.5f;
    bool done = !inside;

    if (a.masks != nullptr && !a.masks[tc.t]) {
        if (!inside) return;
#pragma unroll
        for (int k = 0; k < D; ++k) a.out_colors[pix * D + k] = a.backgrounds ? a.backgrounds[tc.c * D + k] : 0.f;
        a.out_alphas[pix] = 0.f;
        a.out_normals[pix * 3] = a.out_normals[pix * 3 + 1] = a.out_normals[pix * 3 + 2] = 0.f;
        a.out_distort[pix] = 0.f;
        a.out_median[pix] = 0.f;
        a.last_ids[pix] = 0;
        a.median_ids[pix] = 0;
        return;
    }

    const int32_t range_start = tc.range_start;
    const int32_t range_end = tc.range_end;
    const int num_batches = (range_end - range_start + bs - 1) / bs;
    const int64_t tex_stride = (int64_t)a.tex_ry * a.tex_rx;
    const int mip_clen = Filt::kMip ? ((1 << (2 * a.mip_levels)) - 1) / 3 : 0;
    const int n_words = bs >> 5;
    const uint32_t* words = S.words + (size_t)(tr >> 3) * n_words;  // the lane's group's list

    float T = 1.f, pix_out[D], nrm_out[3] = {0.f, 0.f, 0.f}, distort = 0.f, accum_vis_depth = 0.f, median_depth = 0.f;
    int32_t cur_idx = 0, median_idx = 0;
    int32_t rec_n = 0;  // anisotropic_bilinear: contributors whose footprint integral was recorded (or counted)
    const bool records = Filt::kAniso && a.aniso_records != nullptr;
#pragma unroll
    for (int k = 0; k < D; ++k) pix_out[k] = 0.f;
    for (int slot = tr; slot < bs; slot += nt) S.csum[slot] = S.ccnt[slot] = 0u;

    // where the adjoint looks for this pixel's bits: its squares are square_side(ts) wide
    const int mask_side = square_side(ts), mask_sub = ((j - tc.tx * ts) / mask_side) + 2 * ((i - tc.ty * ts) / mask_side);
    const int mask_slot = mask_sub * mask_side * mask_side +
                          slot_of_pixel((j - tc.tx * ts) % mask_side, (i - tc.ty * ts) % mask_side, mask_side);

    // adds a staged slot's statistics to its Gaussian's (by the thread that stages the slot)
    auto flush_stats = [&](int slot) {
        const uint32_t c = S.ccnt[slot];
        if (c == 0u) return;
        const int row = __float_as_int(S.rec[5 * slot + 4].w);
        atomicAdd(a.contrib_sum + row, (float)S.csum[slot] * (1.f / 16777216.f));
        atomicAdd(a.contrib_count + row, (float)c);
        S.csum[slot] = S.ccnt[slot] = 0u;
    };

    for (int b = 0; b < num_batches; ++b) {
        if (crew.count(done) >= nt) break;
        const int32_t batch_start = range_start + bs * b;
        for (int slot = tr; slot < bs; slot += nt) {  // (whole warps: bs and nt are multiples of 32)
            flush_stats(slot);
            const int32_t idx = batch_start + slot;
            uint32_t reach = 0u;
            if (idx < range_end) {
                const int32_t g = a.flatten_ids[idx];
                const EntryRecord r = load_entry<D, true>(a, g);
                r.store(S.rec + 5 * slot);
                if constexpr (D == 5) S.col5[slot] = a.colors[(int64_t)g * D + 4];
                if constexpr (FwdSmem<D, Tex>::kScale) S.scale[slot] = a.tex_scales[__float_as_int(r.nrm.w)];
                reach = group_mask(make_float4(r.m0.w, r.m1.w, r.m2.w, 1.f), r.m0, r.m1, r.m2, kTextured, a.range_x,
                                   a.range_y, a.g_weight, !Filt::kAniso, X0, Y0, side);
            }
            store_group_words(reach, S.words, n_words, slot >> 5, side);
        }
        crew.sync();
        int w = 0;
        uint32_t bits = words[0], own = 0u;  // own: this pixel's contributors among word w's splats
        // the contributors' bits of this batch's words, for the adjoint
        uint32_t* bits_out = a.contrib_masks != nullptr
                                 ? a.contrib_masks + ((int64_t)tc.t + (range_start >> 5) + b * n_words) *
                                                         (int64_t)(ts * ts) + mask_slot
                                 : nullptr;
        const int live_words = min(n_words, (range_end - batch_start + 31) >> 5);
        for (;;) {
            while (bits == 0u && w + 1 < n_words) {
                if (bits_out != nullptr && w < live_words) bits_out[(int64_t)w * (ts * ts)] = own;
                own = 0u;
                bits = words[++w];
            }
            const bool act = bits != 0u && !done;
            if (!__any_sync(kFull, act)) break;  // every list used up, or its pixels done
            const int t = w * 32 + (bits != 0u ? __ffs(bits) - 1 : 0);
            bits &= bits - 1u;
            uint32_t stat = 0u;  // the pair's alpha in 2^-24 fixed point
            if (Filt::kAniso || act) {
                const float4* rec = S.rec + 5 * t;
                const float4 m0 = rec[0], m1 = rec[1], m2 = rec[2], nn = rec[4];
                const int row = __float_as_int(nn.w);
                const int64_t tex_base = (int64_t)row * tex_stride;
                const float4 xyo = make_float4(m0.w, m1.w, m2.w, FwdSmem<D, Tex>::kScale ? S.scale[t] : 1.f);
                PairOf<Filt> e;
                if constexpr (Filt::kAniso) {  // every lane takes part: the warp integrates footprints together
                    eval_aniso_coop<Tex>(e, act, px, py, xyo, m0, m1, m2, a.textures, row, a.tex_rx, a.tex_ry,
                                         a.range_x, a.range_y, a.g_weight, kFull,
                                         reinterpret_cast<const float4*>(a.aniso_prefix), s_aniso);
                } else {
                    eval_pair<Tex, Filt>(e, px, py, xyo, m0, m1, m2, a.textures, tex_base, a.tex_rx, a.tex_ry, a.range_x,
                                         a.range_y, a.g_weight,
                                         MipSrc{a.tex_coarse, (int64_t)row * mip_clen, mip_clen, a.mip_levels});
                }
                if (act && e.valid) {
                    const float next_T = T * (1.f - e.alpha);
                    if (next_T <= 1e-4f) {
                        done = true;
                    } else {
                        const float vis = e.alpha * T;
                        const float4 c4 = rec[3];
                        const float c5 = D == 5 ? S.col5[t] : 0.f;
                        float depth = 0.f;
#pragma unroll
                        for (int k = 0; k < D; ++k) {
                            const float ck = k < 4 ? f4get(c4, k) : c5;
                            pix_out[k] += (ck + (kTextured ? tex_color(e, k) : 0.f)) * vis;
                            if (k == D - 1) depth = ck;
                        }
                        nrm_out[0] += nn.x * vis;
                        nrm_out[1] += nn.y * vis;
                        nrm_out[2] += nn.z * vis;
                        distort += 2.f * (vis * depth * (1.f - T) - vis * accum_vis_depth);
                        accum_vis_depth += vis * depth;
                        if (T > 0.5f) {
                            median_depth = depth;
                            median_idx = batch_start + t;
                        }
                        cur_idx = batch_start + t;
                        if constexpr (Filt::kAniso)
                            if (records) {
                                if (rec_n < a.aniso_record_cap)
                                    reinterpret_cast<float4*>(a.aniso_records)[pix * a.aniso_record_cap + rec_n] =
                                        e.tsum;
                                ++rec_n;
                            }
                        own |= 1u << (t & 31);
                        T = next_T;
                        // counted in the top four bits: eight lanes' alphas (each < 1) fit below them
                        if (e.alpha > a.contrib_threshold) stat = __float2uint_rn(e.alpha * 16777216.f) | (1u << 28);
                    }
                }
            }
            // the group's sum of alphas and count, into the slot's integer statistics (32-bit integer adds to shared
            // memory are single instructions; a square's 256 alphas below 0.999 fit in 32 bits)
            stat += __shfl_xor_sync(kFull, stat, 4);
            stat += __shfl_xor_sync(kFull, stat, 2);
            stat += __shfl_xor_sync(kFull, stat, 1);
            if ((lane & 7) == 0 && stat != 0u) {
                atomicAdd(S.csum + t, stat & 0x0fffffffu);
                atomicAdd(S.ccnt + t, stat >> 28);
            }
        }
        if (bits_out != nullptr)
            for (; w < live_words; ++w, own = 0u) bits_out[(int64_t)w * (ts * ts)] = own;
        if (a.t_checkpoints != nullptr)  // every pixel's transmittance at the end of this batch
            a.t_checkpoints[((int64_t)tc.t + range_start / bs + b) * (int64_t)(ts * ts) +
                            (i - tc.ty * ts) * ts + (j - tc.tx * ts)] = T;
    }
    crew.sync();
    for (int slot = tr; slot < bs; slot += nt) flush_stats(slot);
    if (!inside) return;
    a.out_alphas[pix] = 1.f - T;
#pragma unroll
    for (int k = 0; k < D; ++k)
        a.out_colors[pix * D + k] = a.backgrounds ? pix_out[k] + T * a.backgrounds[tc.c * D + k] : pix_out[k];
    a.out_normals[pix * 3] = nrm_out[0];
    a.out_normals[pix * 3 + 1] = nrm_out[1];
    a.out_normals[pix * 3 + 2] = nrm_out[2];
    a.last_ids[pix] = cur_idx;
    a.out_distort[pix] = distort;
    a.out_median[pix] = median_depth;
    a.median_ids[pix] = median_idx;
    if (records) a.aniso_record_count[pix] = rec_n;
}

// CTA per work item, or (work_queue != NULL) a persistent grid whose CTAs take
// items from the queue counter until none is left.
template <int D, class Tex, bool kPersistent, class Filt = FiltBilinear>
__global__ void __launch_bounds__(256, TG_FWD_MIN_CTAS) raster_fwd_kernel(const tg_raster_fwd_args a,
                                                                                    const int bs,
                                                                                    const int64_t n_items) {
    extern __shared__ float4 smem4[];
    const int side = square_side(a.tile_size), subs = squares_per_tile(a.tile_size);
    if constexpr (!kPersistent) {
        const int item = (int)blockIdx.x;
        fwd_square<D, Tex, Filt>(a, bs, subs == 1 ? item : item / subs, subs == 1 ? 0 : item % subs, side, smem4,
                                 WholeCta{});
        return;
    }
    else {
        __shared__ int64_t s_item;
        for (;;) {
            if (threadIdx.x == 0) s_item = (int64_t)atomicAdd(a.work_queue, 1u);
            __syncthreads();  // also: every thread is done with the previous item's shared memory
            const int64_t item = s_item;
            __syncthreads();  // s_item read by all before it is rewritten
            if (item >= n_items) return;
            fwd_square<D, Tex, Filt>(a, bs, item / subs, (int)(item % subs), side, smem4, WholeCta{});
        }
    }
}

// ---------------------------------------------------------------- anisotropic_bilinear
// Integrating a footprint costs a walk along its boundary, two orders of magnitude more than blending the result,
// and does not depend on what lies in front.  The longest tiles, first in the work order, take a CTA of eight warps
// for each 8x8 square and each step of listed splats in two halves: all warps evaluate the step's (group, splat)
// items, four at a time, whichever group they belong to, into shared memory; then the pixels' own threads blend them
// in order.  With the pixels' two warps doing both, the longest tile's chain of walks set the kernel's time (7.0 ms
// for 60k splats, 800x600, the SMs busy for half of it at 16 % occupancy; 3.25 ms so).  But the halves wait for one
// another, and where every SM is full anyway that costs: 22.1 against 20.5 ms for 300k splats in two 1600x1200
// views.  So only the first kLongTiles squares are taken so, the others four to a CTA, two warps each; and from
// kFullSquares squares on, or where a batch is too deep for that, all take the other filters' kernel.
constexpr int kFullSquares = 128 * kNumSMs;  // eight times what the device holds at once (no size between the two timed)
constexpr int kLongTiles = 3 * kNumSMs;  // of 1, 3 and 6 per SM (60k splats: 3.96, 3.25, 3.32 ms)
constexpr size_t kMaxSmem = 227 * 1024;  // of a CTA
constexpr int kAnisoWarps = 8;
constexpr int kAnisoThreads = 32 * kAnisoWarps;
constexpr int kAnisoItems = 64;  // 32, 48, 64: 3.63, 3.45, 3.25 ms; more leaves the walk's reads less L1
constexpr int kAnisoSide = 8;
struct AnisoStep {
    float4* sum;     // [items][8] footprint integrals
    float2* aux;     // [items][8] alpha (0: not valid) and 1 / area
    float4* warps;   // per-warp areas of the boundary integration
    uint16_t* item;  // [items] group << 5 | splat
    uint32_t* done;  // [2] the pixels that are finished, a word per blending warp
    __device__ __forceinline__ explicit AnisoStep(float4* base) {
        sum = base;
        aux = reinterpret_cast<float2*>(sum + kAnisoItems * 8);
        warps = reinterpret_cast<float4*>(aux + kAnisoItems * 8);
        item = reinterpret_cast<uint16_t*>(warps + kAnisoWarps * kAnisoWarpF4);
        done = reinterpret_cast<uint32_t*>(item + kAnisoItems);
    }
    static constexpr size_t kBytes = kAnisoItems * (8 * 24 + 2) + kAnisoWarps * kAnisoWarpF4 * 16 + 8;
};

template <int D, class Tex>
__device__ __forceinline__ void aniso_long_square(const tg_raster_fwd_args& a, const int bs, const int64_t item,
                                                  const int sub, float4* smem4) {
    constexpr unsigned kFull = 0xffffffffu;
    const int ts = a.tile_size, per_row = ts / kAnisoSide;
    const FwdSmem<D, Tex> S(smem4, bs, kAnisoSide);
    const AnisoStep A(S.extra);
    const TileWork tc = tile_work(a, item);
    if (!tc.valid) return;  // uniform over the CTA
    const int tr = threadIdx.x, lane = tr & 31, warp = tr >> 5;
    const int X0 = tc.tx * ts + (sub % per_row) * kAnisoSide, Y0 = tc.ty * ts + (sub / per_row) * kAnisoSide;
    // the first two warps own the pixels
    const PixelSlot ps = pixel_slot(tr & 63, kAnisoSide);
    const int j = X0 + ps.x, i = Y0 + ps.y;
    const int64_t pix = tr < 64 ? pixel_index(tc, i, j) : -1;
    const bool inside = pix >= 0;
    bool done = !inside;
    if (a.masks != nullptr && !a.masks[tc.t]) {
        if (!inside) return;
#pragma unroll
        for (int k = 0; k < D; ++k) a.out_colors[pix * D + k] = a.backgrounds ? a.backgrounds[tc.c * D + k] : 0.f;
        a.out_alphas[pix] = 0.f;
        a.out_normals[pix * 3] = a.out_normals[pix * 3 + 1] = a.out_normals[pix * 3 + 2] = 0.f;
        a.out_distort[pix] = 0.f;
        a.out_median[pix] = 0.f;
        a.last_ids[pix] = 0;
        a.median_ids[pix] = 0;
        return;
    }
    const int32_t range_start = tc.range_start, range_end = tc.range_end;
    const int num_batches = (range_end - range_start + bs - 1) / bs;
    const int n_words = bs >> 5;
    float T = 1.f, pix_out[D], nrm_out[3] = {0.f, 0.f, 0.f}, distort = 0.f, accum_vis_depth = 0.f, median_depth = 0.f;
    int32_t cur_idx = 0, median_idx = 0;
    int32_t rec_n = 0;  // contributors whose footprint integral was recorded (or counted)
    uint32_t own = 0u;  // this pixel's contributors among word w's splats
#pragma unroll
    for (int k = 0; k < D; ++k) pix_out[k] = 0.f;
    for (int slot = tr; slot < bs; slot += kAnisoThreads) S.csum[slot] = S.ccnt[slot] = 0u;
    auto flush_stats = [&](int slot) {
        const uint32_t c = S.ccnt[slot];
        if (c == 0u) return;
        const int row = __float_as_int(S.rec[5 * slot + 4].w);
        atomicAdd(a.contrib_sum + row, (float)S.csum[slot] * (1.f / 16777216.f));
        atomicAdd(a.contrib_count + row, (float)c);
        S.csum[slot] = S.ccnt[slot] = 0u;
    };
    const int mask_side = square_side(ts);  // the adjoint's pixel order in contrib_masks
    const int mask_slot = slot_of_pixel(j - tc.tx * ts, i - tc.ty * ts, mask_side);

    for (int b = 0; b < num_batches; ++b) {
        if (__syncthreads_count(done || tr >= 64) >= kAnisoThreads) break;
        const int32_t batch_start = range_start + bs * b;
        own = 0u;
        for (int slot = tr; slot < bs; slot += kAnisoThreads) {  // (whole warps)
            flush_stats(slot);
            const int32_t idx = batch_start + slot;
            uint32_t reach = 0u;
            if (idx < range_end) {
                const EntryRecord r = load_entry<D, true>(a, a.flatten_ids[idx]);
                r.store(S.rec + 5 * slot);
                reach = group_mask(make_float4(r.m0.w, r.m1.w, r.m2.w, 1.f), r.m0, r.m1, r.m2, true, a.range_x, a.range_y,
                                   a.g_weight, false, X0, Y0, kAnisoSide);
            }
            store_group_words(reach, S.words, n_words, slot >> 5, kAnisoSide);
        }
        uint32_t* bits_out = a.contrib_masks != nullptr
                                 ? a.contrib_masks + ((int64_t)tc.t + (range_start >> 5) + b * n_words) *
                                                         (int64_t)(ts * ts) + mask_slot
                                 : nullptr;
        const int live_words = min(n_words, (range_end - batch_start + 31) >> 5);
        // steps of up to kAnisoItems items: splats [t0, t1) of word w
        for (int w = 0, t0 = 0; w < live_words;) {
            if (tr < 64) {
                const unsigned d = __ballot_sync(kFull, done);
                if (lane == 0) A.done[warp] = d;
            }
            __syncthreads();  // the lists, and the previous step's results are read
            // lane = splat: its items, one per group that lists it and has a pixel left
            uint32_t bits_of[8];
            int c = 0;
#pragma unroll
            for (int g = 0; g < 8; ++g) {
                const bool live = ((A.done[g >> 2] >> ((g & 3) * 8)) & 0xffu) != 0xffu;
                bits_of[g] = live ? S.words[g * n_words + w] : 0u;
                c += lane >= t0 ? (bits_of[g] >> lane) & 1u : 0u;
            }
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(kFull, c, o);
                if (lane >= o) c += u;
            }
            const unsigned over = __ballot_sync(kFull, c > kAnisoItems);
            const int t1 = over ? __ffs(over) - 1 : 32;
            const uint32_t window = (t1 == 32 ? ~0u : (1u << t1) - 1u) & (~0u << t0);
            int n_items = 0, first = 0;  // first: of the calling (blending) thread's group
#pragma unroll
            for (int g = 0; g < 8; ++g) {
                bits_of[g] &= window;
                if (g == ((tr >> 3) & 7)) first = n_items;
                if (g % kAnisoWarps == warp && ((bits_of[g] >> lane) & 1u))
                    A.item[n_items + __popc(bits_of[g] & ((1u << lane) - 1u))] = (uint16_t)(g * 32 + lane);
                n_items += __popc(bits_of[g]);
            }
            __syncthreads();
            for (int k0 = warp * 4; k0 < n_items; k0 += kAnisoWarps * 4) {  // uniform over the warp
                const int k = k0 + (lane >> 3);
                const bool listed = k < n_items;
                const int it = listed ? A.item[k] : A.item[k0];
                const int g = it >> 5, t = w * 32 + (it & 31), p = g * 8 + (lane & 7);
                const PixelSlot q = pixel_slot(p, kAnisoSide);
                const bool act = listed && ((A.done[p >> 5] >> (p & 31)) & 1u) == 0u;
                const float4* rec = S.rec + 5 * t;
                const float4 m0 = rec[0], m1 = rec[1], m2 = rec[2];
                PairEvalAniso e;
                eval_aniso_coop<Tex>(e, act, (float)(X0 + q.x) + 0.5f, (float)(Y0 + q.y) + 0.5f,
                                     make_float4(m0.w, m1.w, m2.w, 1.f), m0, m1, m2, a.textures,
                                     __float_as_int(rec[4].w), a.tex_rx, a.tex_ry, a.range_x, a.range_y, a.g_weight,
                                     kFull, reinterpret_cast<const float4*>(a.aniso_prefix),
                                     A.warps + warp * kAnisoWarpF4);
                if (listed) {
                    const bool ok = act && e.valid;
                    A.aux[k * 8 + (lane & 7)] = make_float2(ok ? e.alpha : 0.f, ok ? e.F.iarea : 0.f);
                    if (ok) A.sum[k * 8 + (lane & 7)] = e.tsum;
                }
            }
            __syncthreads();
            if (tr < 64) {
                uint32_t bits = 0u;
#pragma unroll
                for (int g = 0; g < 8; ++g)
                    if (g == (tr >> 3)) bits = bits_of[g];
                int k = first * 8 + (lane & 7);  // the group's next result
                for (; __any_sync(kFull, bits != 0u); k += 8) {
                    const int bit = bits != 0u ? __ffs(bits) - 1 : 0, t = w * 32 + bit;
                    const bool listed = bits != 0u;
                    bits &= bits - 1u;
                    uint32_t stat = 0u;
                    if (listed && !done) {
                        const float2 ax = A.aux[k];
                        if (ax.x > 0.f) {
                            const float alpha = ax.x, next_T = T * (1.f - alpha);
                            if (next_T <= 1e-4f) {
                                done = true;
                            } else {
                                const float4 ts4 = A.sum[k], c4 = S.rec[5 * t + 3], nn = S.rec[5 * t + 4];
                                const float vis = alpha * T;
                                float depth = 0.f;
#pragma unroll
                                for (int k = 0; k < D; ++k) {
                                    pix_out[k] += (f4get(c4, k) + f4get(ts4, k) * ax.y) * vis;
                                    if (k == D - 1) depth = f4get(c4, k);
                                }
                                nrm_out[0] += nn.x * vis;
                                nrm_out[1] += nn.y * vis;
                                nrm_out[2] += nn.z * vis;
                                distort += 2.f * (vis * depth * (1.f - T) - vis * accum_vis_depth);
                                accum_vis_depth += vis * depth;
                                if (T > 0.5f) {
                                    median_depth = depth;
                                    median_idx = batch_start + t;
                                }
                                cur_idx = batch_start + t;
                                if (a.aniso_records != nullptr) {
                                    if (rec_n < a.aniso_record_cap)
                                        reinterpret_cast<float4*>(a.aniso_records)[pix * a.aniso_record_cap + rec_n] = ts4;
                                    ++rec_n;
                                }
                                own |= 1u << bit;
                                T = next_T;
                                if (alpha > a.contrib_threshold)
                                    stat = __float2uint_rn(alpha * 16777216.f) | (1u << 28);
                            }
                        }
                    }
                    stat += __shfl_xor_sync(kFull, stat, 4);
                    stat += __shfl_xor_sync(kFull, stat, 2);
                    stat += __shfl_xor_sync(kFull, stat, 1);
                    if ((lane & 7) == 0 && stat != 0u) {
                        atomicAdd(S.csum + t, stat & 0x0fffffffu);
                        atomicAdd(S.ccnt + t, stat >> 28);
                    }
                }
                if (t1 == 32) {
                    if (bits_out != nullptr) bits_out[(int64_t)w * (ts * ts)] = own;
                    own = 0u;
                }
            }
            t0 = t1 & 31;
            w += t1 >> 5;
        }
        if (a.t_checkpoints != nullptr && tr < 64)
            a.t_checkpoints[((int64_t)tc.t + range_start / bs + b) * (int64_t)(ts * ts) + (i - tc.ty * ts) * ts +
                            (j - tc.tx * ts)] = T;
    }
    __syncthreads();
    for (int slot = tr; slot < bs; slot += kAnisoThreads) flush_stats(slot);
    if (!inside) return;
    a.out_alphas[pix] = 1.f - T;
#pragma unroll
    for (int k = 0; k < D; ++k)
        a.out_colors[pix * D + k] = a.backgrounds ? pix_out[k] + T * a.backgrounds[tc.c * D + k] : pix_out[k];
    a.out_normals[pix * 3] = nrm_out[0];
    a.out_normals[pix * 3 + 1] = nrm_out[1];
    a.out_normals[pix * 3 + 2] = nrm_out[2];
    a.last_ids[pix] = cur_idx;
    a.out_distort[pix] = distort;
    a.out_median[pix] = median_depth;
    a.median_ids[pix] = median_idx;
    if (a.aniso_records != nullptr) a.aniso_record_count[pix] = rec_n;
}

// CTAs [0, n_long): one square of the first tiles in work order each; the others: four squares each.
template <int D, class Tex>
__global__ void __launch_bounds__(kAnisoThreads, 4) aniso_fwd_kernel(const tg_raster_fwd_args a, const int bs,
                                                                                 const int n_long, const int n_squares,
                                                                                 const int quarter_f4) {
    extern __shared__ float4 smem4[];
    const int subs = (a.tile_size / kAnisoSide) * (a.tile_size / kAnisoSide);
    if ((int)blockIdx.x < n_long) {
        aniso_long_square<D, Tex>(a, bs, blockIdx.x / subs, blockIdx.x % subs, smem4);
    } else {
        const int q = threadIdx.x >> 6;
        const int64_t k = n_long + ((int64_t)blockIdx.x - n_long) * 4 + q;
        if (k < n_squares)
            fwd_square<D, Tex, FiltAniso>(a, bs, k / subs, (int)(k % subs), kAnisoSide, smem4 + q * quarter_f4, QuarterCta{});
    }
}

template <int D, class Tex, bool kPersistent, class Filt>
cudaError_t launch_fwd_kernel(const tg_raster_fwd_args& a, cudaStream_t s) {
    const int side = square_side(a.tile_size), threads = side * side;
    const int bs = a.batch_depth > 0 ? a.batch_depth : a.tile_size * a.tile_size;
    const size_t smem = FwdSmem<D, Tex>::bytes(bs, side) + (Filt::kAniso ? (size_t)(threads / 32) * kAnisoWarpF4 * 16 : 0);
    const int64_t tiles = a.views ? a.n_tiles : (int64_t)a.C * a.tile_width * a.tile_height;
    const int64_t items = tiles * squares_per_tile(a.tile_size);
    if (items == 0) return cudaSuccess;
    if (items > 0x7fffffff) return cudaErrorInvalidValue;
    const auto fn = raster_fwd_kernel<D, Tex, kPersistent, Filt>;
    cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    int64_t grid = items;
    if (kPersistent) {
        if ((err = cudaMemsetAsync(a.work_queue, 0, sizeof(uint32_t), s)) != cudaSuccess) return err;
        if ((err = persistent_grid((const void*)fn, threads, smem, items, grid)) != cudaSuccess) return err;
    }
    fn<<<(unsigned)grid, threads, smem, s>>>(a, bs, items);
    note_launches(1);
    return cudaGetLastError();
}

template <int D, class Tex>
cudaError_t launch_aniso_fwd(const tg_raster_fwd_args& a, cudaStream_t s) {
    static_assert(kAnisoThreads == 256, "four quarters of 64 threads");
    const int bs = a.batch_depth > 0 ? a.batch_depth : a.tile_size * a.tile_size;
    const size_t quarter = FwdSmem<D, Tex>::bytes(bs, kAnisoSide) + 2 * kAnisoWarpF4 * 16;  // a multiple of 16
    const size_t smem = std::max(FwdSmem<D, Tex>::bytes(bs, kAnisoSide) + AnisoStep::kBytes, 4 * quarter);
    const int64_t tiles = a.views ? a.n_tiles : (int64_t)a.C * a.tile_width * a.tile_height;
    const int64_t subs = (a.tile_size / kAnisoSide) * (a.tile_size / kAnisoSide), squares = tiles * subs;
    if (squares == 0) return cudaSuccess;
    if (squares > 0x7fffffff) return cudaErrorInvalidValue;
    // (batches deeper than 608 splats do not fit a CTA's shared memory four times)
    if (squares >= kFullSquares || smem > kMaxSmem) return launch_fwd_kernel<D, Tex, false, FiltAniso>(a, s);
    const int64_t n_long = std::min<int64_t>(squares, (kLongTiles + subs - 1) / subs * subs);
    const int64_t items = n_long + (squares - n_long + 3) / 4;
    const cudaError_t err = cudaFuncSetAttribute(aniso_fwd_kernel<D, Tex>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)smem);
    if (err != cudaSuccess) return err;
    aniso_fwd_kernel<D, Tex><<<(unsigned)items, kAnisoThreads, smem, s>>>(a, bs, (int)n_long, (int)squares,
                                                                         (int)(quarter / 16));
    note_launches(1);
    return cudaGetLastError();
}

template <int D, class Tex>
cudaError_t launch_fwd_t(const tg_raster_fwd_args& a, cudaStream_t s) {
    // mipmapped2 / anisotropic_bilinear filters: FP32 / BF16 storage, 3 or 4 channels, 8x8 / 16x16 tiles, one CTA per tile
    if constexpr ((D == 3 || D == 4) && (Tex::kFormat == TG_TEX_F32 || Tex::kFormat == TG_TEX_BF16)) {
        if (a.mip_levels > 0) return launch_fwd_kernel<D, Tex, false, FiltMip2>(a, s);
        if (a.filter == TG_FILTER_ANISO_BILINEAR) return launch_aniso_fwd<D, Tex>(a, s);
    }
    if (a.mip_levels > 0 || a.filter != TG_FILTER_BILINEAR) return cudaErrorInvalidValue;
    return a.work_queue != nullptr ? launch_fwd_kernel<D, Tex, true, FiltBilinear>(a, s)
                                   : launch_fwd_kernel<D, Tex, false, FiltBilinear>(a, s);
}

// Packs the entries' records (see load_entry): a warp collects those of 32 entries in shared memory, reading every
// array and writing the records in whole lines.
template <int D>
__global__ void __launch_bounds__(128) pack_entries_kernel(const tg_raster_fwd_args a) {
    __shared__ float4 s4[4 * 32 * 5];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* s = reinterpret_cast<float*>(s4 + warp * 32 * 5);
    const int64_t e0 = ((int64_t)blockIdx.x * 4 + warp) * 32;
    const int n = (int)min((int64_t)32, a.n_entries - e0);
    if (n <= 0) return;  // (whole warps)
    for (int i = lane; i < 9 * n; i += 32) s[(i / 9) * 20 + (i % 9) / 3 * 4 + i % 3] = a.ray_transforms[9 * e0 + i];
    for (int i = lane; i < 3 * n; i += 32) s[(i / 3) * 20 + 16 + i % 3] = a.normals[3 * e0 + i];
    for (int i = lane; i < D * n; i += 32)
        if (i % D < 4) s[(i / D) * 20 + 12 + i % D] = a.colors[D * e0 + i];
    if (lane < n) {
        const int64_t e = e0 + lane;
        const float2 xy = reinterpret_cast<const float2*>(a.means2d)[e];
        float* r = s + lane * 20;
        r[3] = xy.x;
        r[7] = xy.y;
        r[11] = a.opacities[e];
        for (int k = D; k < 4; ++k) r[12 + k] = 0.f;
        r[19] = __int_as_float(a.gaussian_ids ? (int)a.gaussian_ids[e] : (int)(e % a.N));
    }
    __syncwarp();
    float4* dst = reinterpret_cast<float4*>(a.entry_records) + 5 * e0;
    for (int i = lane; i < 5 * n; i += 32) dst[i] = reinterpret_cast<const float4*>(s)[i];
}

cudaError_t launch_pack_entries(const tg_raster_fwd_args& a, cudaStream_t s) {
    if (a.entry_records == nullptr || a.n_entries == 0) return cudaSuccess;
    const unsigned grid = (unsigned)((a.n_entries + 127) / 128);
    switch (a.D) {
        case 1: pack_entries_kernel<1><<<grid, 128, 0, s>>>(a); break;
        case 2: pack_entries_kernel<2><<<grid, 128, 0, s>>>(a); break;
        case 3: pack_entries_kernel<3><<<grid, 128, 0, s>>>(a); break;
        case 4: pack_entries_kernel<4><<<grid, 128, 0, s>>>(a); break;
        case 5: pack_entries_kernel<5><<<grid, 128, 0, s>>>(a); break;
        default: return cudaErrorInvalidValue;
    }
    note_launches(1);
    return cudaGetLastError();
}

template <class Tex>
cudaError_t launch_fwd_d(const tg_raster_fwd_args& a, cudaStream_t s) {
    switch (a.D) {
        case 1: return launch_fwd_t<1, Tex>(a, s);
        case 2: return launch_fwd_t<2, Tex>(a, s);
        case 3: return launch_fwd_t<3, Tex>(a, s);
        case 4: return launch_fwd_t<4, Tex>(a, s);
        case 5: return launch_fwd_t<5, Tex>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

// Low-precision texture forms are built for the RGB and RGB+D channel counts.
template <class Tex>
cudaError_t launch_fwd_d34(const tg_raster_fwd_args& a, cudaStream_t s) {
    switch (a.D) {
        case 3: return launch_fwd_t<3, Tex>(a, s);
        case 4: return launch_fwd_t<4, Tex>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_raster_fwd(const tg_raster_fwd_args& a, cudaStream_t s) {
    const cudaError_t e = launch_pack_entries(a, s);
    if (e != cudaSuccess) return e;
    switch (a.tex_format) {
        case TG_TEX_NONE: return launch_fwd_d<TexNone>(a, s);
        case TG_TEX_F32: return launch_fwd_d<TexF32>(a, s);
        case TG_TEX_BF16: return launch_fwd_d34<TexBF16>(a, s);
        case TG_TEX_F16: return launch_fwd_d34<TexF16>(a, s);
        case TG_TEX_FP8_E4M3: return launch_fwd_d34<TexFP8>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace tg
