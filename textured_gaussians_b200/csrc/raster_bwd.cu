// Textured / plain 2DGS compositor, adjoint, for sm_100a.
//
// One CTA per (camera, tile) work item (a quarter of a 32x32 tile), one thread per pixel, back-to-front in batches
// of `batch_depth` staged splats.  Transmittance is recovered from the stored final T by division, as the
// reference does (rasterize_to_pixels_textured_gaussians_2dgs_bwd.cu:160, :456-457).
//
// What is evaluated: the forward leaves one bit per (pixel, listed splat), set where the pair was composited
// (tg_raster_fwd_args.contrib_masks), and the adjoint visits exactly those pairs.  As in the forward each 4x2 pixel
// group walks its own list -- the union of its eight pixels' bits -- so the four groups of a warp work on four
// splats at once: 0.34 warp evaluations per listed splat on the 1M-splat mixture, against 1.13 with a warp per
// 8x4 block and its box test.  Without the bits (NULL) the groups' lists come from group_mask again and every
// pair is tested.
//
// Reductions:
//  * per-splat gradients (colour, ray transform, means2d, opacity; with an upstream gradient for normals, distortion
//    or median depth, or |means2d| asked for, also those) are summed over a group's eight lanes by a reduce-scatter
//    (14 shuffles for 16 values, 21 for 24) that leaves consecutive values in consecutive lanes, which add them to
//    the entry's row of a packed [E, slots] buffer -- 64 contiguous bytes, two per lane.  A splat meets 1.1 groups
//    per tile that lists it, so collecting a tile's sums in shared memory first would not save adds; the rows are
//    spread to the separate gradient arrays by one pass over the entries afterwards;
//  * per-texel gradients are RGBA float4 vector atomics, one per bilinear tap
//    (4 per pixel-splat pair instead of the reference's up to 4*(D+1) scalar atomics).
//
// Adjoint forms: TG_ADJ_REFERENCE follows ..._bwd.cu:438-627; TG_ADJ_BWD2 adds
// the reference's texture-UV term (..._bwd2.cu:612-676, du/ds = (R-1)/range);
// TG_ADJ_EXACT adds the UV term with the true du/ds = (R-1)/(2 range).
#include "raster_common.cuh"

namespace tg {

// Slots of an entry's row of gradient sums.  kGeo: with the upstream gradients of normals, distortion and median
// depth, and |means2d|.
template <int D, bool kGeo>
struct GradSlots {
    static constexpr int kRgb = 0;
    static constexpr int kM = D;
    static constexpr int kXY = D + 9;
    static constexpr int kOpac = D + 11;
    static constexpr int kNrm = D + 12;
    static constexpr int kAbs = D + 15;
    static constexpr int kUsed = kGeo ? D + 17 : D + 12;
    static constexpr int kCount = kUsed <= 16 ? 16 : 24;
};

// Sum over each 8 lanes of every value; lane l keeps the NS / 8 sums from slot_base<NS>(l) on, in v[0 ..].
template <int NS>
__device__ __forceinline__ void reduce_scatter8(float (&v)[NS]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int s = 4, n = NS / 2; s >= 1; s >>= 1, n >>= 1) {
        const bool upper = (lane & s) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float send = upper ? v[i] : v[i + n];
            const float keep = upper ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
    }
}
template <int NS>
__device__ __forceinline__ int slot_base(int lane) {
    return ((lane & 4) ? NS / 2 : 0) + ((lane & 2) ? NS / 4 : 0) + ((lane & 1) ? NS / 8 : 0);
}

// Resident CTAs of 256 threads per SM the register allocation targets.
#ifndef TG_BWD_MIN_CTAS
#define TG_BWD_MIN_CTAS 3
#endif
// The anisotropic_bilinear adjoint targets 3 CTAs (80 registers allocated): with its clips
// branch-free and its cell boundary sum out of line it spills ~1 KB there but
// runs 3.9 % faster than at 128, which was already 28 % faster than the
// unconstrained 245; 64 registers lose 17 % (1M splats, 4 views, measured).
#ifndef TG_BWD_MIN_CTAS_ANISO
#define TG_BWD_MIN_CTAS_ANISO 3
#endif
// Two CTAs (up to 128 registers) where three spill more than they hide: FP32 textures (1496 against 1560 us for 100k
// splats of 50x50 texels, 800x800), mipmapped2 (687 against 703 us), the geometric sums and the UV term; with 16-bit
// textures three are faster (9.31 against 10.18 ms for the 1M-splat mixture, four views), and four slower throughout.
template <class Tex, class Filt, bool kGeo>
struct BwdBounds {
    static constexpr bool kWide = kGeo || Filt::kUV || Filt::kMip || Tex::kFormat == TG_TEX_F32;
    static constexpr int kMinCtas = Filt::kAniso ? TG_BWD_MIN_CTAS_ANISO : kWide ? 2 : TG_BWD_MIN_CTAS;
};

// Per-pixel state of the back-to-front sweep.  Everything behind the current splat enters its alpha's gradient
// through one number: rest = T_final (v_alpha - v_c . background) - sum over the splats behind of
// weight * (their colour . v_c + normal . v_n + distortion term).
template <int D, bool kGeo>
struct PixelAdj {
    float px, py;
    float T, rest, v_c[D];
    int32_t ck_batch;  // batch whose end transmittance T was last restarted from (-1: none)
    // kGeo only
    float v_n[3], v_dist, v_med, acc_d_buf, acc_d, acc_w_buf, acc_w;
    int32_t median_idx;
};

// Adds one (pixel, splat) pair's gradient contributions to the lane's per-splat
// sums `vals` (slots of GradSlots), issues the pair's texel-gradient atomics,
// and advances the pixel's back-to-front state.  Follows
// rasterize_to_pixels_textured_gaussians_2dgs_bwd.cu:438-627 (+ bwd2.cu:612-676).
template <int D, class Tex, class Filt, bool kGeo, int NS>
__device__ __forceinline__ void accumulate_pair(const tg_raster_bwd_args& a, const PairOf<Filt>& e,
                                                PixelAdj<D, kGeo>& P, const float opac, const float4 nn,
                                                const float (&cp)[D], int32_t idx, float* vt, float uv_scale,
                                                float (&vals)[NS], float* vct = nullptr, int mip_clen = 0,
                                                float4* aniso_g = nullptr) {
    // aniso_g (anisotropic_bilinear): receives the texel-gradient factor of the pair (divided by the area), which
    // the warp scatters over the footprint together
    constexpr bool kTextured = Tex::kFormat != TG_TEX_NONE;
    using GS = GradSlots<D, kGeo>;
    const tg_raster_fwd_args& f = a.f;
    const float ra = 1.f / (1.f - e.alpha);
    P.T *= ra;
    const float T = P.T;
    const float fac = e.alpha * T;
    float q = 0.f;  // d L / d weight of this splat
#pragma unroll
    for (int k = 0; k < D; ++k) {
        vals[GS::kRgb + k] = fac * P.v_c[k];
        q += ((kTextured ? tex_color_adj(e, k) : 0.f) + cp[k]) * P.v_c[k];
    }
    if constexpr (kGeo) {
        if (idx == P.median_idx) vals[GS::kRgb + D - 1] += P.v_med;
        vals[GS::kNrm + 0] = fac * P.v_n[0];
        vals[GS::kNrm + 1] = fac * P.v_n[1];
        vals[GS::kNrm + 2] = fac * P.v_n[2];
        q += nn.x * P.v_n[0] + nn.y * P.v_n[1] + nn.z * P.v_n[2];
        const float depth = cp[D - 1];
        const float dl_dw = 2.f * (2.f * (depth * P.acc_w_buf - P.acc_d_buf) + (P.acc_d - depth * P.acc_w));
        q += dl_dw * P.v_dist;
        P.acc_d_buf -= fac * depth;
        P.acc_w_buf -= fac;
        vals[GS::kRgb + D - 1] += 2.f * fac * (2.f - 2.f * T - P.acc_w + fac) * P.v_dist;
    }
    const float v_alpha = q * T + P.rest * ra;
    P.rest -= fac * q;
    // d L / d s, from the Gaussian kernel (3D branch) and, for the UV-aware adjoints, from the
    // texture lookup; both go back through s = zeta.xy / zeta.z and zeta = h_u x h_v once
    float vsx = 0.f, vsy = 0.f;
    const bool unclamped = kTextured ? (opac * e.vis * e.asf <= 0.999f) : (opac * e.vis <= 0.999f);
    float tex_a_grad = 0.f;  // d L / d (texture alpha) / w_i
    if (unclamped) {
        const float v_G = kTextured ? opac * v_alpha * e.asf : opac * v_alpha;
        const float dG = kTextured ? -f.g_weight * e.kern : -e.vis;
        if (e.g3 <= e.g2) {
            vsx = v_G * dG * e.sx;
            vsy = v_G * dG * e.sy;
        } else {
            const float vx = v_G * (dG * kFilterInvSquare * e.dx);
            const float vy = v_G * (dG * kFilterInvSquare * e.dy);
            vals[GS::kXY] = vx;
            vals[GS::kXY + 1] = vy;
            if constexpr (kGeo) {
                vals[GS::kAbs] = fabsf(vx);
                vals[GS::kAbs + 1] = fabsf(vy);
            }
        }
        vals[GS::kOpac] = kTextured ? e.vis * v_alpha * e.asf : e.vis * v_alpha;
        tex_a_grad = e.vis * opac * v_alpha;
    }
    if constexpr (Filt::kAniso) {
        if (e.tex_valid && vt != nullptr) {
            const float4 g = make_float4(D > 0 ? fac * P.v_c[0] : 0.f, D > 1 ? fac * P.v_c[D > 1 ? 1 : 0] : 0.f,
                                         D > 2 ? fac * P.v_c[D > 2 ? 2 : 0] : 0.f,
                                         (D > 3 ? fac * P.v_c[D > 3 ? 3 : 0] : 0.f) + tex_a_grad);
            const float ia = e.F.iarea;
            *aniso_g = make_float4(g.x * ia, g.y * ia, g.z * ia, g.w * ia);
        }
    } else if (kTextured && e.tex_valid && vt != nullptr) {
        const float4 g = make_float4(D > 0 ? fac * P.v_c[0] : 0.f, D > 1 ? fac * P.v_c[D > 1 ? 1 : 0] : 0.f,
                                     D > 2 ? fac * P.v_c[D > 2 ? 2 : 0] : 0.f,
                                     (D > 3 ? fac * P.v_c[D > 3 ? 3 : 0] : 0.f) + tex_a_grad);
        const bool any = g.x != 0.f || g.y != 0.f || g.z != 0.f || g.w != 0.f;
#pragma unroll
        for (int q = 0; q < Filt::kTaps; ++q) {
            if (any && e.w[q] != 0.f) {
                const float4 gq = make_float4(e.w[q] * g.x, e.w[q] * g.y, e.w[q] * g.z, e.w[q] * g.w);
                if constexpr (Filt::kMip) {  // pyramid coordinate: coarse levels, or level 0 = the texture
                    const int mc = e.toff[q];
                    float* dst = mc < mip_clen ? vct + 4 * (int64_t)mc : vt + 4 * (int64_t)(mc - mip_clen);
                    atomicAdd(reinterpret_cast<float4*>(dst), gq);
                } else {
                    atomicAdd(reinterpret_cast<float4*>(vt + 4 * (int64_t)e.toff[q]), gq);
                }
            }
        }
    }
    if constexpr (Filt::kUV) if (kTextured && e.tex_valid && uv_scale != 0.f) {
        const float wu = e.w[1] + e.w[3], wv = e.w[2] + e.w[3];
        const float dbu[4] = {-(1.f - wv), 1.f - wv, -wv, wv};
        const float dbv[4] = {-(1.f - wu), -wu, 1.f - wu, wu};
        const float du = uv_scale * (float)(f.tex_rx - 1) / f.range_x;
        const float dv = uv_scale * (float)(f.tex_ry - 1) / f.range_y;
        float tsx = 0.f, tsy = 0.f;
#pragma unroll
        for (int k = 0; k < D && k < 4; ++k) {
            const float vt_k = fac * P.v_c[k];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float tv = f4get(e.tx[q], k);
                tsx += vt_k * dbu[q] * tv;
                tsy += vt_k * dbv[q] * tv;
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            tsx += tex_a_grad * dbu[q] * e.tx[q].w;
            tsy += tex_a_grad * dbv[q] * e.tx[q].w;
        }
        vsx += tsx * du;
        vsy += tsy * dv;
    }
    if (vsx != 0.f || vsy != 0.f) {
        const float iz = 1.f / e.z.z;
        const float a_ = vsx * iz, b_ = vsy * iz;
        const f3 vz = mk3(a_, b_, -(a_ * e.sx + b_ * e.sy));
        // The pair's nine products themselves.  As moments of vz about the projected centre (one sum less to form a pair,
        // expanded once per entry) FP32 loses a pixel's place beside a centre far off the image: gradients of splats
        // whose plane passes near the camera were 3e-2 off against 6e-7 (median over 96, 160x120), and the step was
        // no faster (20.11 and 20.17 ms for the 1M-splat mixture, four views).
        const f3 vhu = cross(e.hv, vz), vhv = cross(vz, e.hu);
        vals[GS::kM + 0] = -vhu.x; vals[GS::kM + 1] = -vhu.y; vals[GS::kM + 2] = -vhu.z;
        vals[GS::kM + 3] = -vhv.x; vals[GS::kM + 4] = -vhv.y; vals[GS::kM + 5] = -vhv.z;
        vals[GS::kM + 6] = P.px * vhu.x + P.py * vhv.x;
        vals[GS::kM + 7] = P.px * vhu.y + P.py * vhv.y;
        vals[GS::kM + 8] = P.px * vhu.z + P.py * vhv.z;
    }
}

// Adds one sum straight to its gradient array (a caller without the packed rows).
template <int D, bool kGeo>
__device__ __forceinline__ void scatter_slot(const tg_raster_bwd_args& a, int64_t g, int slot, float v) {
    using GS = GradSlots<D, kGeo>;
    if (v == 0.f || slot >= GS::kUsed) return;
    float* dst;
    if (slot < GS::kM) dst = a.v_colors + g * D + slot;
    else if (slot < GS::kXY) dst = a.v_ray_transforms + g * 9 + (slot - GS::kM);
    else if (slot < GS::kOpac) dst = a.v_means2d + g * 2 + (slot - GS::kXY);
    else if (slot == GS::kOpac) dst = a.v_opacities + g;
    else if (slot < GS::kAbs) dst = a.v_normals + g * 3 + (slot - GS::kNrm);
    else dst = a.v_means2d_abs ? a.v_means2d_abs + g * 2 + (slot - GS::kAbs) : nullptr;
    if (dst) atomicAdd(dst, v);
}

// Staged splats and the lists of a batch.
template <int D, class Tex, bool kGeo>
struct BwdSmem {
    static constexpr bool kScale = Tex::kFormat == TG_TEX_FP8_E4M3;
    static constexpr int kVec = kGeo ? 6 : 5;
    float4* rec;  // [bs][kVec]: three rows, colour, (texture row, entry), and with kGeo the normal
    float *col5, *scale;
    uint32_t *words;   // [groups][n_words]
    uint32_t *pixels;  // [n_words][threads]: the pixels' own bits
    float4* extra;     // anisotropic_bilinear: the boundary integration's per-warp areas
    __device__ __forceinline__ BwdSmem(float4* base, int bs, int side) {
        rec = base;
        scale = reinterpret_cast<float*>(rec + kVec * bs);
        col5 = scale + (kScale ? bs : 0);
        words = reinterpret_cast<uint32_t*>(col5 + (D == 5 ? bs : 0));
        pixels = words + (side * side / kGroupLanes) * (bs / 32);
        extra = reinterpret_cast<float4*>(pixels + side * side * (bs / 32));
    }
    static size_t bytes(int bs, int side) {
        return (size_t)bs * (kVec * sizeof(float4) + (kScale ? 4 : 0) + (D == 5 ? 4 : 0)) +
               (size_t)(side * side / kGroupLanes + side * side) * (bs / 32) * 4;
    }
};

// One work item of the adjoint; every early return is uniform over the CTA.
template <int D, class Tex, class Filt, bool kGeo>
__device__ __forceinline__ void bwd_tile(const tg_raster_bwd_args& a, const float uv_scale, const int bs,
                                         const int64_t item) {
    using GS = GradSlots<D, kGeo>;
    constexpr int NS = GS::kCount;
    constexpr unsigned kFull = 0xffffffffu;
    constexpr bool kTextured = Tex::kFormat != TG_TEX_NONE;
    const tg_raster_fwd_args& f = a.f;
    extern __shared__ float4 smem4[];
    __shared__ int s_max_bin;
    const int nt = blockDim.x;  // one thread per pixel of the square
    const int ts = f.tile_size, side = square_side(ts), subs = squares_per_tile(ts);
    const BwdSmem<D, Tex, kGeo> S(smem4, bs, side);
    constexpr int kVec = BwdSmem<D, Tex, kGeo>::kVec;
    float4* s_aniso = Filt::kAniso ? S.extra + (threadIdx.x >> 5) * kAnisoWarpF4 : nullptr;

    const TileWork tc = tile_work(f, subs == 1 ? item : item / subs);
    if (!tc.valid) return;  // uniform over the CTA
    const int tr = threadIdx.x, lane = tr & 31;
    if (f.masks != nullptr && !f.masks[tc.t]) return;
    const int sub = subs == 1 ? 0 : (int)(item % subs);
    const int X0 = tc.tx * ts + (sub & 1) * side, Y0 = tc.ty * ts + (sub >> 1) * side;
    const PixelSlot ps = pixel_slot(tr, side);
    const int j = X0 + ps.x, i = Y0 + ps.y;
    const int64_t pix = pixel_index(tc, i, j);
    const bool inside = pix >= 0;
    const int32_t range_start = tc.range_start;
    const int32_t range_end = tc.range_end;
    if (tr == 0) s_max_bin = -1;

    PixelAdj<D, kGeo> P;
    P.px = (float)j + 0.5f;
    P.py = (float)i + 0.5f;
    P.T = 1.f;
    P.rest = 0.f;
    P.ck_batch = -1;
    int32_t bin_final = -1;
    int32_t record = -1;  // anisotropic_bilinear: the forward's record of the next footprint integral (counting down)
#pragma unroll
    for (int k = 0; k < D; ++k) P.v_c[k] = 0.f;
    if constexpr (kGeo) {
        P.v_n[0] = P.v_n[1] = P.v_n[2] = P.v_dist = P.v_med = 0.f;
        P.acc_d_buf = P.acc_d = P.acc_w_buf = P.acc_w = 0.f;
        P.median_idx = -1;
    }
    if (inside) {
        const float alpha_out = a.render_alphas[pix];
        P.T = 1.f - alpha_out;
        bin_final = a.last_ids[pix];
        float v_a = a.v_render_alphas ? a.v_render_alphas[pix] : 0.f;
        if (a.v_render_colors) {
#pragma unroll
            for (int k = 0; k < D; ++k) P.v_c[k] = a.v_render_colors[pix * D + k];
        }
        if (f.backgrounds) {
            float bg_dot = 0.f;
#pragma unroll
            for (int k = 0; k < D; ++k) bg_dot += f.backgrounds[tc.c * D + k] * P.v_c[k];
            v_a -= bg_dot;
        }
        P.rest = P.T * v_a;
        if constexpr (kGeo) {
            P.median_idx = a.median_ids[pix];
            if (a.v_render_normals) {
                P.v_n[0] = a.v_render_normals[pix * 3];
                P.v_n[1] = a.v_render_normals[pix * 3 + 1];
                P.v_n[2] = a.v_render_normals[pix * 3 + 2];
            }
            if (a.v_render_distort) P.v_dist = a.v_render_distort[pix];
            if (a.v_render_median) P.v_med = a.v_render_median[pix];
            P.acc_d_buf = P.acc_d = a.render_colors[pix * D + D - 1];
            P.acc_w_buf = P.acc_w = alpha_out;
        }
        if (Filt::kAniso && f.aniso_records != nullptr && f.contrib_masks != nullptr)
            record = f.aniso_record_count[pix] - 1;
    }
    // last contributor over the CTA
    const int32_t warp_bin_final = __reduce_max_sync(kFull, bin_final);
    __syncthreads();
    if (lane == 0) atomicMax(&s_max_bin, warp_bin_final);
    __syncthreads();
    const int32_t max_bin = min(s_max_bin, range_end - 1);
    const int64_t tex_stride = (int64_t)f.tex_ry * f.tex_rx;
    const int mip_clen = Filt::kMip ? ((1 << (2 * f.mip_levels)) - 1) / 3 : 0;
    const int n_words = bs >> 5;
    const bool have_bits = f.contrib_masks != nullptr;
    const uint32_t* bits_base = have_bits ? f.contrib_masks + ((int64_t)tc.t + (range_start >> 5)) * (int64_t)(ts * ts) +
                                                sub * nt + tr
                                          : nullptr;
    const uint32_t* words = S.words + (size_t)(tr >> 3) * n_words;  // the lane's group's list

    for (int b = max_bin < range_start ? -1 : (max_bin - range_start) / bs; b >= 0; --b) {
        const int32_t batch_start = range_start + b * bs;
        __syncthreads();  // previous batch done before restaging
        const int last_word = (max_bin - batch_start) >> 5;  // the forward went at least this far
        for (int slot = tr; slot < bs; slot += nt) {  // (whole warps: bs and nt are multiples of 32)
            const int32_t idx = batch_start + slot;
            uint32_t reach = 0u;
            if (idx <= max_bin) {
                const int32_t g = f.flatten_ids[idx];
                const EntryRecord r = load_entry<D, kGeo>(f, g);
                const int32_t row = __float_as_int(r.nrm.w);
                float4* rec = S.rec + kVec * slot;
                rec[0] = r.m0;
                rec[1] = r.m1;
                rec[2] = r.m2;
                rec[3] = r.col;
                rec[4] = make_float4(r.nrm.w, __int_as_float(g), 0.f, 0.f);
                if constexpr (D == 5) S.col5[slot] = f.colors[(int64_t)g * D + 4];
                if constexpr (kGeo) rec[5] = r.nrm;
                if constexpr (BwdSmem<D, Tex, kGeo>::kScale) S.scale[slot] = f.tex_scales[row];
                if (!have_bits)
                    reach = group_mask(make_float4(r.m0.w, r.m1.w, r.m2.w, 1.f), r.m0, r.m1, r.m2, kTextured, f.range_x,
                                       f.range_y, f.g_weight, !Filt::kAniso, X0, Y0, side);
            }
            if (!have_bits) store_group_words(reach, S.words, n_words, slot >> 5, side);
        }
        for (int w = 0; w < n_words; ++w) {
            uint32_t own = inside ? kFull : 0u;
            if (have_bits) {
                own = w <= last_word ? bits_base[(int64_t)(b * n_words + w) * (ts * ts)] : 0u;
                uint32_t u = own | __shfl_xor_sync(kFull, own, 4);
                u |= __shfl_xor_sync(kFull, u, 2);
                u |= __shfl_xor_sync(kFull, u, 1);
                if ((lane & 7) == 0) S.words[(tr >> 3) * n_words + w] = u;
            }
            S.pixels[w * nt + tr] = own;
        }
        __syncthreads();
        int w = n_words - 1;
        uint32_t bits = words[w], own = S.pixels[w * nt + tr];
        for (;;) {
            while (bits == 0u && w > 0) {
                bits = words[--w];
                own = S.pixels[w * nt + tr];
            }
            if (!__any_sync(kFull, bits != 0u)) break;
            const bool listed = bits != 0u;  // (a group whose list is used up idles until its warp's others are done)
            const int bit = listed ? 31 - __clz(bits) : 0;
            bits &= ~(1u << bit);
            const int t = w * 32 + bit;
            const int32_t idx = batch_start + t;
            const bool act = listed && ((own >> bit) & 1u) != 0u && idx <= bin_final;
            const float4* rec = S.rec + kVec * t;
            float vals[NS];
#pragma unroll
            for (int k = 0; k < NS; ++k) vals[k] = 0.f;
            if (Filt::kAniso || act) {
                const float4 m0 = rec[0], m1 = rec[1], m2 = rec[2];
                const float4 xyo = make_float4(m0.w, m1.w, m2.w, BwdSmem<D, Tex, kGeo>::kScale ? S.scale[t] : 1.f);
                const int row = __float_as_int(rec[4].x);
                const int64_t tex_base = (int64_t)row * tex_stride;
                float* vt = a.v_textures != nullptr ? a.v_textures + 4 * tex_base : nullptr;
                float* vct = Filt::kMip && a.v_tex_coarse != nullptr ? a.v_tex_coarse + 4 * (int64_t)row * mip_clen
                                                                     : nullptr;
                PairOf<Filt> e;
                if constexpr (Filt::kAniso) {  // every lane takes part: the warp integrates footprints together
                    // the forward's integral of this pair's footprint, if it has one (it keeps the first
                    // aniso_record_cap contributors of each pixel, in order; this walks them back to front)
                    const float4* r = act && record >= 0 && record < f.aniso_record_cap
                                          ? reinterpret_cast<const float4*>(f.aniso_records) +
                                                pix * f.aniso_record_cap + record
                                          : nullptr;
                    eval_aniso_coop<Tex, true>(e, act, P.px, P.py, xyo, m0, m1, m2, f.textures, row, f.tex_rx, f.tex_ry,
                                               f.range_x, f.range_y, f.g_weight, kFull,
                                               reinterpret_cast<const float4*>(f.aniso_prefix), s_aniso, r);
                    if (act) --record;
                } else {
                    eval_pair<Tex, Filt>(e, P.px, P.py, xyo, m0, m1, m2, f.textures, tex_base, f.tex_rx, f.tex_ry,
                                         f.range_x, f.range_y, f.g_weight,
                                         MipSrc{f.tex_coarse, (int64_t)row * mip_clen, mip_clen, f.mip_levels});
                }
                float4 g4 = make_float4(0.f, 0.f, 0.f, 0.f);
                const bool use = act && e.valid;
                if (use) {
                    if (f.t_checkpoints != nullptr && b != P.ck_batch) {
                        // first pair of a new forward batch (back to front): T restarts from the forward's exact
                        // value at the batch's end -- no splat after this one in the batch contributed to this
                        // pixel, or it would have been met first
                        P.ck_batch = b;
                        P.T = f.t_checkpoints[((int64_t)tc.t + range_start / bs + b) * (int64_t)(ts * ts) +
                                              (i - tc.ty * ts) * ts + (j - tc.tx * ts)];
                    }
                    const float4 c4 = rec[3];
                    float cp[D];
#pragma unroll
                    for (int k = 0; k < D; ++k) cp[k] = k < 4 ? f4get(c4, k) : S.col5[t];
                    const float4 nn = kGeo ? rec[kVec - 1] : make_float4(0.f, 0.f, 0.f, 0.f);
                    accumulate_pair<D, Tex, Filt, kGeo, NS>(a, e, P, xyo.z, nn, cp, idx, vt, uv_scale, vals, vct,
                                                            mip_clen, &g4);
                }
                if constexpr (Filt::kAniso)
                    aniso_coop_scatter<true>(e.F, g4,
                                             use && e.tex_valid && vt != nullptr &&
                                                 (g4.x != 0.f || g4.y != 0.f || g4.z != 0.f || g4.w != 0.f),
                                             a.v_textures, row, f.tex_rx, f.tex_ry, kFull, a.v_aniso_prefix, s_aniso);
            }
            reduce_scatter8<NS>(vals);
            const int64_t g = __float_as_int(rec[4].y);
            const int slot = slot_base<NS>(lane);
            if (a.v_packed != nullptr) {
                float* dst = a.v_packed + g * NS + slot;
                if constexpr (NS == 16) {
                    if (vals[0] != 0.f || vals[1] != 0.f)
                        atomicAdd(reinterpret_cast<float2*>(dst), make_float2(vals[0], vals[1]));
                } else {
#pragma unroll
                    for (int k = 0; k < NS / 8; ++k)
                        if (vals[k] != 0.f) atomicAdd(dst + k, vals[k]);
                }
            } else {
#pragma unroll
                for (int k = 0; k < NS / 8; ++k) scatter_slot<D, kGeo>(a, g, slot + k, vals[k]);
            }
        }
    }
}

// CTA per work item, or (work_queue != NULL) a persistent grid whose CTAs take
// items from the queue counter until none is left.
template <int D, class Tex, bool kPersistent, class Filt, bool kGeo>
__global__ void __launch_bounds__(256, BwdBounds<Tex, Filt, kGeo>::kMinCtas) raster_bwd_kernel(const tg_raster_bwd_args a,
                                                                                          const float uv_scale,
                                                                                          const int bs,
                                                                                          const int64_t n_items) {
    if constexpr (!kPersistent) {
        bwd_tile<D, Tex, Filt, kGeo>(a, uv_scale, bs, blockIdx.x);
        return;
    }
    else {
        __shared__ int64_t s_item;
        for (;;) {
            if (threadIdx.x == 0) s_item = (int64_t)atomicAdd(a.f.work_queue, 1u);
            __syncthreads();  // also: every thread is done with the previous item's shared memory
            const int64_t item = s_item;
            __syncthreads();  // s_item read by all before it is rewritten
            if (item >= n_items) return;
            bwd_tile<D, Tex, Filt, kGeo>(a, uv_scale, bs, item);
        }
    }
}

// v_densify[e] = (v_M[e][2], v_M[e][5]) * M[e][8], once every contribution is in.
__global__ void densify_grad_kernel(const float* __restrict__ v_M, const float* __restrict__ M, int64_t n,
                                    float* __restrict__ v_densify) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const float depth = M[9 * e + 8];
    v_densify[2 * e] = v_M[9 * e + 2] * depth;
    v_densify[2 * e + 1] = v_M[9 * e + 5] * depth;
}

// Spreads the entries' packed rows over the gradient arrays (every element is written, so none is cleared first)
// and forms v_densify.  128 rows per CTA go through shared memory, so that both the reads and the writes of the
// odd-sized arrays are coalesced; the pass moves its bytes once (HBM-bound).
template <int D, bool kGeo>
__global__ void __launch_bounds__(128) unpack_grads_kernel(const tg_raster_bwd_args a) {
    using GS = GradSlots<D, kGeo>;
    constexpr int NS = GS::kCount, kRows = 128, kPitch = NS + 1;
    __shared__ float s[kRows * kPitch];
    const int64_t e0 = (int64_t)blockIdx.x * kRows;
    const int n = (int)min((int64_t)kRows, a.n_elems - e0);
    const float4* src = reinterpret_cast<const float4*>(a.v_packed + e0 * NS);
    for (int k = threadIdx.x; k < n * (NS / 4); k += kRows) {
        const float4 v = src[k];
        float* d = s + (k / (NS / 4)) * kPitch + (k % (NS / 4)) * 4;
        d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    }
    __syncthreads();
    if ((int)threadIdx.x < n) {
        const int64_t e = e0 + threadIdx.x;
        const float depth = a.f.ray_transforms[9 * e + 8];
        const float* r = s + threadIdx.x * kPitch + GS::kM;
        reinterpret_cast<float2*>(a.v_densify)[e] = make_float2(r[2] * depth, r[5] * depth);
    }
    __syncthreads();
    auto spread = [&](float* dst, int width, int off) {
        for (int k = threadIdx.x; k < n * width; k += kRows) dst[e0 * width + k] = s[(k / width) * kPitch + off + k % width];
    };
    spread(a.v_colors, D, GS::kRgb);
    spread(a.v_ray_transforms, 9, GS::kM);
    spread(a.v_means2d, 2, GS::kXY);
    spread(a.v_opacities, 1, GS::kOpac);
    if constexpr (kGeo) {
        spread(a.v_normals, 3, GS::kNrm);
        if (a.v_means2d_abs) spread(a.v_means2d_abs, 2, GS::kAbs);
    } else {
        for (int k = threadIdx.x; k < n * 3; k += kRows) a.v_normals[e0 * 3 + k] = 0.f;
    }
}

// Whether the call needs the sums of the geometric upstream gradients (else the smaller rows do).
bool bwd_geo(const tg_raster_bwd_args& a) {
    return a.v_render_normals != nullptr || a.v_render_distort != nullptr || a.v_render_median != nullptr ||
           a.v_means2d_abs != nullptr || a.adjoint != TG_ADJ_REFERENCE || !(a.f.D == 3 || a.f.D == 4);
}
// Floats per entry of v_packed that a call uses (include/tg2dgs.h: callers provide the larger size).
int bwd_slots(const tg_raster_bwd_args& a) { return bwd_geo(a) ? 24 : 16; }

template <int D, class Tex, bool kPersistent, class Filt, bool kGeo>
cudaError_t launch_bwd_kernel(const tg_raster_bwd_args& a, float uv_scale, cudaStream_t s) {
    const tg_raster_fwd_args& f = a.f;
    const int side = square_side(f.tile_size), threads = side * side;
    const int bs = f.batch_depth > 0 ? f.batch_depth : f.tile_size * f.tile_size;
    const size_t smem = BwdSmem<D, Tex, kGeo>::bytes(bs, side) +
                        (Filt::kAniso ? (size_t)(threads / 32) * kAnisoWarpF4 * 16 : 0);
    const int64_t tiles = f.views ? f.n_tiles : (int64_t)f.C * f.tile_width * f.tile_height;
    const int64_t items = tiles * squares_per_tile(f.tile_size);
    if (items > 0x7fffffff) return cudaErrorInvalidValue;
    const auto fn = raster_bwd_kernel<D, Tex, kPersistent, Filt, kGeo>;
    cudaError_t err = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    if (items > 0 && f.n_isects > 0) {
        int64_t grid = items;
        if (kPersistent) {
            if ((err = cudaMemsetAsync(f.work_queue, 0, sizeof(uint32_t), s)) != cudaSuccess) return err;
            if ((err = persistent_grid((const void*)fn, threads, smem, items, grid)) != cudaSuccess) return err;
        }
        fn<<<(unsigned)grid, threads, smem, s>>>(a, uv_scale, bs, items);
        note_launches(1);
        if ((err = cudaGetLastError()) != cudaSuccess) return err;
    }
    if (a.n_elems > 0) {
        if (a.v_packed != nullptr)
            unpack_grads_kernel<D, kGeo><<<(unsigned)((a.n_elems + 127) / 128), 128, 0, s>>>(a);
        else
            densify_grad_kernel<<<(unsigned)((a.n_elems + 255) / 256), 256, 0, s>>>(a.v_ray_transforms,
                                                                                   f.ray_transforms, a.n_elems,
                                                                                   a.v_densify);
        note_launches(1);
    }
    return cudaGetLastError();
}

template <int D, class Tex, class Filt, bool kGeo>
cudaError_t launch_bwd_bilinear(const tg_raster_bwd_args& a, float uv_scale, cudaStream_t s) {
    return a.f.work_queue != nullptr ? launch_bwd_kernel<D, Tex, true, Filt, kGeo>(a, uv_scale, s)
                                     : launch_bwd_kernel<D, Tex, false, Filt, kGeo>(a, uv_scale, s);
}

template <int D, class Tex>
cudaError_t launch_bwd_t(const tg_raster_bwd_args& a, cudaStream_t s) {
    constexpr bool kTextured = Tex::kFormat != TG_TEX_NONE;
    constexpr bool kSmallRows = D == 3 || D == 4;  // channel counts with instances for the smaller rows
    const bool geo = bwd_geo(a);
    const bool mip = a.f.mip_levels > 0, aniso = a.f.filter == TG_FILTER_ANISO_BILINEAR;
    if (mip || aniso) {  // FP32 / BF16 storage and 3 or 4 channels only; one CTA per tile
        if constexpr (kSmallRows && (Tex::kFormat == TG_TEX_F32 || Tex::kFormat == TG_TEX_BF16)) {
            if (mip)
                return geo ? launch_bwd_kernel<D, Tex, false, FiltMip2, true>(a, 0.f, s)
                           : launch_bwd_kernel<D, Tex, false, FiltMip2, false>(a, 0.f, s);
            return geo ? launch_bwd_kernel<D, Tex, false, FiltAniso, true>(a, 0.f, s)
                       : launch_bwd_kernel<D, Tex, false, FiltAniso, false>(a, 0.f, s);
        }
        return cudaErrorInvalidValue;
    }
    if constexpr (kTextured)  // the bwd2 / exact adjoints take the instances that carry the UV term
        if (a.adjoint != TG_ADJ_REFERENCE)
            return launch_bwd_bilinear<D, Tex, FiltBilinearUV, true>(a, a.adjoint == TG_ADJ_BWD2 ? 1.f : 0.5f, s);
    if constexpr (kSmallRows)
        if (!geo) return launch_bwd_bilinear<D, Tex, FiltBilinear, false>(a, 0.f, s);
    return launch_bwd_bilinear<D, Tex, FiltBilinear, true>(a, 0.f, s);
}

template <class Tex>
cudaError_t launch_bwd_d(const tg_raster_bwd_args& a, cudaStream_t s) {
    switch (a.f.D) {
        case 1: return launch_bwd_t<1, Tex>(a, s);
        case 2: return launch_bwd_t<2, Tex>(a, s);
        case 3: return launch_bwd_t<3, Tex>(a, s);
        case 4: return launch_bwd_t<4, Tex>(a, s);
        case 5: return launch_bwd_t<5, Tex>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

template <class Tex>
cudaError_t launch_bwd_d34(const tg_raster_bwd_args& a, cudaStream_t s) {
    switch (a.f.D) {
        case 3: return launch_bwd_t<3, Tex>(a, s);
        case 4: return launch_bwd_t<4, Tex>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_raster_bwd(const tg_raster_bwd_args& a, cudaStream_t s) {
    switch (a.f.tex_format) {
        case TG_TEX_NONE: return launch_bwd_d<TexNone>(a, s);
        case TG_TEX_F32: return launch_bwd_d<TexF32>(a, s);
        case TG_TEX_BF16: return launch_bwd_d34<TexBF16>(a, s);
        case TG_TEX_F16: return launch_bwd_d34<TexF16>(a, s);
        case TG_TEX_FP8_E4M3: return launch_bwd_d34<TexFP8>(a, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace tg
