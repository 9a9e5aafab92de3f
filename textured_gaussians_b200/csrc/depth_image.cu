// Last step of the depth render modes, for sm_100a: the accumulated depth channel divided by the accumulated opacity
// (the expected depth), and world-space normals from a depth image: the normalised cross product of the central
// differences of the back-projected pixels, zero on the one-pixel border
// (textured_gaussians/rendering.py:1296-1313, utils.py:81-168).
//
// HBM-bound by need: 4 D + 4 bytes read and 4 D + 12 written a pixel.  As tensor expressions (rays, a batched product
// with K = 3, points, differences, cross, norm, padding) the step was some fifty small launches, which bound a whole
// training step of a plain 150,000-splat scene at 800x800: 2313 us a step.  Here each pixel of a 32x8 tile and its
// halo is back-projected once into shared memory and the differences are taken there, one launch of 17.7 us: 1794 us
// a step.
//
// Roundings follow the expressions one by one (a fused multiply-add only where the library's kernels have one): the
// differences of neighbouring points cancel, so an ulp in a point is far above an ulp in a normal.
#include "tg_common.cuh"

namespace tg {

constexpr int kDiW = 32, kDiH = 8;  // a CTA's tile; one thread per pixel

struct DepthCam {
    float R[9], t[3], fu, fv, cu, cv;
};
__device__ __forceinline__ DepthCam depth_cam(const tg_depth_image_args& a, int c) {
    DepthCam m;
    const float* M = a.camtoworlds + 16 * c;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int j = 0; j < 3; ++j) m.R[3 * i + j] = __ldg(M + 4 * i + j);
        m.t[i] = __ldg(M + 4 * i + 3);
    }
    const float* K = a.Ks + 9 * c;
    m.fu = __ldg(K), m.cu = __ldg(K + 2), m.fv = __ldg(K + 4), m.cv = __ldg(K + 5);
    return m;
}
__device__ __forceinline__ f3 depth_ray(const DepthCam& m, int x, int y) {
    const float u = __fdiv_rn(__fadd_rn(__fsub_rn((float)x, m.cu), 0.5f), m.fu);
    const float v = __fdiv_rn(__fadd_rn(__fsub_rn((float)y, m.cv), 0.5f), m.fv);
    f3 r;
    r.x = __fmaf_rn(m.R[2], 1.f, __fmaf_rn(m.R[1], v, __fmul_rn(m.R[0], u)));
    r.y = __fmaf_rn(m.R[5], 1.f, __fmaf_rn(m.R[4], v, __fmul_rn(m.R[3], u)));
    r.z = __fmaf_rn(m.R[8], 1.f, __fmaf_rn(m.R[7], v, __fmul_rn(m.R[6], u)));
    return r;
}
// The divisor of the expected depth (a NaN stays one).
__device__ __forceinline__ float depth_divisor(const tg_depth_image_args& a, int64_t p) {
    const float al = a.alphas[p];
    return al < 1e-10f ? 1e-10f : al;
}
__device__ __forceinline__ float depth_of(const tg_depth_image_args& a, int64_t p) {
    if (a.depth != nullptr) return a.depth[p];
    const float z = a.colors[p * a.D + a.D - 1];
    return a.alphas != nullptr ? __fdiv_rn(z, depth_divisor(a, p)) : z;
}
// Points of the tile at (x0, y0) with a halo of kHalo pixels into s (component planes); zero outside the image.
template <int kHalo>
__device__ __forceinline__ void stage_points(const tg_depth_image_args& a, const DepthCam& m, int64_t p0, int x0, int y0,
                                             float (*s)[(kDiH + 2 * kHalo) * (kDiW + 2 * kHalo)]) {
    constexpr int kW = kDiW + 2 * kHalo, kN = kW * (kDiH + 2 * kHalo);
    for (int i = threadIdx.x; i < kN; i += kDiW * kDiH) {
        const int x = x0 + i % kW - kHalo, y = y0 + i / kW - kHalo;
        f3 q = mk3(0.f, 0.f, 0.f);
        if (x >= 0 && x < a.width && y >= 0 && y < a.height) {
            const float z = depth_of(a, p0 + (int64_t)y * a.width + x);
            const f3 r = depth_ray(m, x, y);
            q.x = __fadd_rn(m.t[0], __fmul_rn(z, r.x));
            q.y = __fadd_rn(m.t[1], __fmul_rn(z, r.y));
            q.z = __fadd_rn(m.t[2], __fmul_rn(z, r.z));
        }
        s[0][i] = q.x, s[1][i] = q.y, s[2][i] = q.z;
    }
}
// Central differences around entry i of staged rows kW long, their cross product and its norm (at least 1e-12).
struct DepthNormal {
    f3 dr, dc, raw;
    float norm, d;
};
template <int kW, int kN>
__device__ __forceinline__ DepthNormal depth_normal(const float (*s)[kN], int i) {
    DepthNormal o;
    o.dr = mk3(__fsub_rn(s[0][i + kW], s[0][i - kW]), __fsub_rn(s[1][i + kW], s[1][i - kW]),
               __fsub_rn(s[2][i + kW], s[2][i - kW]));
    o.dc = mk3(__fsub_rn(s[0][i + 1], s[0][i - 1]), __fsub_rn(s[1][i + 1], s[1][i - 1]),
               __fsub_rn(s[2][i + 1], s[2][i - 1]));
    o.raw.x = __fmaf_rn(o.dr.y, o.dc.z, -__fmul_rn(o.dr.z, o.dc.y));
    o.raw.y = __fmaf_rn(o.dr.z, o.dc.x, -__fmul_rn(o.dr.x, o.dc.z));
    o.raw.z = __fmaf_rn(o.dr.x, o.dc.y, -__fmul_rn(o.dr.y, o.dc.x));
    o.norm = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(o.raw.x, o.raw.x), __fmul_rn(o.raw.z, o.raw.z)),
                                  __fmul_rn(o.raw.y, o.raw.y)));
    o.d = o.norm < 1e-12f ? 1e-12f : o.norm;
    return o;
}

// Grid: x over the tiles of a view, y over views.
__global__ void __launch_bounds__(kDiW * kDiH) depth_image_fwd_kernel(tg_depth_image_args a, int tiles_x) {
    constexpr int kW = kDiW + 2, kN = kW * (kDiH + 2);
    __shared__ float s[3][kN];
    const int c = blockIdx.y, x0 = blockIdx.x % tiles_x * kDiW, y0 = blockIdx.x / tiles_x * kDiH;
    const int lx = threadIdx.x % kDiW, ly = threadIdx.x / kDiW, x = x0 + lx, y = y0 + ly;
    const int64_t p0 = (int64_t)c * a.width * a.height, p = p0 + (int64_t)y * a.width + x;
    const bool inside = x < a.width && y < a.height;
    if (a.out_colors != nullptr && inside) {
        for (int k = 0; k + 1 < a.D; ++k) a.out_colors[p * a.D + k] = a.colors[p * a.D + k];
        a.out_colors[p * a.D + a.D - 1] = __fdiv_rn(a.colors[p * a.D + a.D - 1], depth_divisor(a, p));
    }
    if (a.out_normals == nullptr) return;
    const DepthCam m = depth_cam(a, c);
    stage_points<1>(a, m, p0, x0, y0, s);
    __syncthreads();
    if (!inside) return;
    f3 n = mk3(0.f, 0.f, 0.f);
    if (x >= 1 && x + 1 < a.width && y >= 1 && y + 1 < a.height) {
        const DepthNormal o = depth_normal<kW, kN>(s, (ly + 1) * kW + lx + 1);
        n = mk3(__fdiv_rn(o.raw.x, o.d), __fdiv_rn(o.raw.y, o.d), __fdiv_rn(o.raw.z, o.d));
    }
    a.out_normals[3 * p] = n.x;
    a.out_normals[3 * p + 1] = n.y;
    a.out_normals[3 * p + 2] = n.z;
}

// Adjoint: the gradients of the two differences at each pixel of the tile and its one-pixel halo into shared memory
// (points with a halo of two), then each pixel gathers those of its four neighbours (no atomics).
__global__ void __launch_bounds__(kDiW * kDiH) depth_image_bwd_kernel(tg_depth_image_args a, int tiles_x) {
    constexpr int kW = kDiW + 4, kN = kW * (kDiH + 4);
    constexpr int kGW = kDiW + 2, kGN = kGW * (kDiH + 2);
    __shared__ float s[3][kN];
    __shared__ float g[6][kGN];
    const int c = blockIdx.y, x0 = blockIdx.x % tiles_x * kDiW, y0 = blockIdx.x / tiles_x * kDiH;
    const int lx = threadIdx.x % kDiW, ly = threadIdx.x / kDiW, x = x0 + lx, y = y0 + ly;
    const int64_t p0 = (int64_t)c * a.width * a.height, p = p0 + (int64_t)y * a.width + x;
    const bool inside = x < a.width && y < a.height;
    float v_z = 0.f;
    if (a.v_normals != nullptr) {
        const DepthCam m = depth_cam(a, c);
        stage_points<2>(a, m, p0, x0, y0, s);
        __syncthreads();
        for (int i = threadIdx.x; i < kGN; i += kDiW * kDiH) {
            const int gx = x0 + i % kGW - 1, gy = y0 + i / kGW - 1;
            f3 v_dr = mk3(0.f, 0.f, 0.f), v_dc = v_dr;
            if (gx >= 1 && gx + 1 < a.width && gy >= 1 && gy + 1 < a.height) {
                const DepthNormal o = depth_normal<kW, kN>(s, (i / kGW + 1) * kW + i % kGW + 1);
                const float* up = a.v_normals + 3 * (p0 + (int64_t)gy * a.width + gx);
                const f3 v = mk3(up[0], up[1], up[2]);
                const float inv = 1.f / o.d;
                f3 w = v;
                if (o.norm >= 1e-12f) {
                    const f3 n = inv * o.raw;
                    w = v - dot(v, n) * n;
                }
                w = inv * w;
                v_dr = cross(o.dc, w);
                v_dc = cross(w, o.dr);
            }
            g[0][i] = v_dr.x, g[1][i] = v_dr.y, g[2][i] = v_dr.z;
            g[3][i] = v_dc.x, g[4][i] = v_dc.y, g[5][i] = v_dc.z;
        }
        __syncthreads();
        if (inside) {
            const int i = (ly + 1) * kGW + lx + 1;
            f3 v = mk3(0.f, 0.f, 0.f);
            v.x = (g[0][i - kGW] - g[0][i + kGW]) + (g[3][i - 1] - g[3][i + 1]);
            v.y = (g[1][i - kGW] - g[1][i + kGW]) + (g[4][i - 1] - g[4][i + 1]);
            v.z = (g[2][i - kGW] - g[2][i + kGW]) + (g[5][i - 1] - g[5][i + 1]);
            v_z = dot(depth_ray(m, x, y), v);
        }
    }
    if (!inside) return;
    if (a.depth != nullptr) {
        if (a.v_depth != nullptr) a.v_depth[p] = v_z;
        v_z = 0.f;
    }
    if (a.v_colors == nullptr) return;
    const float* up = a.v_out_colors != nullptr ? a.v_out_colors + p * a.D : nullptr;
    for (int k = 0; k + 1 < a.D; ++k) a.v_colors[p * a.D + k] = up != nullptr ? up[k] : 0.f;
    if (up != nullptr) v_z += up[a.D - 1];
    if (a.alphas != nullptr) {
        const float div = depth_divisor(a, p), z = a.colors[p * a.D + a.D - 1] / div;
        if (a.v_alphas != nullptr) a.v_alphas[p] = a.alphas[p] < 1e-10f ? 0.f : -v_z * (z / div);
        v_z = v_z / div;
    }
    a.v_colors[p * a.D + a.D - 1] = v_z;
}

cudaError_t launch_depth_image(const tg_depth_image_args& a, bool adjoint, cudaStream_t s) {
    const int64_t tx = (a.width + kDiW - 1) / kDiW, ty = (a.height + kDiH - 1) / kDiH;
    if (tx * ty > 0x7fffffff) return cudaErrorInvalidValue;
    const dim3 grid((unsigned)(tx * ty), (unsigned)a.C);
    if (adjoint)
        depth_image_bwd_kernel<<<grid, kDiW * kDiH, 0, s>>>(a, (int)tx);
    else
        depth_image_fwd_kernel<<<grid, kDiW * kDiH, 0, s>>>(a, (int)tx);
    note_launches(1);
    return cudaGetLastError();
}

}  // namespace tg
