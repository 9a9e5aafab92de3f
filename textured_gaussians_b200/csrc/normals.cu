// Camera-space normal images to world space, for sm_100a.
//
// out[p] = A_c n[p] for the pixels p of view c, A_c the upper-left 3x3 block of the inverse of the view matrix (the
// renderer's last step; its adjoint is the same pass with the block transposed).  HBM-bound: 24 bytes a pixel.  As
// a batched matrix product with K = 3 the library's SGEMM took 503 us for four 1600x1200 views, and the batched LU
// inverse before it nine launches; this pass is one launch.  Each CTA inverts its view's matrix
// itself (one thread, FP64 cofactors, about a microsecond, hidden behind the other CTAs' copies).
#include "tg_common.cuh"

namespace tg {

constexpr int kNrmThreads = 256;
constexpr int kNrmItems = 4;  // float4 vectors of the [pixels, 3] image per thread and step: three hold four pixels

// Upper-left 3x3 of the inverse of the row-major 4x4 matrix m, in FP64.
__device__ void inverse_block(const float* __restrict__ m, float* A) {
    double a[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) a[i] = (double)m[i];
    // 2x2 minors of the two row pairs
    const double s0 = a[0] * a[5] - a[4] * a[1], s1 = a[0] * a[6] - a[4] * a[2], s2 = a[0] * a[7] - a[4] * a[3];
    const double s3 = a[1] * a[6] - a[5] * a[2], s4 = a[1] * a[7] - a[5] * a[3], s5 = a[2] * a[7] - a[6] * a[3];
    const double c5 = a[10] * a[15] - a[14] * a[11], c4 = a[9] * a[15] - a[13] * a[11];
    const double c3 = a[9] * a[14] - a[13] * a[10], c2 = a[8] * a[15] - a[12] * a[11];
    const double c1 = a[8] * a[14] - a[12] * a[10], c0 = a[8] * a[13] - a[12] * a[9];
    const double inv = 1.0 / (s0 * c5 - s1 * c4 + s2 * c3 + s3 * c2 - s4 * c1 + s5 * c0);
    A[0] = (float)((a[5] * c5 - a[6] * c4 + a[7] * c3) * inv);
    A[1] = (float)((-a[1] * c5 + a[2] * c4 - a[3] * c3) * inv);
    A[2] = (float)((a[13] * s5 - a[14] * s4 + a[15] * s3) * inv);
    A[3] = (float)((-a[4] * c5 + a[6] * c2 - a[7] * c1) * inv);
    A[4] = (float)((a[0] * c5 - a[2] * c2 + a[3] * c1) * inv);
    A[5] = (float)((-a[12] * s5 + a[14] * s2 - a[15] * s1) * inv);
    A[6] = (float)((a[4] * c4 - a[5] * c2 + a[7] * c0) * inv);
    A[7] = (float)((-a[0] * c4 + a[1] * c2 - a[3] * c0) * inv);
    A[8] = (float)((a[12] * s4 - a[13] * s2 + a[15] * s0) * inv);
}

// Grid: x over chunks of 1024 pixels of a view, y over views.
__global__ void __launch_bounds__(kNrmThreads) rotate_normals_kernel(const float* __restrict__ viewmats,
                                                                     const tg_view* __restrict__ views,
                                                                     int64_t view_pixels, int64_t n_pixels,
                                                                     int transpose, const float* __restrict__ in,
                                                                     float* __restrict__ out) {
    constexpr int kChunk = kNrmThreads * kNrmItems;
    __shared__ float A[9];
    __shared__ float4 s4[kChunk * 3 / 4];
    const int c = blockIdx.y;
    int64_t base = (int64_t)c * view_pixels, count = view_pixels;
    if (views != nullptr) {
        base = views[c].pix_base;
        count = (int64_t)views[c].width * views[c].height;
    }
    const int64_t p0 = (int64_t)blockIdx.x * kChunk;
    // (a malformed view table stays inside the image)
    const int64_t left = min(count - p0, n_pixels - base - p0);
    if (left <= 0 || base < 0) return;
    const int n = (int)min(left, (int64_t)kChunk) * 3;
    const int64_t f0 = (base + p0) * 3;  // first float
    float* s = reinterpret_cast<float*>(s4);
    // aligned whole chunks move as vectors, ragged ones as floats
    const bool vec = (f0 & 3) == 0 && n == kChunk * 3 &&
                     ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    if (vec) {
#pragma unroll
        for (int k = 0; k < 3; ++k)
            s4[threadIdx.x + k * kNrmThreads] = __ldg(reinterpret_cast<const float4*>(in + f0) + threadIdx.x + k * kNrmThreads);
    } else {
        for (int k = threadIdx.x; k < n; k += kNrmThreads) s[k] = in[f0 + k];
    }
    if (threadIdx.x == 0) inverse_block(viewmats + 16 * c, A);
    __syncthreads();
    float a[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) a[k] = transpose ? A[(k % 3) * 3 + k / 3] : A[k];
    for (int p = threadIdx.x; 3 * p < n; p += kNrmThreads) {  // stride 3: no bank conflicts
        const float x = s[3 * p], y = s[3 * p + 1], z = s[3 * p + 2];
        s[3 * p] = a[0] * x + a[1] * y + a[2] * z;
        s[3 * p + 1] = a[3] * x + a[4] * y + a[5] * z;
        s[3 * p + 2] = a[6] * x + a[7] * y + a[8] * z;
    }
    __syncthreads();
    if (vec) {
#pragma unroll
        for (int k = 0; k < 3; ++k)
            reinterpret_cast<float4*>(out + f0)[threadIdx.x + k * kNrmThreads] = s4[threadIdx.x + k * kNrmThreads];
    } else {
        for (int k = threadIdx.x; k < n; k += kNrmThreads) out[f0 + k] = s[k];
    }
}

cudaError_t launch_rotate_normals(const float* viewmats, int C, const tg_view* views, int64_t view_pixels,
                                  int64_t n_pixels, int transpose, const float* in, float* out, cudaStream_t s) {
    if (C == 0 || view_pixels == 0 || n_pixels == 0) return cudaSuccess;
    const int64_t chunks = (view_pixels + kNrmThreads * kNrmItems - 1) / (kNrmThreads * kNrmItems);
    if (chunks > 0x7fffffff || C > 65535) return cudaErrorInvalidValue;
    rotate_normals_kernel<<<dim3((unsigned)chunks, (unsigned)C), kNrmThreads, 0, s>>>(viewmats, views, view_pixels,
                                                                                      n_pixels, transpose, in, out);
    note_launches(1);
    return cudaGetLastError();
}

}  // namespace tg
