// Intrinsics resample: the 2-D homography warp of the reference's
// camera/homography.py:6-58. Destination pixel (x, y) of batch b samples the
// source image at p = H_b (x, y, 1) after the perspective divide, bilinearly,
// with align_corners semantics (pixel centres at integer coordinates 0..W-1,
// 0..H-1) and zero padding per corner.
//
// Forward: one thread per destination pixel, all channels (the source
// position is shared by the channels). Adjoint: the image gradient scattered
// to the four corners with atomics (caller-zeroed), and the homography
// gradient through the bilinear position derivative and the perspective
// divide, reduced per CTA in a fixed order and per batch element by a second
// kernel (deterministic).
#include <cuda_runtime.h>

#include "../../include/nanodrr_gb300.h"

namespace ndrr {

constexpr int kHomBlock = 256;

struct HomTap {
    float a, b, c;    // H (x, y, 1)
    float sx, sy;     // source position
    int x0, y0;
    float fx, fy;
};

__device__ __forceinline__ HomTap hom_tap(const float* __restrict__ Hm, int x, int y) {
    HomTap t;
    const float fx = (float)x, fy = (float)y;
    t.a = fmaf(__ldg(Hm + 0), fx, fmaf(__ldg(Hm + 1), fy, __ldg(Hm + 2)));
    t.b = fmaf(__ldg(Hm + 3), fx, fmaf(__ldg(Hm + 4), fy, __ldg(Hm + 5)));
    t.c = fmaf(__ldg(Hm + 6), fx, fmaf(__ldg(Hm + 7), fy, __ldg(Hm + 8)));
    t.sx = t.a / t.c;
    t.sy = t.b / t.c;
    // Clamp far-outside positions before the float -> int conversion: beyond
    // one pixel outside the image every corner is zero padding either way.
    const float cx = fminf(fmaxf(t.sx, -2.0f), 1.0e8f), cy = fminf(fmaxf(t.sy, -2.0f), 1.0e8f);
    const float xf = floorf(cx), yf = floorf(cy);
    t.x0 = (int)xf;
    t.y0 = (int)yf;
    t.fx = cx - xf;
    t.fy = cy - yf;
    return t;
}

__global__ void __launch_bounds__(kHomBlock) homography_fwd_kernel(const float* __restrict__ img,
                                                                   const float* __restrict__ hom,
                                                                   float* __restrict__ out, int C, int H, int W) {
    const int b = blockIdx.y;
    const int pix = blockIdx.x * kHomBlock + threadIdx.x;
    if (pix >= H * W) return;
    const int x = pix % W, y = pix / W;
    const HomTap t = hom_tap(hom + (size_t)b * 9, x, y);
    const bool okx0 = t.x0 >= 0 && t.x0 <= W - 1, okx1 = t.x0 + 1 >= 0 && t.x0 + 1 <= W - 1;
    const bool oky0 = t.y0 >= 0 && t.y0 <= H - 1, oky1 = t.y0 + 1 >= 0 && t.y0 + 1 <= H - 1;
    const float w00 = (1.f - t.fx) * (1.f - t.fy), w01 = t.fx * (1.f - t.fy);
    const float w10 = (1.f - t.fx) * t.fy, w11 = t.fx * t.fy;
    const size_t plane = (size_t)H * W;
    for (int c = 0; c < C; ++c) {
        const float* im = img + ((size_t)b * C + c) * plane;
        float v = 0.f;
        if (oky0 && okx0) v = fmaf(w00, __ldg(im + (size_t)t.y0 * W + t.x0), v);
        if (oky0 && okx1) v = fmaf(w01, __ldg(im + (size_t)t.y0 * W + t.x0 + 1), v);
        if (oky1 && okx0) v = fmaf(w10, __ldg(im + (size_t)(t.y0 + 1) * W + t.x0), v);
        if (oky1 && okx1) v = fmaf(w11, __ldg(im + (size_t)(t.y0 + 1) * W + t.x0 + 1), v);
        out[((size_t)b * C + c) * plane + pix] = v;
    }
}

__global__ void __launch_bounds__(kHomBlock) homography_bwd_kernel(const float* __restrict__ go,
                                                                   const float* __restrict__ img,
                                                                   const float* __restrict__ hom,
                                                                   float* __restrict__ gimg,
                                                                   float* __restrict__ partials, int C, int H, int W) {
    __shared__ float red[kHomBlock / 32][9];
    const int b = blockIdx.y;
    const int pix = blockIdx.x * kHomBlock + threadIdx.x;
    float gh[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) gh[j] = 0.f;
    if (pix < H * W) {
        const int x = pix % W, y = pix / W;
        const HomTap t = hom_tap(hom + (size_t)b * 9, x, y);
        const bool okx0 = t.x0 >= 0 && t.x0 <= W - 1, okx1 = t.x0 + 1 >= 0 && t.x0 + 1 <= W - 1;
        const bool oky0 = t.y0 >= 0 && t.y0 <= H - 1, oky1 = t.y0 + 1 >= 0 && t.y0 + 1 <= H - 1;
        const float w00 = (1.f - t.fx) * (1.f - t.fy), w01 = t.fx * (1.f - t.fy);
        const float w10 = (1.f - t.fx) * t.fy, w11 = t.fx * t.fy;
        const size_t plane = (size_t)H * W;
        float dsx = 0.f, dsy = 0.f;
        for (int c = 0; c < C; ++c) {
            const size_t base = ((size_t)b * C + c) * plane;
            const float g = __ldg(go + base + pix);
            if (g == 0.f) continue;
            const float* im = img + base;
            const float v00 = (oky0 && okx0) ? __ldg(im + (size_t)t.y0 * W + t.x0) : 0.f;
            const float v01 = (oky0 && okx1) ? __ldg(im + (size_t)t.y0 * W + t.x0 + 1) : 0.f;
            const float v10 = (oky1 && okx0) ? __ldg(im + (size_t)(t.y0 + 1) * W + t.x0) : 0.f;
            const float v11 = (oky1 && okx1) ? __ldg(im + (size_t)(t.y0 + 1) * W + t.x0 + 1) : 0.f;
            // derivative of the bilinear interpolant in the source position
            dsx = fmaf(g, (1.f - t.fy) * (v01 - v00) + t.fy * (v11 - v10), dsx);
            dsy = fmaf(g, (1.f - t.fx) * (v10 - v00) + t.fx * (v11 - v01), dsy);
            if (gimg != nullptr) {
                float* gi = gimg + base;
                if (oky0 && okx0) atomicAdd(gi + (size_t)t.y0 * W + t.x0, g * w00);
                if (oky0 && okx1) atomicAdd(gi + (size_t)t.y0 * W + t.x0 + 1, g * w01);
                if (oky1 && okx0) atomicAdd(gi + (size_t)(t.y0 + 1) * W + t.x0, g * w10);
                if (oky1 && okx1) atomicAdd(gi + (size_t)(t.y0 + 1) * W + t.x0 + 1, g * w11);
            }
        }
        // Positions clamped above had a zero derivative in the reference too:
        // every corner there is padding, so dsx = dsy = 0 already.
        // sx = a / c, sy = b / c; p = (x, y, 1)
        const float inv_c = 1.f / t.c;
        const float ga = dsx * inv_c, gb = dsy * inv_c;
        const float gc = -(dsx * t.sx + dsy * t.sy) * inv_c;
        const float p[3] = {(float)x, (float)y, 1.f};
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            gh[j] = ga * p[j];
            gh[3 + j] = gb * p[j];
            gh[6 + j] = gc * p[j];
        }
    }
    if (partials == nullptr) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < 9; ++j) {
        float v = gh[j];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][j] = v;
    }
    __syncthreads();
    if (threadIdx.x < 9) {
        float s = 0.f;
        for (int w = 0; w < kHomBlock / 32; ++w) s += red[w][threadIdx.x];
        partials[((size_t)b * gridDim.x + blockIdx.x) * 9 + threadIdx.x] = s;
    }
}

// Per-batch fixed-order sum of the CTA partials into ghom [B, 3, 3]: each
// thread takes a strided share in double, then a shuffle tree (one thread per
// entry walking all 1024 partials of a 512^2 image took 22 us).
// With `k_old`, ghom is not written but chained to the two inverse intrinsics
// of H = inv(k_old) k_new (float64): g_new = A^T g, g_old = -A^T (g k_new^T)
// A^T with A = inv(k_old).
constexpr int kHomReduce = 128;

__device__ __forceinline__ void inverse3(const double (&m)[9], double (&r)[9]) {
    r[0] = m[4] * m[8] - m[5] * m[7];
    r[1] = m[2] * m[7] - m[1] * m[8];
    r[2] = m[1] * m[5] - m[2] * m[4];
    r[3] = m[5] * m[6] - m[3] * m[8];
    r[4] = m[0] * m[8] - m[2] * m[6];
    r[5] = m[2] * m[3] - m[0] * m[5];
    r[6] = m[3] * m[7] - m[4] * m[6];
    r[7] = m[1] * m[6] - m[0] * m[7];
    r[8] = m[0] * m[4] - m[1] * m[3];
    const double inv = 1.0 / (m[0] * r[0] + m[1] * r[3] + m[2] * r[6]);
    for (int i = 0; i < 9; ++i) r[i] *= inv;
}

__global__ void __launch_bounds__(kHomReduce) homography_reduce_kernel(const float* __restrict__ partials, int nblk,
                                                                       float* __restrict__ ghom,
                                                                       const float* __restrict__ k_old, int n_old,
                                                                       const float* __restrict__ k_new, int n_new,
                                                                       float* __restrict__ g_old,
                                                                       float* __restrict__ g_new) {
    __shared__ double red[kHomReduce / 32][9];
    __shared__ double g[9], A[9], t[9];
    const int b = blockIdx.x, j = threadIdx.x;
    double s[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) s[k] = 0.0;
    for (int i = threadIdx.x; i < nblk; i += kHomReduce)
#pragma unroll
        for (int k = 0; k < 9; ++k) s[k] += (double)partials[((size_t)b * nblk + i) * 9 + k];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
        if ((j & 31) == 0) red[j >> 5][k] = s[k];
    }
    __syncthreads();
    if (j < 9) {
        double v = red[0][j];
        for (int w = 1; w < kHomReduce / 32; ++w) v += red[w][j];
        g[j] = v;
        if (ghom != nullptr) ghom[(size_t)b * 9 + j] = (float)v;
    }
    if (k_old == nullptr) return;
    const float* ko = k_old + (n_old == 1 ? 0 : (size_t)b * 9);
    const float* kn = k_new + (n_new == 1 ? 0 : (size_t)b * 9);
    if (j == 32) {
        double m[9], r[9];
        for (int i = 0; i < 9; ++i) m[i] = (double)ko[i];
        inverse3(m, r);
        for (int i = 0; i < 9; ++i) A[i] = r[i];
    }
    __syncthreads();
    if (j >= 9) return;
    const int r = j / 3, c = j % 3;
    const unsigned lanes = 0x1ffu;  // the nine threads that go on
    double v = 0.0, u = 0.0;
    for (int i = 0; i < 3; ++i) {
        v += A[3 * i + r] * g[3 * i + c];                   // A^T g
        u += g[3 * r + i] * (double)kn[3 * c + i];          // g k_new^T
    }
    g_new[(size_t)b * 9 + j] = (float)v;
    t[j] = u;
    __syncwarp(lanes);
    double w = 0.0;
    for (int i = 0; i < 3; ++i) w += A[3 * i + r] * t[3 * i + c];  // A^T (g k_new^T)
    __syncwarp(lanes);
    t[j] = w;
    __syncwarp(lanes);
    double x = 0.0;
    for (int i = 0; i < 3; ++i) x += t[3 * r + i] * A[3 * c + i];  // ... A^T
    g_old[(size_t)b * 9 + j] = (float)-x;
}

// H = inv(k_old) k_new per batch element, one thread each: the float32
// cofactor inverse and products in the order of the tensor expression
// (homography.py::_inv3, mm_small), so the homography is bitwise its.
__global__ void __launch_bounds__(32) homography_matrix_kernel(const float* __restrict__ k_old, int n_old,
                                                               const float* __restrict__ k_new, int n_new, int B,
                                                               float* __restrict__ hom) {
    const int t = blockIdx.x * 32 + threadIdx.x;
    if (t >= B) return;
    const float* m = k_old + (n_old == 1 ? 0 : (size_t)t * 9);
    const float* q = k_new + (n_new == 1 ? 0 : (size_t)t * 9);
    const float a = m[0], b = m[1], c = m[2], d = m[3], e = m[4], f = m[5], g = m[6], h = m[7], i = m[8];
    auto minor = [](float w, float x, float y, float z) { return __fsub_rn(__fmul_rn(w, x), __fmul_rn(y, z)); };
    float co[9] = {minor(e, i, f, h), minor(c, h, b, i), minor(b, f, c, e), minor(f, g, d, i), minor(a, i, c, g),
                   minor(c, d, a, f), minor(d, h, e, g), minor(b, g, a, h), minor(a, e, b, d)};
    const float det = __fadd_rn(__fadd_rn(__fmul_rn(a, co[0]), __fmul_rn(b, co[3])), __fmul_rn(c, co[6]));
#pragma unroll
    for (int k = 0; k < 9; ++k) co[k] = __fdiv_rn(co[k], det);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            hom[(size_t)t * 9 + 3 * r + k] =
                __fadd_rn(__fadd_rn(__fmul_rn(co[3 * r], q[k]), __fmul_rn(co[3 * r + 1], q[3 + k])),
                          __fmul_rn(co[3 * r + 2], q[6 + k]));
}

cudaError_t launch_homography_matrix(const float* k_old, int n_old, const float* k_new, int n_new, int B, float* hom,
                                     cudaStream_t st) {
    homography_matrix_kernel<<<(B + 31) / 32, 32, 0, st>>>(k_old, n_old, k_new, n_new, B, hom);
    return cudaGetLastError();
}

int homography_blocks(int H, int W) { return (H * W + kHomBlock - 1) / kHomBlock; }

cudaError_t launch_homography_fwd(const float* img, const float* hom, int B, int C, int H, int W, float* out,
                                  cudaStream_t st) {
    const dim3 grid((unsigned)homography_blocks(H, W), (unsigned)B);
    homography_fwd_kernel<<<grid, kHomBlock, 0, st>>>(img, hom, out, C, H, W);
    return cudaGetLastError();
}

cudaError_t launch_homography_bwd(const float* go, const float* img, const float* hom, int B, int C, int H, int W,
                                  float* gimg, float* ghom, float* partials, const float* k_old, int n_old,
                                  const float* k_new, int n_new, float* g_old, float* g_new, cudaStream_t st) {
    const int nblk = homography_blocks(H, W);
    const dim3 grid((unsigned)nblk, (unsigned)B);
    const bool reduce = ghom != nullptr || k_old != nullptr;
    homography_bwd_kernel<<<grid, kHomBlock, 0, st>>>(go, img, hom, gimg, reduce ? partials : nullptr, C, H, W);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !reduce) return e;
    homography_reduce_kernel<<<B, kHomReduce, 0, st>>>(partials, nblk, ghom, k_old, n_old, k_new, n_new, g_old, g_new);
    return cudaGetLastError();
}

}  // namespace ndrr
