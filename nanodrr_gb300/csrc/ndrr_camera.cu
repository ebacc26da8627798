// Camera-space ray endpoints of a detector in one launch: the reference's
// _make_tgt / _make_src (src/nanodrr/drr/renderer.py:101-132), which as
// tensor expressions take a dozen small launches per render call.
//
// tgt[b, n] = sdd[b] * (K0 * (u + 0.5) + K1 * (v + 0.5) + K2), n = v * W + u,
// where Kc is column c of K^-1[b]; every product and sum is rounded on its
// own and summed left to right, the order of the broadcast expression
// (renderer.py::_make_tgt), so the rays are bitwise those of the tensor path.
// src is the camera origin ([B, 1, 3] zeros) for a pinhole, or tgt with
// z - sdd ([B, N, 3]) for parallel rays.
#include <cuda_runtime.h>

#include "ndrr_launch.h"

namespace ndrr {

__global__ void __launch_bounds__(256) camera_rays_kernel(const float* __restrict__ k_inv, int k_stride,
                                                          const float* __restrict__ sdd, int s_stride, int B,
                                                          int height, int width, int orthographic,
                                                          float* __restrict__ src, float* __restrict__ tgt) {
    const long long N = (long long)height * width;
    const long long total = (long long)B * N;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int b = (int)(i / N);
        const long long n = i - (long long)b * N;
        const int v = (int)(n / width), u = (int)(n - (long long)v * width);
        const float uf = __fadd_rn((float)u, 0.5f), vf = __fadd_rn((float)v, 0.5f);
        const float* k = k_inv + (long long)b * k_stride;
        const float s = sdd[(long long)b * s_stride];
        float t[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            // K[r,2] * 1 is exact, so the third term adds K[r,2] itself.
            const float ray = __fadd_rn(__fadd_rn(__fmul_rn(k[3 * r + 0], uf), __fmul_rn(k[3 * r + 1], vf)), k[3 * r + 2]);
            t[r] = __fmul_rn(s, ray);
        }
        float* o = tgt + 3 * i;
        o[0] = t[0];
        o[1] = t[1];
        o[2] = t[2];
        if (orthographic) {
            float* p = src + 3 * i;
            p[0] = t[0];
            p[1] = t[1];
            p[2] = __fsub_rn(t[2], s);
        } else if (n == 0) {
            float* p = src + 3 * (long long)b;
            p[0] = 0.f;
            p[1] = 0.f;
            p[2] = 0.f;
        }
    }
}

// The whole ray set-up of a render call in one launch: endpoints as above,
// expanded to the pose batch, and the camera-space sample spacing
// |tgt - src| / (S - 1), rounded as the tensor expression rounds it (the
// three squares added first and third, then second, and the division by a
// scalar as a product with its reciprocal), so the rays are bitwise its.
// Writing 16 B per ray is the bound; as tensor operations it was six more
// launches and three passes over the rays.
__device__ __forceinline__ void setup_ray(const float* k, float s, float uf, float vf, float (&ray)[3],
                                          float (&t)[3]) {
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        ray[r] = __fadd_rn(__fadd_rn(__fmul_rn(k[3 * r + 0], uf), __fmul_rn(k[3 * r + 1], vf)), k[3 * r + 2]);
        t[r] = __fmul_rn(s, ray[r]);
    }
}

__device__ __forceinline__ float ray_norm(float x, float y, float z) {
    return __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(z, z)), __fmul_rn(y, y)));
}

__global__ void __launch_bounds__(256) ray_setup_kernel(const float* __restrict__ k_inv, int k_stride,
                                                        const float* __restrict__ sdd, int s_stride, int N, int width,
                                                        int orthographic, float inv_s, float* __restrict__ src,
                                                        float* __restrict__ tgt, float* __restrict__ step) {
    const int b = blockIdx.y, n = blockIdx.x * 256 + threadIdx.x;
    if (n >= N) return;
    const int v = n / width, u = n - v * width;
    const float s = __ldg(sdd + (size_t)b * s_stride);
    float k[9], ray[3], t[3];
#pragma unroll
    for (int j = 0; j < 9; ++j) k[j] = __ldg(k_inv + (size_t)b * k_stride + j);
    setup_ray(k, s, __fadd_rn((float)u, 0.5f), __fadd_rn((float)v, 0.5f), ray, t);
    const size_t i = (size_t)b * N + n;
    tgt[3 * i + 0] = t[0];
    tgt[3 * i + 1] = t[1];
    tgt[3 * i + 2] = t[2];
    float e[3] = {t[0], t[1], t[2]};
    if (orthographic) {
        const float z = __fsub_rn(t[2], s);
        src[3 * i + 0] = t[0];
        src[3 * i + 1] = t[1];
        src[3 * i + 2] = z;
        e[0] = __fsub_rn(t[0], t[0]);
        e[1] = __fsub_rn(t[1], t[1]);
        e[2] = __fsub_rn(t[2], z);
    } else if (n == 0) {
        src[3 * (size_t)b + 0] = 0.f;
        src[3 * (size_t)b + 1] = 0.f;
        src[3 * (size_t)b + 2] = 0.f;
    }
    step[i] = __fmul_rn(ray_norm(e[0], e[1], e[2]), inv_s);
}

// Adjoint of the set-up: per ray, the gradient g of the target (its own, the
// spacing's along the ray and, for parallel rays, the source's), then
// dL/dK^-1[r][c] = sum sdd g_r (u, v, 1)_c and dL/dsdd = sum g . ray. A CTA
// sums kSetupRays rays in a fixed order; the second kernel sums the CTAs.
constexpr int kSetupRays = 2048;

__global__ void __launch_bounds__(256) ray_setup_bwd_kernel(const float* __restrict__ k_inv, int k_stride,
                                                            const float* __restrict__ sdd, int s_stride, int N,
                                                            int width, int orthographic, float inv_s,
                                                            const float* __restrict__ gsrc,
                                                            const float* __restrict__ gtgt,
                                                            const float* __restrict__ gstep,
                                                            float* __restrict__ partials) {
    __shared__ float red[8][10];
    const int b = blockIdx.y;
    const float s = __ldg(sdd + (size_t)b * s_stride);
    float k[9], acc[10];
#pragma unroll
    for (int j = 0; j < 9; ++j) k[j] = __ldg(k_inv + (size_t)b * k_stride + j);
#pragma unroll
    for (int j = 0; j < 10; ++j) acc[j] = 0.f;
    const int end = min(N, (int)(blockIdx.x + 1) * kSetupRays);
    for (int n = blockIdx.x * kSetupRays + threadIdx.x; n < end; n += 256) {
        const int v = n / width, u = n - v * width;
        const float uf = (float)u + 0.5f, vf = (float)v + 0.5f;
        float ray[3], t[3], g[3] = {0.f, 0.f, 0.f}, gs = 0.f;
        setup_ray(k, s, uf, vf, ray, t);
        const size_t i = (size_t)b * N + n;
        if (gtgt != nullptr)
#pragma unroll
            for (int r = 0; r < 3; ++r) g[r] = __ldg(gtgt + 3 * i + r);
        const float gl = gstep != nullptr ? __ldg(gstep + i) * inv_s : 0.f;
        if (orthographic) {
            // the spacing is |sdd|: its gradients through tgt and src cancel
            if (gsrc != nullptr) {
#pragma unroll
                for (int r = 0; r < 3; ++r) g[r] += __ldg(gsrc + 3 * i + r);
                gs -= __ldg(gsrc + 3 * i + 2);
            }
            const float e = t[2] - __fsub_rn(t[2], s);
            gs += e > 0.f ? gl : (e < 0.f ? -gl : 0.f);
        } else {
            const float len = ray_norm(t[0], t[1], t[2]);
            const float w = len > 0.f ? gl / len : 0.f;
#pragma unroll
            for (int r = 0; r < 3; ++r) g[r] = fmaf(w, t[r], g[r]);
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const float h = s * g[r];
            acc[3 * r + 0] = fmaf(h, uf, acc[3 * r + 0]);
            acc[3 * r + 1] = fmaf(h, vf, acc[3 * r + 1]);
            acc[3 * r + 2] += h;
        }
        acc[9] += fmaf(g[0], ray[0], fmaf(g[1], ray[1], fmaf(g[2], ray[2], gs)));
    }
#pragma unroll
    for (int j = 0; j < 10; ++j) {
        float x = acc[j];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][j] = x;
    }
    __syncthreads();
    if (threadIdx.x < 10) {
        float x = red[0][threadIdx.x];
        for (int w = 1; w < 8; ++w) x += red[w][threadIdx.x];
        partials[((size_t)b * gridDim.x + blockIdx.x) * 10 + threadIdx.x] = x;
    }
}

__global__ void __launch_bounds__(320) ray_setup_reduce_kernel(const float* __restrict__ partials, int blocks,
                                                               float* __restrict__ g_k, float* __restrict__ g_s) {
    const int b = blockIdx.x, j = threadIdx.x >> 5, lane = threadIdx.x & 31;  // a warp per term
    double x = 0.0;
    for (int i = lane; i < blocks; i += 32) x += (double)partials[((size_t)b * blocks + i) * 10 + j];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane != 0) return;
    if (j < 9)
        g_k[(size_t)b * 9 + j] = (float)x;
    else
        g_s[b] = (float)x;
}

// The camera -> voxel affine M = (world_to_voxel @ rt_inv)[:3] in float32,
// each product and sum rounded in the order of the broadcast expression
// (renderer.py::_affine_product), and with M_lo the float64 product's
// remainder, in one launch instead of a dozen; one thread per entry.
__global__ void __launch_bounds__(96) camera_affine_kernel(const float* __restrict__ w2v,
                                                           const float* __restrict__ rt, int B,
                                                           float* __restrict__ M, float* __restrict__ M_lo) {
    const int t = blockIdx.x * 96 + threadIdx.x;
    if (t >= B * 12) return;
    const int b = t / 12, i = (t % 12) / 4, j = t % 4;
    float m = 0.f;
    double d = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float x = __ldg(w2v + 4 * i + k), y = __ldg(rt + (size_t)b * 16 + 4 * k + j);
        m = __fadd_rn(m, __fmul_rn(x, y));
        d = __dadd_rn(d, __dmul_rn((double)x, (double)y));
    }
    M[t] = m;
    if (M_lo != nullptr) M_lo[t] = (float)(d - (double)m);
}

// Its adjoint: g_rt[k][j] = sum_i world_to_voxel[i][k] gM[i][j], rows summed
// in order.
__global__ void __launch_bounds__(128) camera_affine_bwd_kernel(const float* __restrict__ w2v,
                                                                const float* __restrict__ gM, int B,
                                                                float* __restrict__ g_rt) {
    const int t = blockIdx.x * 128 + threadIdx.x;
    if (t >= B * 16) return;
    const int b = t / 16, k = (t % 16) / 4, j = t % 4;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i)
        s = __fadd_rn(s, __fmul_rn(__ldg(w2v + 4 * i + k), __ldg(gM + (size_t)b * 12 + 4 * i + j)));
    g_rt[t] = s;
}

static dim3 setup_grid(int N, int rays, int B) { return dim3((unsigned)((N + rays - 1) / rays), (unsigned)B); }

cudaError_t launch_ray_setup(const float* k_inv, int n_k, const float* sdd, int n_s, int B, int height, int width,
                             int orthographic, int n_samples, float* src, float* tgt, float* step, cudaStream_t st) {
    const int N = height * width;
    ray_setup_kernel<<<setup_grid(N, 256, B), 256, 0, st>>>(k_inv, n_k == 1 ? 0 : 9, sdd, n_s == 1 ? 0 : 1, N, width,
                                                            orthographic, 1.0f / (float)(n_samples - 1), src, tgt,
                                                            step);
    return cudaGetLastError();
}

uint64_t ray_setup_workspace_bytes(int B, int height, int width) {
    return (uint64_t)B * ((height * width + kSetupRays - 1) / kSetupRays) * 10 * sizeof(float);
}

cudaError_t launch_ray_setup_bwd(const float* k_inv, int n_k, const float* sdd, int n_s, int B, int height, int width,
                                 int orthographic, int n_samples, const float* gsrc, const float* gtgt,
                                 const float* gstep, float* g_k, float* g_s, void* workspace, cudaStream_t st) {
    const int N = height * width;
    const dim3 grid = setup_grid(N, kSetupRays, B);
    float* partials = reinterpret_cast<float*>(workspace);
    ray_setup_bwd_kernel<<<grid, 256, 0, st>>>(k_inv, n_k == 1 ? 0 : 9, sdd, n_s == 1 ? 0 : 1, N, width, orthographic,
                                               1.0f / (float)(n_samples - 1), gsrc, gtgt, gstep, partials);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    ray_setup_reduce_kernel<<<B, 320, 0, st>>>(partials, (int)grid.x, g_k, g_s);
    return cudaGetLastError();
}

cudaError_t launch_camera_affine(const float* w2v, const float* rt, int B, float* M, float* M_lo, cudaStream_t st) {
    camera_affine_kernel<<<(unsigned)(((long long)B * 12 + 95) / 96), 96, 0, st>>>(w2v, rt, B, M, M_lo);
    return cudaGetLastError();
}

cudaError_t launch_camera_affine_bwd(const float* w2v, const float* gM, int B, float* g_rt, cudaStream_t st) {
    camera_affine_bwd_kernel<<<(unsigned)(((long long)B * 16 + 127) / 128), 128, 0, st>>>(w2v, gM, B, g_rt);
    return cudaGetLastError();
}

cudaError_t launch_camera_rays(const float* k_inv, int n_k, const float* sdd, int n_s, int B, int height, int width,
                               int orthographic, float* src, float* tgt, cudaStream_t st) {
    const long long total = (long long)B * height * width;
    const long long blocks = (total + 255) / 256;
    const int grid = (int)(blocks < 152 * 16 ? blocks : 152 * 16);
    camera_rays_kernel<<<grid, 256, 0, st>>>(k_inv, n_k == 1 ? 0 : 9, sdd, n_s == 1 ? 0 : 1, B, height, width,
                                             orthographic, src, tgt);
    return cudaGetLastError();
}

}  // namespace ndrr
