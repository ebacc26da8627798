// Local NCC: the NCC of ndrr_ncc.cu over every p x p window of an image pair
// (the reference's metrics/ncc.py:8-37, 65-74, which unfolds the windows into
// channels), computed from the images themselves.
//
// A window's statistics are five box sums (x1, x2, x1^2, x2^2, x1 x2), and
// its adjoint is linear in the pixels with per-window coefficients, so the
// pixel gradient is three box sums of coefficient maps. Both are separable:
// rows first (p taps), then columns of the row sums (p taps), 2 p additions
// per window where the unfolded form reads p^2 pixels per window. Sums only
// add (no running subtraction), in fp64, so there is no cancellation between
// windows and a NaN stays in the windows that contain it.
//
// Bound: the fp64 pipe (2 lanes per clock and SM). Four neighbouring windows
// are summed by one thread from their shared taps (p - 3 common ones added
// once), 27 additions per window and moment in each direction at p = 13
// instead of 65 for the moments of a window alone. 8 x 200^2, p = 13, forward
// and adjoint: 0.16 ms of kernels, where unfolding, moments of 283,000 planes of 169
// pixels and the fold took 8.2 ms.
#include <cuda_runtime.h>

#include "../../include/nanodrr_gb300.h"
#include "ndrr_launch.h"

namespace ndrr {

constexpr int kPatchTX = 32;      // windows (adjoint: pixels) per tile row
constexpr int kPatchTY = 16;      // rows per tile
constexpr int kPatchThreads = 128;
constexpr int kPatchMaps = 5;     // saved per window: mu1, mu2, 1 / (s1 s2), c1, c2 (see below)

// v[j] = sum of the p taps at(j), .., at(j + p - 1) for j = 0 .. 3, K
// quantities each: the taps the four windows share (3 .. p - 1) are added
// once.
template <int K, typename At>
__device__ __forceinline__ void four_windows(int p, At at, double (&v)[4][K]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int k = 0; k < K; ++k) v[j][k] = 0.0;
    double x[K];
    if (p < 4) {
        for (int i = 0; i < p + 3; ++i) {
            at(i, x);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i >= j && i < j + p)
#pragma unroll
                    for (int k = 0; k < K; ++k) v[j][k] += x[k];
        }
        return;
    }
    for (int i = 3; i < p; ++i) {
        at(i, x);
#pragma unroll
        for (int k = 0; k < K; ++k) v[3][k] += x[k];
    }
#pragma unroll
    for (int k = 0; k < K; ++k) v[0][k] = v[1][k] = v[2][k] = v[3][k];
#pragma unroll
    for (int i = 0; i < 3; ++i) {  // taps 0 .. 2 belong to windows 0 .. i
        at(i, x);
#pragma unroll
        for (int j = 0; j <= i; ++j)
#pragma unroll
            for (int k = 0; k < K; ++k) v[j][k] += x[k];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {  // taps p .. p + 2 belong to windows i + 1 .. 3
        at(p + i, x);
#pragma unroll
        for (int j = i + 1; j < 4; ++j)
#pragma unroll
            for (int k = 0; k < K; ++k) v[j][k] += x[k];
    }
}

// Tile of windows: row sums of the tile's (kPatchTY + p - 1) pixel rows in
// shared memory, then each thread's four windows down a column, their
// statistics, and the tile's part of the score (fixed order).
__global__ void __launch_bounds__(kPatchThreads) ncc_patch_fwd_kernel(const float* __restrict__ x1,
                                                                      const float* __restrict__ x2, int H, int W,
                                                                      int p, float eps, int tiles_x, int tiles,
                                                                      double* __restrict__ maps,
                                                                      double* __restrict__ partials) {
    extern __shared__ double rows[];  // [5][R][kPatchTX]
    __shared__ double red[kPatchThreads / 32];
    const int R = kPatchTY + p - 1;
    const int tile = blockIdx.x % tiles, plane = blockIdx.x / tiles;
    const int px = (tile % tiles_x) * kPatchTX, py = (tile / tiles_x) * kPatchTY;
    const int HO = H - p + 1, WO = W - p + 1;
    const float* a = x1 + (size_t)plane * H * W;
    const float* b = x2 + (size_t)plane * H * W;
    const int RS = R * kPatchTX;
    for (int item = threadIdx.x; item < R * (kPatchTX / 4); item += kPatchThreads) {
        const int r = item / (kPatchTX / 4), c = (item % (kPatchTX / 4)) * 4;
        const int y = py + r, x0 = px + c;
        double v[4][5];
        if (y < H && x0 < WO) {
            const float* ra = a + (size_t)y * W;
            const float* rb = b + (size_t)y * W;
            four_windows<5>(p, [&](int i, double (&q)[5]) {
                // taps past the row's end belong to windows past it
                const int x = min(x0 + i, W - 1);
                const double u = (double)__ldg(ra + x), w = (double)__ldg(rb + x);
                q[0] = u;
                q[1] = w;
                q[2] = u * u;
                q[3] = w * w;
                q[4] = u * w;
            }, v);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int k = 0; k < 5; ++k) v[j][k] = 0.0;
        }
#pragma unroll
        for (int k = 0; k < 5; ++k)
#pragma unroll
            for (int j = 0; j < 4; ++j) rows[k * RS + r * kPatchTX + c + j] = v[j][k];
    }
    __syncthreads();
    const double n = (double)p * p;
    double score = 0.0;
    {
        const int c = threadIdx.x % kPatchTX, r0 = (threadIdx.x / kPatchTX) * 4;
        double v[4][5];
        four_windows<5>(p, [&](int i, double (&q)[5]) {
#pragma unroll
            for (int k = 0; k < 5; ++k) q[k] = rows[k * RS + (r0 + i) * kPatchTX + c];
        }, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int x = px + c, y = py + r0 + j;
            if (x >= WO || y >= HO) continue;
            const double mu1 = v[j][0] / n, mu2 = v[j][1] / n;
            const double c11 = fmax(v[j][2] - n * mu1 * mu1, 0.0), c22 = fmax(v[j][3] - n * mu2 * mu2, 0.0);
            const double c12 = v[j][4] - n * mu1 * mu2;
            const double s1 = sqrt(c11 / n + (double)eps), s2 = sqrt(c22 / n + (double)eps);
            const double is = 1.0 / (s1 * s2);
            score += c12 * is;
            // d(window score) / d x1 = is (x2 - mu2) - c1 (x1 - mu1), c1 =
            // c12 is / (n s1^2); symmetric for x2 with c2
            double* m = maps + (size_t)plane * kPatchMaps * HO * WO + (size_t)y * WO + x;
            const size_t ms = (size_t)HO * WO;
            m[0] = mu1;
            m[ms] = mu2;
            m[2 * ms] = is;
            m[3 * ms] = c12 * is / (n * s1 * s1);
            m[4 * ms] = c12 * is / (n * s2 * s2);
        }
    }
    for (int o = 16; o > 0; o >>= 1) score += __shfl_xor_sync(0xffffffffu, score, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = score;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = red[0];
        for (int w = 1; w < kPatchThreads / 32; ++w) s += red[w];
        partials[blockIdx.x] = s;
    }
}
static_assert(kPatchTX * kPatchTY == 4 * kPatchThreads, "one column group of four windows per thread");

// Score of a batch element: fixed-order sum of its tiles' parts.
__global__ void __launch_bounds__(256) ncc_patch_score_kernel(const double* __restrict__ partials, int per_batch,
                                                              double norm, float* __restrict__ score) {
    __shared__ double red[8];
    double s = 0.0;
    for (int i = threadIdx.x; i < per_batch; i += 256) s += partials[(size_t)blockIdx.x * per_batch + i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = red[0];
        for (int w = 1; w < 8; ++w) t += red[w];
        score[blockIdx.x] = (float)(t / norm);
    }
}

// Pixel gradient of one image of the pair: xa is the image differentiated, xb
// the other; the windows containing pixel (y, x) start at (y - p + 1 .. y,
// x - p + 1 .. x). With d(window) / d xa = is (xb - mub) - ca (xa - mua):
//   g = go / (windows p^2) [ xb sum(is) - xa sum(ca) - sum(is mub - ca mua) ].
__global__ void __launch_bounds__(kPatchThreads) ncc_patch_bwd_kernel(const float* __restrict__ go,
                                                                      const float* __restrict__ xa,
                                                                      const float* __restrict__ xb,
                                                                      const double* __restrict__ maps, int which,
                                                                      int C, int H, int W, int p, int tiles_x,
                                                                      int tiles, double norm,
                                                                      float* __restrict__ g) {
    extern __shared__ double rows[];  // [3][R][kPatchTX]
    const int R = kPatchTY + p - 1;
    const int tile = blockIdx.x % tiles, plane = blockIdx.x / tiles;
    const int px = (tile % tiles_x) * kPatchTX, py = (tile / tiles_x) * kPatchTY;
    const int HO = H - p + 1, WO = W - p + 1;
    const size_t ms = (size_t)HO * WO;
    const double* m = maps + (size_t)plane * kPatchMaps * ms;
    const double* mua = m + (which ? ms : 0);
    const double* mub = m + (which ? 0 : ms);
    const double* mis = m + 2 * ms;
    const double* mca = m + (which ? 4 : 3) * ms;
    const int RS = R * kPatchTX;
    for (int item = threadIdx.x; item < R * (kPatchTX / 4); item += kPatchThreads) {
        const int r = item / (kPatchTX / 4), c = (item % (kPatchTX / 4)) * 4;
        const int y = py + r - (p - 1), x0 = px + c - (p - 1);
        double v[4][3];
        if (y >= 0 && y < HO) {
            const size_t row = (size_t)y * WO;
            four_windows<3>(p, [&](int i, double (&q)[3]) {
                const int x = x0 + i;
                q[0] = q[1] = q[2] = 0.0;
                if (x >= 0 && x < WO) {
                    const double is = __ldg(mis + row + x), ca = __ldg(mca + row + x);
                    q[0] = is;
                    q[1] = ca;
                    q[2] = is * __ldg(mub + row + x) - ca * __ldg(mua + row + x);
                }
            }, v);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int k = 0; k < 3; ++k) v[j][k] = 0.0;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int j = 0; j < 4; ++j) rows[k * RS + r * kPatchTX + c + j] = v[j][k];
    }
    __syncthreads();
    const int c = threadIdx.x % kPatchTX, r0 = (threadIdx.x / kPatchTX) * 4;
    double v[4][3];
    four_windows<3>(p, [&](int i, double (&q)[3]) {
#pragma unroll
        for (int k = 0; k < 3; ++k) q[k] = rows[k * RS + (r0 + i) * kPatchTX + c];
    }, v);
    const double s = (double)__ldg(go + plane / C) / norm;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int x = px + c, y = py + r0 + j;
        if (x >= W || y >= H) continue;
        const size_t at = (size_t)plane * H * W + (size_t)y * W + x;
        g[at] = (float)(s * ((double)__ldg(xb + at) * v[j][0] - (double)__ldg(xa + at) * v[j][1] - v[j][2]));
    }
}

static size_t patch_smem(int p, int k) { return (size_t)k * (kPatchTY + p - 1) * kPatchTX * sizeof(double); }

// Lets `kern` have the shared memory of the largest window (183 and 110 KB),
// whatever this call's: the limit belongs to the device, and a call that set
// its own would lower it between another host thread's setting and launch.
template <typename K>
static cudaError_t allow_largest(K kern, int k) {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)patch_smem(NDRR_NCC_PATCH_MOST, k));
}

static int cover(int n, int t) { return (n + t - 1) / t; }

static long long patch_tiles(int rows, int cols) {
    return (long long)cover(rows, kPatchTY) * cover(cols, kPatchTX);
}

uint64_t ncc_patch_workspace_bytes(int B, int C, int H, int W, int p) {
    return (uint64_t)B * C * patch_tiles(H - p + 1, W - p + 1) * sizeof(double);
}

cudaError_t launch_ncc_patch_fwd(const float* x1, const float* x2, int B, int C, int H, int W, int p, float eps,
                                 float* score, double* maps, void* workspace, cudaStream_t st) {
    const int HO = H - p + 1, WO = W - p + 1;
    const int tiles = (int)patch_tiles(HO, WO);
    const size_t smem = patch_smem(p, 5);
    cudaError_t e = allow_largest(ncc_patch_fwd_kernel, 5);
    if (e != cudaSuccess) return e;
    double* partials = reinterpret_cast<double*>(workspace);
    ncc_patch_fwd_kernel<<<(unsigned)((long long)B * C * tiles), kPatchThreads, smem, st>>>(
        x1, x2, H, W, p, eps, cover(WO, kPatchTX), tiles, maps, partials);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const double norm = (double)C * HO * WO * ((double)p * p);
    ncc_patch_score_kernel<<<B, 256, 0, st>>>(partials, C * tiles, norm, score);
    return cudaGetLastError();
}

cudaError_t launch_ncc_patch_bwd(const float* go, const float* x1, const float* x2, const double* maps, int B, int C,
                                 int H, int W, int p, float* g1, float* g2, cudaStream_t st) {
    const int tiles = (int)patch_tiles(H, W);
    const size_t smem = patch_smem(p, 3);
    cudaError_t e = allow_largest(ncc_patch_bwd_kernel, 3);
    const double norm = (double)C * (H - p + 1) * (W - p + 1) * ((double)p * p);
    const unsigned grid = (unsigned)((long long)B * C * tiles);
    for (int which = 0; which < 2 && e == cudaSuccess; ++which) {
        float* g = which ? g2 : g1;
        if (g == nullptr) continue;
        ncc_patch_bwd_kernel<<<grid, kPatchThreads, smem, st>>>(go, which ? x2 : x1, which ? x1 : x2, maps, which, C, H,
                                                               W, p, cover(W, kPatchTX), tiles, norm, g);
        e = cudaGetLastError();
    }
    return e;
}

}  // namespace ndrr
