// Normalised cross-correlation of image pairs, forward and adjoint (the
// reference's metrics/ncc.py:8-37 NormalizedCrossCorrelation2d): per plane
// (an image channel, or a patch when the caller unfolds patches into planes)
// both images are centred and scaled by sqrt(population variance + eps), and
// the score of a batch element is the mean over its planes' pixels of the
// product.
//
// Forward: chunks of 1024 pixels per CTA accumulate moments about the chunk's
// first pixel in pairs of floats (Knuth's error-free sum and difference, and
// products by a fused multiply-add; about 46 bits) and shift them to raw
// moments in fp64, so centring after the fact is as accurate as with moments
// summed in fp64: the pairs' error is relative to the chunk's own spread about
// one of its pixels, not to its offset. A warp per plane sums the chunks in a
// fixed order in fp64 and forms the centred statistics (and, with one plane
// per batch element, the score), and a CTA per batch element sums several
// planes. The adjoint is the closed form of d score / d x, elementwise from
// the saved statistics.
//
// The pairs are there because the fp64 pipe (2 lanes per clock and SM) bound
// the moments: 8 x 1024^2 took 139 us in fp64, 45 so (10 at memory speed).
// Raw moments in pairs (36 us) are a tenth as accurate where the mean is large:
// error of the score 8e-8, 8e-6 at means of 1e4, 1e5 standard deviations, in
// fp64 and about the first pixel 1e-8, 6e-7.
#include <cuda_runtime.h>

#include "../../include/nanodrr_gb300.h"

namespace ndrr {

constexpr int kNccBlock = 256;
constexpr int kNccStats = 8;  // mu1, mu2, s1, s2, S12, sum a1, sum a2, plane score
constexpr int kNccMomentBlock = 128;
constexpr int kNccChunk = 1024;      // pixels per CTA of the moment pass
constexpr int kNccBwdChunk = 4096;   // pixels per CTA of the adjoint

static int ncc_chunks(int N) { return (N + kNccChunk - 1) / kNccChunk; }
static int ncc_bwd_chunks(int N) { return (N + kNccBwdChunk - 1) / kNccBwdChunk; }

// x + err without rounding (up to the pair's 46 bits): a float and what it lacks.
struct Pair {
    float x, err;
};

__device__ __forceinline__ Pair pair_diff(float a, float b) {  // a - b
    const float d = __fsub_rn(a, b), bb = __fsub_rn(d, a);
    return {d, __fsub_rn(__fsub_rn(a, __fsub_rn(d, bb)), __fadd_rn(b, bb))};
}

__device__ __forceinline__ Pair pair_product(Pair a, Pair b) {
    const float p = __fmul_rn(a.x, b.x);
    return {p, __fmaf_rn(a.x, b.err, __fmaf_rn(a.err, b.x, __fmaf_rn(a.x, b.x, -p)))};
}

// Sum kept as hi + lo: each term's rounding error against hi goes into lo.
struct PairSum {
    float hi, lo;
    __device__ __forceinline__ void add(Pair t) {
        const float s = __fadd_rn(hi, t.x);
        const float bb = __fsub_rn(s, hi);
        const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(t.x, bb));
        hi = s;
        lo = __fadd_rn(lo, __fadd_rn(e, t.err));
    }
};

// Raw moments of one chunk of one plane: sum x1, sum x2, sum x1^2, sum x2^2,
// sum x1 x2, reduced in a fixed order into partials[plane][chunk][5]. Pairs
// need products and their errors inside float's range: a chunk with a
// non-zero pixel outside (1e-15, 1e16), an infinity or a NaN is summed in
// fp64.
__global__ void __launch_bounds__(kNccMomentBlock) ncc_moments_kernel(const float* __restrict__ x1,
                                                                      const float* __restrict__ x2, int N, int nch,
                                                                      double* __restrict__ partials) {
    __shared__ double sh[kNccMomentBlock / 32][5];
    const size_t plane = blockIdx.x / (unsigned)nch;
    const int chunk = blockIdx.x % (unsigned)nch;
    const int beg = chunk * kNccChunk, end = min(N, beg + kNccChunk);
    const float* a = x1 + plane * N;
    const float* b = x2 + plane * N;
    const float c1 = __ldg(a + beg), c2 = __ldg(b + beg);
    PairSum s[5] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
    bool plain = true;
#pragma unroll 4
    for (int i = beg + threadIdx.x; i < end; i += kNccMomentBlock) {
        const float u = __ldg(a + i), v = __ldg(b + i);
        plain &= (u == 0.f || (fabsf(u) > 1e-15f && fabsf(u) < 1e16f)) &&
                 (v == 0.f || (fabsf(v) > 1e-15f && fabsf(v) < 1e16f));
        const Pair d = pair_diff(u, c1), e = pair_diff(v, c2);
        s[0].add(d);
        s[1].add(e);
        s[2].add(pair_product(d, d));
        s[3].add(pair_product(e, e));
        s[4].add(pair_product(d, e));
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool all_plain = __syncthreads_and(plain) != 0;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        double x;
        if (all_plain) {
            PairSum t = s[k];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float h = __shfl_xor_sync(0xffffffffu, t.hi, o), l = __shfl_xor_sync(0xffffffffu, t.lo, o);
                t.add({h, l});
            }
            x = (double)t.hi + (double)t.lo;
        } else {
            x = 0.0;
            for (int i = beg + threadIdx.x; i < end; i += kNccMomentBlock) {
                const double u = (double)__ldg(a + i), v = (double)__ldg(b + i);
                x += k == 0 ? u : k == 1 ? v : k == 2 ? u * u : k == 3 ? v * v : u * v;
            }
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        }
        if (lane == 0) sh[warp][k] = x;
    }
    __syncthreads();
    if (threadIdx.x < 5) {
        const int k = threadIdx.x;
        const int l = k == 3 ? 1 : k == 4 ? 1 : 0, r = k == 3 ? 1 : 0;  // first moments of a product's factors
        double x = 0.0, sl = 0.0, sr = 0.0;
        for (int w = 0; w < kNccMomentBlock / 32; ++w) {
            x += sh[w][k];
            sl += sh[w][l];
            sr += sh[w][r];
        }
        if (all_plain) {  // sum (c + d) = sum d + n c; sum (c + d)(f + e) = sum d e + f sum d + c (sum e + n f)
            const double n = (double)(end - beg), cl = (double)(l ? c2 : c1), cr = (double)(r ? c2 : c1);
            if (k < 2)
                x += n * (double)(k ? c2 : c1);
            else
                x += cl * sr + cr * (sl + n * cl);
        }
        partials[(plane * nch + chunk) * 5 + k] = x;
    }
}

// Per plane (a warp): fixed-order sum of the chunk moments, then the centred
// statistics and the plane's score; `score` (one plane per batch element)
// takes it directly.
__global__ void __launch_bounds__(128) ncc_stats_kernel(const double* __restrict__ partials, int nch, int N,
                                                        float eps, float* __restrict__ stats, int planes,
                                                        float* __restrict__ score) {
    const int plane = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (plane >= planes) return;
    double m[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int c = lane; c < nch; c += 32)
#pragma unroll
        for (int k = 0; k < 5; ++k) m[k] += partials[((size_t)plane * nch + c) * 5 + k];
#pragma unroll
    for (int k = 0; k < 5; ++k)
        for (int o = 16; o > 0; o >>= 1) m[k] += __shfl_xor_sync(0xffffffffu, m[k], o);
    if (lane != 0) return;
    const double n = (double)N;
    const double mu1 = m[0] / n, mu2 = m[1] / n;
    const double c11 = fmax(m[2] - n * mu1 * mu1, 0.0), c22 = fmax(m[3] - n * mu2 * mu2, 0.0);
    const double c12 = m[4] - n * mu1 * mu2;
    const double s1 = sqrt(c11 / n + (double)eps), s2 = sqrt(c22 / n + (double)eps);
    const float own = (float)(c12 / (s1 * s2));
    float* st = stats + (size_t)plane * kNccStats;
    st[0] = (float)mu1;
    st[1] = (float)mu2;
    st[2] = (float)s1;
    st[3] = (float)s2;
    st[4] = (float)c12;
    st[5] = (float)(m[0] - n * mu1);  // centred first moments: zero up to rounding
    st[6] = (float)(m[1] - n * mu2);
    st[7] = own;
    if (score != nullptr) score[plane] = (float)((double)own / n);
}

// Score of a batch element of several planes: fixed-order sum.
__global__ void __launch_bounds__(kNccBlock) ncc_score_kernel(const float* __restrict__ stats, int P, int N,
                                                              float* __restrict__ score) {
    __shared__ double red[kNccBlock / 32];
    const int b = blockIdx.x;
    double s = 0.0;
    for (int p = threadIdx.x; p < P; p += kNccBlock) s += (double)stats[((size_t)b * P + p) * kNccStats + 7];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = red[0];
        for (int w = 1; w < kNccBlock / 32; ++w) t += red[w];
        score[b] = (float)(t / ((double)P * N));
    }
}

// d score_b / d x1_j = g [ x2n_j / s1 - sum(x2n) / (N s1) - a1_j S12 / (s2 N s1^3) ],
// g = go_b / (P N), x2n = (x2 - mu2) / s2; symmetric for x2.
__global__ void __launch_bounds__(kNccBlock) ncc_bwd_kernel(const float* __restrict__ go,
                                                            const float* __restrict__ x1,
                                                            const float* __restrict__ x2,
                                                            const float* __restrict__ stats, int P, int N,
                                                            float* __restrict__ g1, float* __restrict__ g2) {
    const size_t plane = blockIdx.x;
    const int b = (int)(plane / P);
    const float* st = stats + plane * kNccStats;
    const float m1 = st[0], m2 = st[1], s1 = st[2], s2 = st[3], S12 = st[4], z1 = st[5], z2 = st[6];
    const float g = __ldg(go + b) / ((float)P * (float)N);
    const float inv_n = 1.f / (float)N;
    // x1 side
    const float k1a = g / (s1 * s2), k1b = g * z2 / (s2 * N * s1), k1c = g * S12 * inv_n / (s2 * s1 * s1 * s1);
    const float k2a = g / (s1 * s2), k2b = g * z1 / (s1 * N * s2), k2c = g * S12 * inv_n / (s1 * s2 * s2 * s2);
    const float* a = x1 + plane * N;
    const float* c = x2 + plane * N;
    const int beg = blockIdx.y * kNccBwdChunk, end = min(N, beg + kNccBwdChunk);
    for (int i = beg + threadIdx.x; i < end; i += kNccBlock) {
        const float d1 = __ldg(a + i) - m1, d2 = __ldg(c + i) - m2;
        if (g1 != nullptr) g1[plane * N + i] = k1a * d2 - k1b - k1c * d1;
        if (g2 != nullptr) g2[plane * N + i] = k2a * d1 - k2b - k2c * d2;
    }
}

size_t ncc_workspace_bytes(int B, int P, int N) { return (size_t)B * P * ncc_chunks(N) * 5 * sizeof(double); }

cudaError_t launch_ncc_fwd(const float* x1, const float* x2, int B, int P, int N, float eps, float* score,
                           float* stats, void* workspace, cudaStream_t st) {
    const int planes = B * P, nch = ncc_chunks(N);
    double* partials = reinterpret_cast<double*>(workspace);
    ncc_moments_kernel<<<(unsigned)((long long)planes * nch), kNccMomentBlock, 0, st>>>(x1, x2, N, nch, partials);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    ncc_stats_kernel<<<(planes + 3) / 4, 128, 0, st>>>(partials, nch, N, eps, stats, planes, P == 1 ? score : nullptr);
    if ((e = cudaGetLastError()) != cudaSuccess || P == 1) return e;
    ncc_score_kernel<<<B, kNccBlock, 0, st>>>(stats, P, N, score);
    return cudaGetLastError();
}

cudaError_t launch_ncc_bwd(const float* go, const float* x1, const float* x2, const float* stats, int B, int P,
                           int N, float* g1, float* g2, cudaStream_t st) {
    ncc_bwd_kernel<<<dim3((unsigned)((size_t)B * P), (unsigned)ncc_bwd_chunks(N)), kNccBlock, 0, st>>>(go, x1, x2, stats,
                                                                                                 P, N, g1, g2);
    return cudaGetLastError();
}

}  // namespace ndrr
