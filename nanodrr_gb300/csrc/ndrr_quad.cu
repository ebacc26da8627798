// Volume preparation and the quad layout: the HU -> attenuation conversion,
// the quad build (one pass over the padded extent) and the fold of the
// quad-layout volume gradient back into the volume's layout. The layout is
// defined in ndrr_device.cuh (QuadOf, make_quadgeom).
#include "ndrr_march.cuh"

namespace ndrr {

// Quad builds: a thread keeps one column qx of a plane and walks down
// kBuildRows of its quad rows, so each row's corner pair (x0, x0 + 1) is
// loaded once and serves as the lower row of one quad and the upper row of
// the next; stores are one element per lane, consecutive along the row. One
// element per thread with its index divided out of a linear counter and four
// corner loads took 479 us at 512 x 512 x 400 f32, this 323 (2.1 GB read and
// written, 310 us at copy speed).
constexpr int kBuildRows = 16;
constexpr int kBuildThreads = 128;

// 32-bit float volume -> float4 quads.
struct QuadF32 {
    using Elem = float4;
    struct Corner {
        float v;
    };
    const float* __restrict__ v;
    __device__ __forceinline__ Corner load(size_t i) const { return Corner{__ldg(v + i)}; }
    static __device__ __forceinline__ Corner zero() { return Corner{0.f}; }
    static __device__ __forceinline__ Elem pack(Corner a, Corner b, Corner c, Corner d) {
        return make_float4(a.v, b.v, c.v, d.v);
    }
};

// 16-bit volume -> four raw 16-bit values per quad (bit-exact copies).
struct QuadB16 {
    using Elem = uint2;
    struct Corner {
        uint32_t v;
    };
    const uint16_t* __restrict__ v;
    __device__ __forceinline__ Corner load(size_t i) const { return Corner{(uint32_t)__ldg(v + i)}; }
    static __device__ __forceinline__ Corner zero() { return Corner{0u}; }
    static __device__ __forceinline__ Elem pack(Corner a, Corner b, Corner c, Corner d) {
        return make_uint2(a.v | (b.v << 16), c.v | (d.v << 16));
    }
};

// 16-bit volume + label map -> labelled quads: the four raw 16-bit corner
// values as above, and the four corners' classes (class in [0, C) as uint8,
// 255 for a label outside it; 0 for a corner outside the volume, the class
// the nearest-label rule gives a position there).
struct QuadLabeled {
    using Elem = uint4;
    struct Corner {
        uint32_t v, cls;
    };
    const uint16_t* __restrict__ v;
    const void* __restrict__ lab;
    int lab_dtype, C;
    __device__ __forceinline__ Corner load(size_t i) const {
        const int cls = ld_label(lab, lab_dtype, (int)i);
        return Corner{(uint32_t)__ldg(v + i), (uint32_t)((unsigned)cls < (unsigned)C ? cls : 255)};
    }
    static __device__ __forceinline__ Corner zero() { return Corner{0u, 0u}; }
    static __device__ __forceinline__ Elem pack(Corner a, Corner b, Corner c, Corner d) {
        return make_uint4(a.v | (b.v << 16), c.v | (d.v << 16), a.cls | (b.cls << 8) | (c.cls << 16) | (d.cls << 24),
                          0u);
    }
};

template <typename Q>
__global__ void __launch_bounds__(kBuildThreads) quad_build_kernel(const Q src, int D, int H, int W, int row_groups,
                                                                   typename Q::Elem* __restrict__ q) {
    using Corner = typename Q::Corner;
    const int QX = W + 3, QY = H + 3;
    const int qz = (int)(blockIdx.x / (unsigned)row_groups);
    const int qy0 = (int)(blockIdx.x % (unsigned)row_groups) * kBuildRows, qy1 = min(QY, qy0 + kBuildRows);
    const int z = qz - 2;
    const bool plane = (unsigned)z < (unsigned)D;
    typename Q::Elem* out = q + ((size_t)qz * QY + qy0) * QX;
    for (int qx = threadIdx.x; qx < QX; qx += kBuildThreads) {
        const int x0 = qx - 2;
        const bool in0 = plane && (unsigned)x0 < (unsigned)W, in1 = plane && (unsigned)(x0 + 1) < (unsigned)W;
        // corner pair of volume row y (zeros outside)
        auto pair = [&](int y, Corner& a, Corner& b) {
            const bool row = (unsigned)y < (unsigned)H;
            const size_t i = ((size_t)z * H + y) * W + x0;
            a = row && in0 ? src.load(i) : Q::zero();
            b = row && in1 ? src.load(i + 1) : Q::zero();
        };
        Corner a, b;
        pair(qy0 - 2, a, b);
        if (qy1 - qy0 == kBuildRows) {
            Corner c[kBuildRows], d[kBuildRows];
#pragma unroll
            for (int r = 0; r < kBuildRows; ++r) pair(qy0 + r - 1, c[r], d[r]);
#pragma unroll
            for (int r = 0; r < kBuildRows; ++r) {
                out[(size_t)r * QX + qx] = Q::pack(a, b, c[r], d[r]);
                a = c[r];
                b = d[r];
            }
        } else {
            for (int qy = qy0; qy < qy1; ++qy) {
                Corner c, d;
                pair(qy - 1, c, d);
                out[(size_t)(qy - qy0) * QX + qx] = Q::pack(a, b, c, d);
                a = c;
                b = d;
            }
        }
    }
}

template <typename Q>
static cudaError_t quad_build(const Q& src, int D, int H, int W, void* quad, cudaStream_t st) {
    const int groups = (H + 3 + kBuildRows - 1) / kBuildRows;
    const long long grid = (long long)(D + 4) * groups;
    quad_build_kernel<Q><<<(unsigned)grid, kBuildThreads, 0, st>>>(src, D, H, W, groups,
                                                                   (typename Q::Elem*)quad);
    return cudaGetLastError();
}

// gvol[z][y][x] += the four quad entries in which voxel (x, y) of plane z is
// a corner: (x, y) as (x0, y0), (x0 + 1, y0), (x0, y0 + 1), (x0 + 1, y0 + 1).
// One CTA per kFoldRows consecutive lines (z, y) of the volume, four
// consecutive x per thread: the five quad entries of a quad row are 16-byte
// loads, and walking down the lines each quad row is loaded once and serves
// as the upper row of one line and the lower row of the next.
constexpr int kFoldRows = 8;

template <bool OVERWRITE>
__global__ void __launch_bounds__(128) quad_fold_kernel(const float4* __restrict__ gq, int D, int H, int W,
                                                        float* __restrict__ gvol) {
    const int QX = W + 3, QY = H + 3;
    const int nyb = (H + kFoldRows - 1) / kFoldRows;
    const int z = (int)(blockIdx.x / (unsigned)nyb), y0 = (int)(blockIdx.x % (unsigned)nyb) * kFoldRows;
    const int y1 = min(H, y0 + kFoldRows);
    const bool vec = (W & 3) == 0;
    for (int x0 = threadIdx.x * 4; x0 < W; x0 += blockDim.x * 4) {
        // entries x0 + 1 .. x0 + 5 (all inside the padded row of W + 3)
        int e[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) e[k] = min(x0 + 1 + k, QX - 1);
        const float4* row = gq + ((size_t)(z + 2) * QY + (y0 + 1)) * QX;  // entries with y0 = y - 1
        float4 c[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) c[k] = __ldg(row + e[k]);
        for (int y = y0; y < y1; ++y) {
            row += QX;  // entries with y0 = y
            float4 a[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) a[k] = __ldg(row + e[k]);
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = (a[j + 1].x + a[j].y) + (c[j + 1].z + c[j].w);
            float* out = gvol + ((size_t)z * H + y) * W;
            if (vec) {
                float4 o = OVERWRITE ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<float4*>(out + x0);
                o.x += v[0];
                o.y += v[1];
                o.z += v[2];
                o.w += v[3];
                *reinterpret_cast<float4*>(out + x0) = o;
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (x0 + j < W) out[x0 + j] = OVERWRITE ? v[j] : out[x0 + j] + v[j];
            }
#pragma unroll
            for (int k = 0; k < 5; ++k) c[k] = a[k];
        }
    }
}

// HU -> linear attenuation (1/mm), the reference's piecewise-linear map
// (nanodrr src/nanodrr/data/preprocess.py:44-50): clamp HU at -1000; at or
// below 0 HU the air-water line (h / 1000 + 1) * mu_water, above it the
// water-bone line mu_water + (h / hu_bone) * dmu with dmu = mu_bone -
// mu_water; clamp at 0 (NaN passes through both clamps, as torch.clamp lets
// it), in fp32; the 16-bit types convert on load and round to nearest-even
// on store. Sixteen bytes per thread and step where both arrays are aligned to
// them (the head and tail, and other alignments, go one by one), and one
// division per element, by the divisor of its branch: 512 x 512 x 400 f32 took
// 224 us element by element with both branches, 142 now (124 at copy speed).
template <typename T>
struct __align__(16) HuVec {
    T e[16 / sizeof(T)];
};

__device__ __forceinline__ float hu_mu(float x, float mu_water, float dmu, float hu_bone) {
    const float h = x < -1000.0f ? -1000.0f : x;  // NaN stays NaN, as in torch.clamp
    const bool dense = h > 0.0f;
    const float q = __fdiv_rn(h, dense ? hu_bone : 1000.0f);
    const float m = dense ? __fadd_rn(mu_water, __fmul_rn(q, dmu)) : __fmul_rn(__fadd_rn(q, 1.0f), mu_water);
    return m > 0.0f ? m : (m == m ? 0.0f : m);
}

__device__ __forceinline__ float hu_in(float v) { return v; }
__device__ __forceinline__ float hu_in(__half v) { return __half2float(v); }
__device__ __forceinline__ float hu_in(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T>
__global__ void __launch_bounds__(256) hu_to_mu_kernel(const T* __restrict__ hu, long long n, float mu_water,
                                                       float dmu, float hu_bone, T* __restrict__ mu, bool vec) {
    constexpr int V = 16 / sizeof(T);
    const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    const long long nv = vec ? n / V : 0;
    for (long long i = first; i < nv; i += step) {
        union {
            uint4 raw;
            HuVec<T> v;
        } a;
        a.raw = __ldg(reinterpret_cast<const uint4*>(hu) + i);
        HuVec<T> o;
#pragma unroll
        for (int k = 0; k < V; ++k) st_out(o.e, (size_t)k, hu_mu(hu_in(a.v.e[k]), mu_water, dmu, hu_bone));
        *reinterpret_cast<uint4*>(mu + i * V) = *reinterpret_cast<const uint4*>(&o);
    }
    for (long long i = nv * V + first; i < n; i += step)
        st_out(mu, (size_t)i, hu_mu(hu_in(hu[i]), mu_water, dmu, hu_bone));
}

static int grid_for(long long n) { return (int)std::max(1LL, std::min((n + 255) / 256, 152LL * 32)); }

cudaError_t launch_quad_build(const void* vol, int dtype, int D, int H, int W, void* quad, cudaStream_t st) {
    if (dtype == NDRR_F32) return quad_build(QuadF32{(const float*)vol}, D, H, W, quad, st);
    if (dtype == NDRR_F16 || dtype == NDRR_BF16)
        return quad_build(QuadB16{(const uint16_t*)vol}, D, H, W, quad, st);
    return cudaErrorInvalidValue;
}

cudaError_t launch_quad_build_labeled(const void* vol, int dtype, const void* lab, int lab_dtype, int C, int D, int H,
                                      int W, void* quad, cudaStream_t st) {
    if (dtype != NDRR_F16 && dtype != NDRR_BF16) return cudaErrorInvalidValue;
    return quad_build(QuadLabeled{(const uint16_t*)vol, lab, lab_dtype, C}, D, H, W, quad, st);
}

template <typename T>
static cudaError_t hu_to_mu(const void* hu, long long n, float mu_water, float dmu, float hu_bone, void* mu,
                            cudaStream_t st) {
    const bool vec = ((uintptr_t)hu | (uintptr_t)mu) % 16 == 0;
    hu_to_mu_kernel<T><<<grid_for(vec ? n * (long long)sizeof(T) / 16 : n), 256, 0, st>>>(
        (const T*)hu, n, mu_water, dmu, hu_bone, (T*)mu, vec);
    return cudaGetLastError();
}

cudaError_t launch_hu_to_mu(const void* hu, int dtype, long long n, float mu_water, float dmu, float hu_bone,
                            void* mu, cudaStream_t st) {
    switch (dtype) {
        case NDRR_F32: return hu_to_mu<float>(hu, n, mu_water, dmu, hu_bone, mu, st);
        case NDRR_F16: return hu_to_mu<__half>(hu, n, mu_water, dmu, hu_bone, mu, st);
        case NDRR_BF16: return hu_to_mu<__nv_bfloat16>(hu, n, mu_water, dmu, hu_bone, mu, st);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_quad_fold(const float* gquad, int D, int H, int W, float* gvol, bool overwrite,
                             cudaStream_t st) {
    const unsigned grid = (unsigned)((long long)D * ((H + kFoldRows - 1) / kFoldRows));
    if (overwrite)
        quad_fold_kernel<true><<<grid, 128, 0, st>>>((const float4*)gquad, D, H, W, gvol);
    else
        quad_fold_kernel<false><<<grid, 128, 0, st>>>((const float4*)gquad, D, H, W, gvol);
    return cudaGetLastError();
}

}  // namespace ndrr
