// Forward of a large one-channel render whose pose needs a gradient: the image
// and, per ray, the sums the pose adjoint needs from the samples,
//   G = sum_s dv_s,  Gt = sum_s t_s dv_s   (dv_s the position gradient),
// since dL/dM_ij = sum_rays go step sum_s dv_s,i [src + t_s e, 1]_j is linear in
// them: the adjoint then reads 24 bytes per ray instead of marching the
// volume a second time (pose_sums_kernel). Positions, cells and gradients are
// those of the adjoint (32.32 fixed point, ndrr_march.cuh). The image takes the
// same corners at the forward's float positions. It is not bitwise the image of
// a render without a gradient: the two positions differ by an ulp of the float,
// and where that puts them on two sides of a cell face, this image extrapolates
// its cell by as much, while the plain one is in the next cell. The two are
// equally far from the exact image and up to 2e-6 of the maximum apart on smooth
// volumes, 4e-6 on white noise.
//
// Both marches wait for the same gathers, so the one that does both costs about
// what the adjoint alone does (kernels alone): 16 poses x 200^2 x 500 samples of
// 512 x 512 x 400 f32 0.74 ms for 0.69 + 0.73, 8 poses x 1024^2 x 1000 with
// occupancy windows 6.5 for 3.4 + 6.1.
#include "ndrr_march.cuh"

namespace ndrr {

// The trilinear derivative (cell_grad) from first differences of the corners
// and their differences, which the three components share: 20 operations where
// each component interpolated by itself takes 33 (with those the kernel's steps
// take 1.18 times as long at 8 x 1024^2 x 1000, 1.06 at 32 x 256^2 x 800 of
// 512^3). dL/dM is as accurate with either, and as the marching adjoint's: root
// mean square error against float64 over 12 seeded volumes and poses at four
// sizes 1.38e-7 (16 x 181^2: 1.05e-7) for 1.26e-7 (1.14e-7).
__device__ __forceinline__ void cell_grad_shared(const Cell& c, float& gx, float& gy, float& gz) {
    const float x00 = c.v001 - c.v000, x01 = c.v011 - c.v010;  // d/dx at (z, y) = (0, 0), (0, 1)
    const float x10 = c.v101 - c.v100, x11 = c.v111 - c.v110;
    const float y0 = c.v010 - c.v000, y1 = c.v110 - c.v100;    // d/dy at x = 0, z = 0 and 1
    const float xy0 = x01 - x00, xy1 = x11 - x10;
    const float a0 = fmaf(c.fy, xy0, x00), a1 = fmaf(c.fy, xy1, x10);  // d/dx at z = 0 and 1
    const float b0 = fmaf(c.fx, xy0, y0), b1 = fmaf(c.fx, xy1, y1);
    const float xz = a1 - a0;                                  // d2 / dx dz at this y
    gx = fmaf(c.fz, xz, a0);
    gy = fmaf(c.fz, b1 - b0, b0);
    gz = fmaf(c.fx, xz, fmaf(c.fy, y1 - y0, c.v100 - c.v000));
}

// Register cap 96 (71 used, seven CTAs an SM): 0.74 and 6.52 ms at the sizes above,
// 2.62 for 32 poses x 256^2 x 800 of 512^3; scheduled under a cap of 80: 0.75, 6.64,
// 2.68; of 72: 0.75, 6.65, 2.70; 64 spill. Three samples in flight at 112: 0.80,
// 6.76, 2.78.
template <typename VT>
__global__ void __maxnreg__(96) raymarch_fwd_sums_kernel(const MarchParams p, float* __restrict__ sums) {
    const int tile = (int)(blockIdx.x % (unsigned)p.tm.tiles), b = (int)(blockIdx.x / (unsigned)p.tm.tiles);
    const int n = tile_ray(p.tm, p.N, p.tw, p.th, tile, threadIdx.x);
    if (n < 0) return;
    ThreadRay tr;
    {
        float m[12];
#pragma unroll
        for (int j = 0; j < 12; ++j) m[j] = __ldg(p.M + (size_t)b * 12 + j);
        init_thread_ray(p, m, b, n, tr);
    }
    // Offset of float position p0 + t d from the cell corner i. The march is
    // bound by issue (73 % of slots) and the conversion pipe is idle, so i is
    // converted: two instructions where forming it from bits took three.
    auto offset = [](float t, float d, float p0, int i) { return fmaf(t, d, p0) - (float)i; };
    int s = tr.ray.lo, s1 = tr.ray.hi;
    trim_inside(p, tr, s, s1);
    float acc = 0.f, G[3] = {0.f, 0.f, 0.f}, Gt[3] = {0.f, 0.f, 0.f};
    auto take = [&](float sf, Cell& c) {
        const float t = sf * p.inv_s;
        float dx, dy, dz;
        cell_grad_shared(c, dx, dy, dz);
        c.fx = offset(t, tr.ray.dx, tr.ray.p0x, c.ix);
        c.fy = offset(t, tr.ray.dy, tr.ray.p0y, c.iy);
        c.fz = offset(t, tr.ray.dz, tr.ray.p0z, c.iz);
        acc += cell_value(c);
        G[0] += dx;
        G[1] += dy;
        G[2] += dz;
        Gt[0] = fmaf(dx, t, Gt[0]);
        Gt[1] = fmaf(dy, t, Gt[1]);
        Gt[2] = fmaf(dz, t, Gt[2]);
    };
    for (; s + 1 < s1; s += 2) {
        const float sf = (float)s;
        Cell a, c;
        fetch_cell<VT, kLayoutQuad>(p, fix_at(tr, s), a);
        fetch_cell<VT, kLayoutQuad>(p, fix_at(tr, s + 1), c);
        take(sf, a);
        take(sf + 1.f, c);
    }
    if (s < s1) {
        Cell c;
        fetch_cell<VT, kLayoutQuad>(p, fix_at(tr, s), c);
        take((float)s, c);
    }
    st_out(reinterpret_cast<VT*>(p.out), tr.bn, acc * tr.stepv);
    const size_t rays = (size_t)p.B * p.N;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        sums[j * rays + tr.bn] = G[j];
        sums[(3 + j) * rays + tr.bn] = Gt[j];
    }
}

// Pose partials from the sums: a CTA takes kSumRays rays of a pose, each
// thread's in order, then the fixed shuffle tree; pose_partials_reduce_kernel
// sums the CTAs. Bound by reading 44 bytes per ray.
constexpr int kSumRays = 2048;

__global__ void __launch_bounds__(256) pose_sums_kernel(const MarchParams p, const float* __restrict__ sums,
                                                        int chunks) {
    __shared__ float red[8][12];
    const int b = (int)(blockIdx.x / (unsigned)chunks), chunk = (int)(blockIdx.x % (unsigned)chunks);
    const size_t rays = (size_t)p.B * p.N;
    float a[12];
#pragma unroll
    for (int j = 0; j < 12; ++j) a[j] = 0.f;
    const int end = min(p.N, (chunk + 1) * kSumRays);
    for (int n = chunk * kSumRays + (int)threadIdx.x; n < end; n += 256) {
        const size_t bn = (size_t)b * p.N + n;
        const float go = ld_any_f(p.go, p.go_dtype, bn);
        if (go == 0.f) continue;  // as the marching adjoint: every term is proportional to go
        const float g = go * __ldg(p.step + bn);
        const float* sp = p.src_per_ray ? p.src + bn * 3 : p.src + (size_t)b * 3;
        float s[3], e[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            s[j] = __ldg(sp + j);
            e[j] = __ldg(p.tgt + bn * 3 + j) - s[j];
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float G = g * __ldg(sums + i * rays + bn), Gt = g * __ldg(sums + (3 + i) * rays + bn);
#pragma unroll
            for (int j = 0; j < 3; ++j) a[4 * i + j] += fmaf(Gt, e[j], G * s[j]);
            a[4 * i + 3] += G;
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < 12; ++j) {
        const float v = warp_sum(a[j]);
        if (lane == 0) red[warp][j] = v;
    }
    __syncthreads();
    if (threadIdx.x < 12) {
        float v = red[0][threadIdx.x];
        for (int w = 1; w < 8; ++w) v += red[w][threadIdx.x];
        p.partials[(size_t)blockIdx.x * kPartialStride + threadIdx.x] = v;
    }
}

template <typename VT>
static cudaError_t fwd_sums(const MarchParams& p, float* sums, cudaStream_t st) {
    const KernelEvents& ev = kernel_events();
    if (ev.start != nullptr) cudaEventRecord(ev.start, st);
    raymarch_fwd_sums_kernel<VT><<<(unsigned)((size_t)p.B * p.tm.tiles), (unsigned)(p.tw * p.th), 0, st>>>(p, sums);
    cudaError_t e = cudaGetLastError();
    if (ev.stop != nullptr && e == cudaSuccess) e = cudaEventRecord(ev.stop, st);
    return e;
}

cudaError_t launch_fwd_sums(const ndrr_raymarch_args& a, LaunchShape ls, float* sums, cudaStream_t st) {
    ls.K = 1;
    const MarchParams p = make_params(a, ls);
    switch (a.vol_dtype) {
        case NDRR_F32: return fwd_sums<float>(p, sums, st);
        case NDRR_F16: return fwd_sums<__half>(p, sums, st);
        case NDRR_BF16: return fwd_sums<__nv_bfloat16>(p, sums, st);
        default: return cudaErrorInvalidValue;
    }
}

static int sum_chunks(int N) { return (N + kSumRays - 1) / kSumRays; }

uint64_t pose_sums_workspace_bytes(int B, int N) {
    return (uint64_t)B * sum_chunks(N) * kPartialStride * sizeof(float);
}

cudaError_t launch_pose_sums(const ndrr_raymarch_args& a, const float* sums, cudaStream_t st) {
    const MarchParams p = make_params(a, LaunchShape{});
    const int chunks = sum_chunks(a.N);
    pose_sums_kernel<<<(unsigned)((size_t)a.B * chunks), 256, 0, st>>>(p, sums, chunks);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_pose_reduce(p.partials, a.B, chunks, a.gM, nullptr, st);
}

}  // namespace ndrr
