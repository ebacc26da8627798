// Empty-space structures for the proposal-guided march.
//
// 1. Occupancy / distance grid. The volume is covered by cells of `cell`^3
//    voxels plus a one-cell border on every side; grid cell g (per axis) spans
//    voxels [(g - 1) * cell, g * cell). A cell is occupied when any voxel
//    within two voxels of it is non-zero: a sample whose floor position lies in
//    an unoccupied cell therefore has eight zero corners even if its position
//    is off by up to a voxel, so it contributes exactly nothing to the image,
//    the pose gradient or the camera gradients. The grid stores the Chebyshev
//    distance (in cells) to the nearest occupied cell, 0 for occupied cells,
//    capped at `max_dist`.
// 2. Extent labels. For every ray, the first and last sample of the box-culled
//    march whose eight corners are not all zero, as t = s / (S - 1) — the
//    non-empty interval the plain renderer itself sees (training labels for the
//    learned proposal).
#include <algorithm>

#include "ndrr_device.cuh"
#include "ndrr_launch.h"

namespace ndrr {

// ---------------------------------------------------------------- occupancy
// A CTA takes two planes of cells (along z) of a tile of cells in y and x, and
// reads its voxels once: a warp takes 128 voxels of a volume line, four per
// lane (one vector load where lines and base allow it), through the voxel
// planes that the two cell planes span, and leaves the line's non-zero bits
// per cell plane in shared memory; a cell is occupied when any line of its y
// range has a bit in its x range. Reading each cell's (cell + 4)^3 voxels per
// thread took 325 us at 512 x 512 x 400 (cell 4, every voxel read eight times
// through L1), this 142: every voxel is read 1.9 times, once from DRAM (62 us
// at copy speed). Tiles of 16 lines give CTAs enough for eight an SM in whole
// waves; with 64 lines (1.6 reads) and four voxel planes in flight, not six, it
// was 196. Six planes are half of a cell pair's twelve; 32 lines 144, 8 lines
// 145, 3 planes 153, 12 planes 160, four cell planes a CTA 182-195.
constexpr int kOccThreads = 256;
constexpr int kOccPlanes = 2;   // cell planes per CTA
constexpr int kOccLines = 16;   // volume lines of a tile's cells (without the two-voxel margins); one cell if larger
constexpr int kOccMaxCell = 64;
constexpr int kOccBatch = 6;    // voxel planes in flight
constexpr int kOccSpan = 1024;  // voxels in x of a tile's cells (without the margins)
constexpr int kOccWords = (kOccSpan / 128 + 2) * 4;

// Bits 0 .. 3: which of voxels x .. x + 3 of a line are non-zero (x < W).
template <typename VT, bool VEC>
__device__ __forceinline__ unsigned nonzero4(const VT* __restrict__ line, int x, int W) {
    unsigned m = 0u;
    if constexpr (VEC) {
        if (x < W) {
            if constexpr (sizeof(VT) == 4) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(line + x));
                m = (v.x != 0.f) | (v.y != 0.f) << 1 | (v.z != 0.f) << 2 | (v.w != 0.f) << 3;
            } else {  // 16-bit floats: non-zero apart from the sign
                const uint2 v = __ldg(reinterpret_cast<const uint2*>(line + x));
                m = ((v.x & 0x7fffu) != 0u) | ((v.x & 0x7fff0000u) != 0u) << 1 | ((v.y & 0x7fffu) != 0u) << 2 |
                    ((v.y & 0x7fff0000u) != 0u) << 3;
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (x + k < W) m |= (unsigned)(ld_vox(line, x + k) != 0.f) << k;
    }
    return m;
}

template <typename VT, bool VEC>
__global__ void __launch_bounds__(kOccThreads) occupancy_kernel(const VT* __restrict__ vol, int D, int H, int W,
                                                                int cell, int gx, int gy, int gz, int ty, int tx,
                                                                int tiles_y, int tiles_x, uint8_t* __restrict__ dist,
                                                                int max_dist) {
    __shared__ unsigned bits[kOccPlanes][kOccMaxCell + 4][kOccWords];
    const int tile = (int)(blockIdx.x % (unsigned)(tiles_x * tiles_y));
    const int cz0 = (int)(blockIdx.x / (unsigned)(tiles_x * tiles_y)) * kOccPlanes;
    const int cy0 = (tile / tiles_x) * ty, cx0 = (tile % tiles_x) * tx;
    // voxel ranges, clipped to the volume: cell c spans (c - 1) cell - 2 .. c cell + 1
    const int ylo = max((cy0 - 1) * cell - 2, 0), yhi = min((cy0 + ty - 1) * cell + 1, H - 1);
    const int xlo = max((cx0 - 1) * cell - 2, 0) & ~31, xhi = min((cx0 + tx - 1) * cell + 1, W - 1);
    const int chunks = xhi >= xlo ? (xhi - xlo) / 128 + 1 : 0;
    const int lines = yhi - ylo + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int zlo[kOccPlanes], zhi[kOccPlanes];
#pragma unroll
    for (int k = 0; k < kOccPlanes; ++k) {
        zlo[k] = max((cz0 + k - 1) * cell - 2, 0);
        zhi[k] = min((cz0 + k) * cell + 1, D - 1);
    }
    const size_t plane = (size_t)H * W;
    for (int item = warp; item < lines * chunks; item += kOccThreads / 32) {
        const int line = item / chunks, w = item - line * chunks;
        const int x = xlo + 128 * w + 4 * lane;
        const VT* p = vol + ((size_t)zlo[0] * H + (ylo + line)) * W;
        unsigned m[kOccPlanes];
#pragma unroll
        for (int k = 0; k < kOccPlanes; ++k) m[k] = 0u;
        int z = zlo[0];
        for (; z + kOccBatch - 1 <= zhi[kOccPlanes - 1]; z += kOccBatch, p += kOccBatch * plane) {
            unsigned v[kOccBatch];
#pragma unroll
            for (int j = 0; j < kOccBatch; ++j) v[j] = nonzero4<VT, VEC>(p + j * plane, x, W);
#pragma unroll
            for (int j = 0; j < kOccBatch; ++j)
#pragma unroll
                for (int k = 0; k < kOccPlanes; ++k)
                    if (z + j >= zlo[k] && z + j <= zhi[k]) m[k] |= v[j];
        }
        for (; z <= zhi[kOccPlanes - 1]; ++z, p += plane) {
            const unsigned v = nonzero4<VT, VEC>(p, x, W);
#pragma unroll
            for (int k = 0; k < kOccPlanes; ++k)
                if (z >= zlo[k] && z <= zhi[k]) m[k] |= v;
        }
#pragma unroll
        for (int k = 0; k < kOccPlanes; ++k) {
            unsigned v = m[k] << (4 * (lane & 7));  // eight lanes make a word of 32 voxels
            v |= __shfl_xor_sync(0xffffffffu, v, 1);
            v |= __shfl_xor_sync(0xffffffffu, v, 2);
            v |= __shfl_xor_sync(0xffffffffu, v, 4);
            if ((lane & 7) == 0) bits[k][line][4 * w + (lane >> 3)] = v;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kOccPlanes * ty * tx; i += kOccThreads) {
        const int k = i / (ty * tx), cy = cy0 + (i / tx) % ty, cx = cx0 + i % tx;
        if (cz0 + k >= gz || cy >= gy || cx >= gx) continue;
        const int y0 = max((cy - 1) * cell - 2, 0) - ylo, y1 = min(cy * cell + 1, H - 1) - ylo;
        const int x0 = max((cx - 1) * cell - 2, 0) - xlo, x1 = min(cx * cell + 1, W - 1) - xlo;
        bool occ = false;
        if (x0 <= x1) {
            const int w0 = x0 >> 5, w1 = x1 >> 5;
            const unsigned first = 0xffffffffu << (x0 & 31), last = 0xffffffffu >> (31 - (x1 & 31));
            for (int y = y0; y <= y1 && !occ; ++y)
                for (int w = w0; w <= w1; ++w) {
                    unsigned v = bits[k][y][w];
                    if (w == w0) v &= first;
                    if (w == w1) v &= last;
                    occ |= v != 0u;
                }
        }
        dist[((size_t)(cz0 + k) * gy + cy) * gx + cx] = occ ? 0 : (uint8_t)max_dist;
    }
}

// One axis of the capped Chebyshev distance transform, which is separable:
// d(i) = min over j of max(|j - i|, src(j)) along the axis, for the axes in
// turn. The search stops at the best distance so far. Three passes; relaxing
// over the 26 neighbours took max_dist of them (372 us for 16 at 130 x 130 x
// 102 cells, 60 now).
template <typename I>
__global__ void __launch_bounds__(256) distance_axis_kernel(const uint8_t* __restrict__ src,
                                                            uint8_t* __restrict__ dst, int gx, int gy, int gz,
                                                            int axis) {
    const I ncell = (I)gx * gy * gz;
    const I stride = axis == 0 ? 1 : (axis == 1 ? (I)gx : (I)gx * gy);
    const int len = axis == 0 ? gx : (axis == 1 ? gy : gz);
    for (I i = blockIdx.x * (I)blockDim.x + threadIdx.x; i < ncell; i += (I)gridDim.x * blockDim.x) {
        const int at = (int)((i / stride) % len);
        int d = __ldg(src + i);
        for (int r = 1; r < d; ++r) {
            int v = 255;
            if (at - r >= 0) v = __ldg(src + i - r * stride);
            if (at + r < len) v = min(v, (int)__ldg(src + i + r * stride));
            d = min(d, max(r, v));
        }
        dst[i] = (uint8_t)d;
    }
}

template <typename VT>
static cudaError_t occupancy(const void* vol, int D, int H, int W, int cell, int gx, int gy, int gz, int max_dist,
                             uint8_t* dist, cudaStream_t st) {
    const int ty = std::max(1, kOccLines / cell), tx = kOccSpan / cell;  // cell <= kOccMaxCell
    const int tiles_y = (gy + ty - 1) / ty, tiles_x = (gx + tx - 1) / tx;
    const long long grid = (long long)tiles_y * tiles_x * ((gz + kOccPlanes - 1) / kOccPlanes);
    const bool vec = W % 4 == 0 && (uintptr_t)vol % (4 * sizeof(VT)) == 0;  // vector loads of four voxels
    auto kern = vec ? occupancy_kernel<VT, true> : occupancy_kernel<VT, false>;
    kern<<<(unsigned)grid, kOccThreads, 0, st>>>((const VT*)vol, D, H, W, cell, gx, gy, gz, ty, tx, tiles_y, tiles_x,
                                                 dist, max_dist);
    return cudaGetLastError();
}

cudaError_t launch_occupancy(const void* vol, int vol_dtype, int D, int H, int W, int cell, int max_dist,
                             uint8_t* dist, uint8_t* scratch, cudaStream_t st) {
    const int gx = (W + cell - 1) / cell + 2, gy = (H + cell - 1) / cell + 2, gz = (D + cell - 1) / cell + 2;
    const long long ncell = (long long)gx * gy * gz;
    const int block = 256;
    const int grid = (int)std::min<long long>((ncell + block - 1) / block, 152LL * 64);
    cudaError_t e;
    switch (vol_dtype) {
        case NDRR_F32: e = occupancy<float>(vol, D, H, W, cell, gx, gy, gz, max_dist, scratch, st); break;
        case NDRR_F16: e = occupancy<__half>(vol, D, H, W, cell, gx, gy, gz, max_dist, scratch, st); break;
        case NDRR_BF16: e = occupancy<__nv_bfloat16>(vol, D, H, W, cell, gx, gy, gz, max_dist, scratch, st); break;
        default: return cudaErrorInvalidValue;
    }
    // scratch -> dist -> scratch -> dist
    for (int axis = 0; axis < 3 && e == cudaSuccess; ++axis) {
        const uint8_t* from = axis == 1 ? dist : scratch;
        uint8_t* to = axis == 1 ? scratch : dist;
        if (ncell < (1LL << 30))  // 32-bit indices, their step included
            distance_axis_kernel<unsigned><<<grid, block, 0, st>>>(from, to, gx, gy, gz, axis);
        else
            distance_axis_kernel<long long><<<grid, block, 0, st>>>(from, to, gx, gy, gz, axis);
        e = cudaGetLastError();
    }
    return e;
}

}  // namespace ndrr
