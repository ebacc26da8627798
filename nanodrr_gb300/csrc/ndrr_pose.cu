// Registration pose on the device (ndrr_pose_so3_fwd/bwd): the reference's
// Registration.pose (registration/registration.py:64-68) for the "so3_log"
// parameterisation (geometry/se3.py:179-221),
//   pose = rt_inv @ pivot @ T @ pivot_inv,  T = [[R, R xyz], [0, 1]],
//   R = exp([v]x) = I + a K + b K^2,  K = [v]x,
//   a = sin(t) / t,  b = (1 - cos t) / t^2,  t = |v|,
// and its adjoint to (v, xyz). One warp per pose in float64: the handful
// of 4x4 products replace about thirty elementwise torch launches per
// direction, and float64 keeps b and the derivatives of a and b accurate
// where float32 cancels (t between 1e-4 and 1e-2).
#include <cuda_runtime.h>

#include "../../include/nanodrr_gb300.h"

namespace ndrr {

constexpr int kPoseBlock = 64;

// a, b and their derivatives divided by t (da/dv = ca v, db/dv = cb v).
// Below t = 0.1 the Taylor series (error < 1e-15 there), above it the
// closed forms, whose cancellation in float64 stays below 1e-10 relative.
__device__ __forceinline__ void rodrigues_coefficients(double t2, double& a, double& b, double& ca, double& cb) {
    if (t2 < 1e-2) {
        a = 1.0 + t2 * (-1.0 / 6 + t2 * (1.0 / 120 + t2 * (-1.0 / 5040 + t2 * (1.0 / 362880))));
        b = 0.5 + t2 * (-1.0 / 24 + t2 * (1.0 / 720 + t2 * (-1.0 / 40320 + t2 * (1.0 / 3628800))));
        ca = -1.0 / 3 + t2 * (1.0 / 30 + t2 * (-1.0 / 840 + t2 * (1.0 / 45360)));
        cb = -1.0 / 12 + t2 * (1.0 / 180 + t2 * (-1.0 / 6720 + t2 * (1.0 / 453600)));
    } else {
        const double t = sqrt(t2), s = sin(t), c = cos(t);
        a = s / t;
        b = (1.0 - c) / t2;
        ca = (t * c - s) / (t2 * t);
        cb = (t * s - 2.0 + 2.0 * c) / (t2 * t2);
    }
}

// One warp per pose: lane l < 16 owns entry (l / 4, l % 4) of every 4x4
// matrix, exchanged through shared memory. What bounds these kernels is the
// fp64 pipe, which takes a warp instruction every 16 cycles whatever its
// active lanes, and the chain of dependent operations: one thread per pose
// issued about 400 of them (12 and 14 us); 16 lanes issue 40 and 80 (3.7 and
// 5.3 us).
struct PoseShared {
    double A[16], P[16], C[16], G[16], X[16], Y[16];
    double K[3][3], K2[3][3], R[3][3];
};

struct PoseCoef {
    double v[3], x[3], a, b, ca, cb;
};

__device__ __forceinline__ double mul_entry(const double* A, const double* B, int i, int j) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 4; ++k) s += A[4 * i + k] * B[4 * k + j];
    return s;
}

// Loads the pose's matrices, forms K, K^2, R and leaves rt_inv @ pivot in X.
__device__ __forceinline__ void pose_setup(PoseShared& q, PoseCoef& c, const float* rot, const float* xyz, int row,
                                           const float* rt_inv, const float* pivot, const float* pivot_inv, int b,
                                           int l) {
    const int i = l >> 2, j = l & 3;
    if (l < 16) {
        q.A[l] = (double)rt_inv[(size_t)b * 16 + l];
        q.P[l] = (double)pivot[(size_t)b * 16 + l];
        q.C[l] = (double)pivot_inv[(size_t)b * 16 + l];
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        c.v[k] = (double)rot[row * 3 + k];
        c.x[k] = (double)xyz[row * 3 + k];
    }
    const double vx = c.v[0], vy = c.v[1], vz = c.v[2];
    rodrigues_coefficients(vx * vx + vy * vy + vz * vz, c.a, c.b, c.ca, c.cb);
    const bool rotation = l < 16 && i < 3 && j < 3;
    if (rotation) {  // K = [v]x: row i has -v at the axis after i's next, v at its next
        const int n = 3 - i - j;  // the third axis (i != j)
        q.K[i][j] = i == j ? 0.0 : ((j - i + 3) % 3 == 1 ? -1.0 : 1.0) * c.v[n];
    }
    __syncwarp();
    if (rotation) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) s += q.K[i][k] * q.K[k][j];
        q.K2[i][j] = s;
        q.R[i][j] = (i == j ? 1.0 : 0.0) + c.a * q.K[i][j] + c.b * s;
    }
    if (l < 16) q.X[l] = mul_entry(q.A, q.P, i, j);
    __syncwarp();
}

__global__ void __launch_bounds__(kPoseBlock) pose_so3_fwd_kernel(const float* __restrict__ rot,
                                                                  const float* __restrict__ xyz, int param_rows,
                                                                  const float* __restrict__ rt_inv,
                                                                  const float* __restrict__ pivot,
                                                                  const float* __restrict__ pivot_inv, int B,
                                                                  float* __restrict__ pose) {
    __shared__ PoseShared sh[kPoseBlock / 32];
    const int l = threadIdx.x & 31, b = blockIdx.x * (kPoseBlock / 32) + (threadIdx.x >> 5);
    if (b >= B) return;  // whole warps
    PoseShared& q = sh[threadIdx.x >> 5];
    PoseCoef c;
    pose_setup(q, c, rot, xyz, param_rows == 1 ? 0 : b, rt_inv, pivot, pivot_inv, b, l);
    const int i = l >> 2, j = l & 3;
    if (l < 16) {
        if (i == 3)
            q.Y[l] = j == 3 ? 1.0 : 0.0;
        else
            q.Y[l] = j < 3 ? q.R[i][j] : q.R[i][0] * c.x[0] + q.R[i][1] * c.x[1] + q.R[i][2] * c.x[2];
    }
    __syncwarp();
    const double at = l < 16 ? mul_entry(q.X, q.Y, i, j) : 0.0;
    __syncwarp();
    if (l < 16) q.X[l] = at;
    __syncwarp();
    if (l < 16) pose[(size_t)b * 16 + l] = (float)mul_entry(q.X, q.C, i, j);
}

// gT = (rt_inv pivot)^T gpose pivot_inv^T; gR = gT[:3, :3] + gT[:3, 3] xyz^T,
// g_xyz = R^T gT[:3, 3]; g_v = (ca <gR, K> + cb <gR, K^2>) v + a vee(gR)
// + b vee(gR K^T + K^T gR), with vee(G) = (G21 - G12, G02 - G20, G10 - G01)
// the gradient of <G, [v]x> in v.
__global__ void __launch_bounds__(kPoseBlock) pose_so3_bwd_kernel(const float* __restrict__ gpose,
                                                                  const float* __restrict__ rot,
                                                                  const float* __restrict__ xyz, int param_rows,
                                                                  const float* __restrict__ rt_inv,
                                                                  const float* __restrict__ pivot,
                                                                  const float* __restrict__ pivot_inv, int B,
                                                                  float* __restrict__ g_rot,
                                                                  float* __restrict__ g_xyz) {
    __shared__ PoseShared sh[kPoseBlock / 32];
    const int l = threadIdx.x & 31, b = blockIdx.x * (kPoseBlock / 32) + (threadIdx.x >> 5);
    if (b >= B) return;  // whole warps
    PoseShared& q = sh[threadIdx.x >> 5];
    PoseCoef c;
    if (l < 16) q.G[l] = (double)gpose[(size_t)b * 16 + l];
    pose_setup(q, c, rot, xyz, param_rows == 1 ? 0 : b, rt_inv, pivot, pivot_inv, b, l);
    const int i = l >> 2, j = l & 3;
    if (l < 16) {  // L = (rt_inv pivot)^T gpose
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) s += q.X[4 * k + i] * q.G[4 * k + j];
        q.Y[l] = s;
    }
    __syncwarp();
    if (l < 16) {  // gT = L pivot_inv^T
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) s += q.Y[4 * i + k] * q.C[4 * j + k];
        q.G[l] = s;
    }
    __syncwarp();
    const bool rotation = l < 16 && i < 3 && j < 3;
    if (rotation) q.P[3 * i + j] = q.G[l] + q.G[4 * i + 3] * c.x[j];  // gR
    if (l < 3)
        g_xyz[(size_t)b * 3 + l] = (float)(q.R[0][l] * q.G[3] + q.R[1][l] * q.G[7] + q.R[2][l] * q.G[11]);
    __syncwarp();
    const double* gR = q.P;
    double sK = 0.0, sK2 = 0.0;
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        sK += gR[k] * q.K[k / 3][k % 3];
        sK2 += gR[k] * q.K2[k / 3][k % 3];
    }
    if (rotation) {  // H = gR K^T + K^T gR
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) s += gR[3 * i + k] * q.K[j][k] + q.K[k][i] * gR[3 * k + j];
        q.A[3 * i + j] = s;
    }
    __syncwarp();
    if (l < 3) {
        const double* H = q.A;
        const int u = (l + 2) % 3, w = (l + 1) % 3;  // vee(G)_l = G[u][w] - G[w][u]
        const double radial = c.ca * sK + c.cb * sK2;
        const double vr = gR[3 * u + w] - gR[3 * w + u], vh = H[3 * u + w] - H[3 * w + u];
        const double v = l == 0 ? c.v[0] : (l == 1 ? c.v[1] : c.v[2]);
        g_rot[(size_t)b * 3 + l] = (float)(radial * v + c.a * vr + c.b * vh);
    }
}

static unsigned pose_grid(int B) { return (unsigned)((B + kPoseBlock / 32 - 1) / (kPoseBlock / 32)); }

cudaError_t launch_pose_fwd(const float* rot, const float* xyz, int param_rows, const float* rt_inv,
                            const float* pivot, const float* pivot_inv, int B, float* pose, cudaStream_t st) {
    pose_so3_fwd_kernel<<<pose_grid(B), kPoseBlock, 0, st>>>(rot, xyz, param_rows, rt_inv, pivot, pivot_inv, B, pose);
    return cudaGetLastError();
}

cudaError_t launch_pose_bwd(const float* gpose, const float* rot, const float* xyz, int param_rows,
                            const float* rt_inv, const float* pivot, const float* pivot_inv, int B, float* g_rot,
                            float* g_xyz, cudaStream_t st) {
    pose_so3_bwd_kernel<<<pose_grid(B), kPoseBlock, 0, st>>>(gpose, rot, xyz, param_rows, rt_inv, pivot, pivot_inv, B,
                                                             g_rot, g_xyz);
    return cudaGetLastError();
}

}  // namespace ndrr
