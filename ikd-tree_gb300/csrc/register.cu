// Point-to-plane scan-to-map residuals and their adjoint.
//
// The reference stops at Nearest_Search; its main consumer (FAST-LIO2) fits a
// plane through the k neighbours of every transformed scan point and
// minimises the point-to-plane residuals.  This file provides that step on
// the GPU, next to the kNN it builds on:
//
//   w_i = R(omega) p_i + t                      (scan point to map frame)
//   plane through the k neighbours of w_i:      min |A x + 1|^2,  A = [m_j^T]
//     (solved by an orthogonal factorisation, as FAST-LIO2's QR solve: the
//     normal equations square the condition number of A, which is large for
//     planes far from the origin or nearly through it)
//   n_i = x / |x|,  d_i = 1 / |x|               (plane n . q + d = 0)
//   valid_i  if every |n_i . m_j + d_i| <= plane_thresh
//   r_i = n_i . w_i + d_i,   L = 1/2 sum_valid r_i^2
// Each plane is stored as {n, d} and a point c on it (the neighbours' centroid
// projected onto the plane); residuals are evaluated as n . (w - c) in double
// from the double pose, which avoids cancelling two ~|w|-sized terms.
//
// With the neighbour sets held fixed, the planes do not depend on the pose, so
// the adjoint is closed form:
//   g_i = dL * r_i * n_i;   dL/dt = sum g_i;   dL/dp_i = R^T g_i;
//   dL/domega = J_r(omega)^T sum_i p_i x (R^T g_i)
// (J_r: right Jacobian of the SO(3) exponential).
#include <cuda_runtime.h>

#include "kernels.cuh"

namespace ikdg {
namespace {

// 64 threads per CTA: a 20k-point scan fills every SM (the doubles of a point are
// a long chain, and an SM has few double units).
constexpr int RG_THREADS = 64;

__device__ __forceinline__ void transform_d(const RegPose& P, double x, double y, double z, double w[3]) {
    for (int r = 0; r < 3; ++r)
        w[r] = fma(P.R[3 * r], x, fma(P.R[3 * r + 1], y, fma(P.R[3 * r + 2], z, P.t[r])));
}

__global__ void transform_kernel(const float* __restrict__ p, long long n, RegPose P, float* __restrict__ w) {
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double wd[3];
    transform_d(P, p[3 * i], p[3 * i + 1], p[3 * i + 2], wd);
    for (int r = 0; r < 3; ++r) w[3 * i + r] = (float)wd[r];
}

// Least squares min |A x - b| for the k rows of A (k x 3) and b by a QR
// factorisation built one row at a time with Givens rotations (R upper
// triangular 3 x 3, z = Q^T b), then back substitution.  Returns false when R
// is singular.  The rows are floats, so the squares neither overflow nor
// underflow in double and a rotation needs one reciprocal square root (hypot and
// two divisions before: the double units bound the kernel, 20k points, k = 5:
// 62 us before, 25 now).
__device__ __forceinline__ bool lsq3_givens(const float* __restrict__ rows, int k, double b_all, double x[3]) {
    double R[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    double z[3] = {0, 0, 0};
    for (int j = 0; j < k; ++j) {
        double r[3] = {rows[3 * j], rows[3 * j + 1], rows[3 * j + 2]};
        double b = b_all;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (r[c] == 0.0) continue;
            const double inv = rsqrt(fma(R[c][c], R[c][c], r[c] * r[c]));
            const double cs = R[c][c] * inv, sn = r[c] * inv;
#pragma unroll
            for (int m = c; m < 3; ++m) {
                const double t = fma(cs, R[c][m], sn * r[m]);
                r[m] = fma(cs, r[m], -sn * R[c][m]);
                R[c][m] = t;
            }
            const double t = fma(cs, z[c], sn * b);
            b = fma(cs, b, -sn * z[c]);
            z[c] = t;
        }
    }
    const double scale = fmax(fabs(R[0][0]), fmax(fabs(R[1][1]), fabs(R[2][2])));
    for (int c = 0; c < 3; ++c)
        if (!(fabs(R[c][c]) > 1e-12 * scale)) return false;
    x[2] = z[2] / R[2][2];
    x[1] = (z[1] - R[1][2] * x[2]) / R[1][1];
    x[0] = (z[0] - R[0][1] * x[1] - R[0][2] * x[2]) / R[0][0];
    return true;
}

// Sum of v over the block, valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0;
    if (threadIdx.x == 0)
        for (int i = 0; i < RG_THREADS / 32; ++i) s += sh[i];
    __syncthreads();
    return s;
}

// Plane fit (least squares by Givens QR) and residual; per block the sum of
// 1/2 r^2 over its valid points.
__global__ void __launch_bounds__(RG_THREADS) plane_residual_kernel(const float* __restrict__ p, RegPose P, long long n,
                                                                    int k, const float* __restrict__ nb,
                                                                    const int* __restrict__ cnt, float thresh,
                                                                    float4* __restrict__ planes,
                                                                    float* __restrict__ res, int* __restrict__ valid,
                                                                    double* __restrict__ partial) {
    __shared__ double sh[RG_THREADS / 32];
    double loss = 0;
    for (long long i = (long long)blockIdx.x * RG_THREADS + threadIdx.x; i < n;
         i += (long long)gridDim.x * RG_THREADS) {
        float4 pl = make_float4(0.f, 0.f, 0.f, 0.f);
        float4 pc = make_float4(0.f, 0.f, 0.f, 0.f);
        int ok = 0;
        float r = 0.f;
        double xs[3];
        if (cnt[i] >= k && k >= 3 && lsq3_givens(nb + i * k * 3, k, -1.0, xs)) {
            const double x0 = xs[0], x1 = xs[1], x2 = xs[2];
            const double nrm = sqrt(fma(x0, x0, fma(x1, x1, x2 * x2)));
            if (nrm > 0) {
                const double dd = 1.0 / nrm;
                const double nx = x0 * dd, ny = x1 * dd, nz = x2 * dd;
                double cx = 0, cy = 0, cz = 0;
                ok = 1;
                for (int j = 0; j < k; ++j) {
                    const float* m = nb + (i * k + j) * 3;
                    const double mx = m[0], my = m[1], mz = m[2];
                    const double e = fma(nx, mx, fma(ny, my, fma(nz, mz, dd)));
                    if (fabs(e) > thresh) ok = 0;
                    cx += mx;
                    cy += my;
                    cz += mz;
                }
                const double ik = 1.0 / k;
                cx *= ik;
                cy *= ik;
                cz *= ik;
                const double off = fma(nx, cx, fma(ny, cy, fma(nz, cz, dd)));  // centroid -> plane
                cx = fma(-off, nx, cx);
                cy = fma(-off, ny, cy);
                cz = fma(-off, nz, cz);
                pl = make_float4((float)nx, (float)ny, (float)nz, (float)dd);
                pc = make_float4((float)cx, (float)cy, (float)cz, 0.f);
                if (ok) {
                    double wd[3];
                    transform_d(P, p[3 * i], p[3 * i + 1], p[3 * i + 2], wd);
                    r = (float)fma((double)pl.x, wd[0] - (double)pc.x,
                                   fma((double)pl.y, wd[1] - (double)pc.y, (double)pl.z * (wd[2] - (double)pc.z)));
                    loss = fma(0.5 * (double)r, (double)r, loss);
                }
            }
        }
        planes[2 * i] = pl;
        planes[2 * i + 1] = pc;
        res[i] = r;
        valid[i] = ok;
    }
    loss = block_sum(loss, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = loss;
}

// Adjoint: per point dL/dp_i; per block partial sums of g (for t) and
// p x (R^T g) (for omega, before J_r^T).
__global__ void __launch_bounds__(RG_THREADS) adjoint_kernel(const float* __restrict__ p, long long n, RegPose P,
                               const float4* __restrict__ planes, const float* __restrict__ res,
                               const int* __restrict__ valid, float dl, float* __restrict__ grad_p,
                               double* __restrict__ partial) {
    __shared__ double sh[RG_THREADS / 32];
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (long long i = (long long)blockIdx.x * RG_THREADS + threadIdx.x; i < n;
         i += (long long)gridDim.x * RG_THREADS) {
        double gx = 0, gy = 0, gz = 0;
        if (valid[i]) {
            const double s = (double)dl * (double)res[i];
            const float4 pl = planes[2 * i];
            gx = s * pl.x;
            gy = s * pl.y;
            gz = s * pl.z;
        }
        // v = R^T g  (R row-major)
        const double vx = fma(P.R[0], gx, fma(P.R[3], gy, P.R[6] * gz));
        const double vy = fma(P.R[1], gx, fma(P.R[4], gy, P.R[7] * gz));
        const double vz = fma(P.R[2], gx, fma(P.R[5], gy, P.R[8] * gz));
        if (grad_p != nullptr) {
            grad_p[3 * i] = (float)vx;
            grad_p[3 * i + 1] = (float)vy;
            grad_p[3 * i + 2] = (float)vz;
        }
        const double px = p[3 * i], py = p[3 * i + 1], pz = p[3 * i + 2];
        acc[0] += gx;
        acc[1] += gy;
        acc[2] += gz;
        acc[3] = fma(py, vz, fma(-pz, vy, acc[3]));
        acc[4] = fma(pz, vx, fma(-px, vz, acc[4]));
        acc[5] = fma(px, vy, fma(-py, vx, acc[5]));
    }
    for (int c = 0; c < 6; ++c) {
        const double s = block_sum(acc[c], sh);
        if (threadIdx.x == 0) partial[blockIdx.x * 6 + c] = s;
    }
}

inline unsigned blocks_for(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

int reg_blocks(long long n) {
    long long b = (n + RG_THREADS - 1) / RG_THREADS;
    return (int)(b < 2048 ? (b > 0 ? b : 1) : 2048);
}

void launch_transform(const float* p, long long n, const RegPose& pose, float* w, cudaStream_t s) {
    if (n <= 0) return;
    transform_kernel<<<blocks_for(n, 128), 128, 0, s>>>(p, n, pose, w);
}

void launch_plane_residual(const float* p, const RegPose& pose, long long n, int k, const float* nb, const int* cnt,
                           float thresh, float4* planes, float* res, int* valid, double* partial, cudaStream_t s) {
    if (n <= 0) return;
    plane_residual_kernel<<<reg_blocks(n), RG_THREADS, 0, s>>>(p, pose, n, k, nb, cnt, thresh, planes, res, valid,
                                                               partial);
}

void launch_adjoint(const float* p, long long n, const RegPose& pose, const float4* planes, const float* res,
                    const int* valid, float dl, float* grad_p, double* partial, cudaStream_t s) {
    if (n <= 0) return;
    adjoint_kernel<<<reg_blocks(n), RG_THREADS, 0, s>>>(p, n, pose, planes, res, valid, dl, grad_p, partial);
}

}  // namespace ikdg
