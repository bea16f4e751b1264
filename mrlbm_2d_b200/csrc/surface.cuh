// surface.cuh -- surface pressure on the cylinder, its Gaussian smoothing over theta, and the
// four wake probes (write_statistics_out / extrapolate_var_on_cylinder / gaussian_smoothing /
// quadratic_interpolation, 2d_mrlbm.f90:593-766, and the probe records, 2d_mrlbm.f90:462-476).
//
// Runs after a statistics step on the populations that step gathered, so it sees the field
// the reference's p = rho cs2 is computed from (2d_mrlbm.f90:236; p is not updated by the
// boundary closures).  Kernel A: per wall node, p at the bilinear stencils of reference points 2, 3
// and 4, quadratic extrapolation in r to the wall point, stored in theta order; the probes.
// Kernel B: the smoothing, p_fit(i) = sum_j W(i,j) ps(j) / sum_j W(i,j), with the weights
// exp(-(theta_i - theta_j)^2 / (2 sigma^2)) (sigma = 0.1) computed once on the host with the same
// libm the reference uses.  Every sum runs in the reference's index order.  Both are launched with
// programmatic dependence: A waits for the step, B for A, the next step for B.
#pragma once
#include "surface.h"
#include "step_fp64.cuh"

namespace mrlbm {
namespace surf {

// Populations of node (i, j) as the reference's f (FP64; FP32 storage adds back w_k).
template <class T>
__device__ __forceinline__ void gather_f(const StepParams<T>& p, int i, int j, double f[Q]) {
    T g[Q];
    gather(p, i, j, g);
#pragma unroll
    for (int k = 0; k < Q; ++k) f[k] = sizeof(T) == 8 ? (double)g[k] : (double)p.w[k] + (double)g[k];
}

template <class T>
__device__ __forceinline__ double node_p(const StepParams<T>& p, int i, int j) {
    T g[Q];
    double f[Q];
    gather_interior(p, i, j, g);                  // a stencil node is an interior fluid node
#pragma unroll
    for (int k = 0; k < Q; ++k) f[k] = sizeof(T) == 8 ? (double)g[k] : (double)p.w[k] + (double)g[k];
    double s = f[0];
    s = s + f[1]; s = s + f[2]; s = s + f[3]; s = s + f[4];
    s = s + f[5]; s = s + f[6]; s = s + f[7]; s = s + f[8];
    return s * (1.0 / 3.0);                       // p = rho * cs2, cs2 = 1.0d0/3.0d0
}

// Sixteen lanes per wall node, lane c < 12 with corner c % 4 of reference point 2 + c / 4: all of a node's
// 108 loads leave in one round trip, its tables before the wait for the step.  One thread per node took its twelve
// corners one after another (on one block, with the smoothing 33 us of a 41 us step at 800 x 200).
constexpr int SURF_THREADS = 128;
template <class T>
__global__ void __launch_bounds__(SURF_THREADS) surface_a(const __grid_constant__ StepParams<T> p, const __grid_constant__ SurfaceTables t,
                                                          double* rec, double* prec) {
    const int nb = t.nb, tid = threadIdx.x;
    if (blockIdx.x == gridDim.x - 1) {            // the probes
        wait_prior_grid();
        if (tid < 4 && prec) {
            const int i = t.probe_i[tid], j = t.probe_j[tid];
            double f[Q];
            gather_f(p, i, j, f);
            double rho, ux, uy;
            if (sizeof(T) == 8 && !is_interior(p, i, j)) {
                const fp64::Mac m = fp64::node_macro(reinterpret_cast<const StepParams<double>&>(p), i, j, f);
                rho = m.rho; ux = m.ux; uy = m.uy;
            } else {
                fp64::moments_u(f, rho, ux, uy);
            }
            prec[tid] = rho / 3.0;                 // 2d_mrlbm.f90:470-475: rho/3, ux/3, uy/3
            prec[4 + tid] = ux / 3.0;
            prec[8 + tid] = uy / 3.0;
        }
        return;
    }
    const int l = (int)blockIdx.x * (SURF_THREADS / 16) + (tid >> 4), c = min(tid & 15, 11), r = c >> 2;
    const int lt = min(l, nb - 1);
    const int si = __ldg(p.bint + (I_SI + c) * nb + lt), sj = __ldg(p.bint + (I_SJ + c) * nb + lt);
    const double xd = (double)__ldg(p.bgeo + (G_XD2 + 2 * r) * nb + lt), yd = (double)__ldg(p.bgeo + (G_YD2 + 2 * r) * nb + lt);
    const double r1 = t.quad[5 * lt], r2 = t.quad[5 * lt + 1], r3 = t.quad[5 * lt + 2];
    const double rs = t.quad[5 * lt + 3], denom = t.quad[5 * lt + 4];
    const int place = __ldg(t.place + lt);
    wait_prior_grid();
    const unsigned all = 0xffffffffu;
    const double p1 = node_p(p, si, sj);
    const double p2 = __shfl_down_sync(all, p1, 1, 16), p3 = __shfl_down_sync(all, p1, 2, 16), p4 = __shfl_down_sync(all, p1, 3, 16);
    const double v0 = (1.0 - xd) * p1 + xd * p2;
    const double v1 = (1.0 - xd) * p3 + xd * p4;
    const double var = (1.0 - yd) * v0 + yd * v1;
    // quadratic_interpolation(x2,y2,var2, x3,y3,var3, x4,y4,var4, xs,ys): its (r1, r2, r3)
    // are the radii of points 2, 3, 4 and rs that of the wall point
    const double q1 = __shfl_sync(all, var, 0, 16), q2 = __shfl_sync(all, var, 4, 16), q3 = __shfl_sync(all, var, 8, 16);
    const double a0 = (r1 * r3 * q2 * (r3 - r1) + (r2 * r2) * (r3 * q1 - r1 * q3) + r2 * ((r1 * r1) * q3 - (r3 * r3) * q1)) / denom;
    const double a1 = ((r3 * r3) * (q1 - q2) + (r1 * r1) * (q2 - q3) + (r2 * r2) * (q3 - q1)) / denom;
    const double a2 = (r3 * (q2 - q1) + r2 * (q1 - q3) + r1 * (q3 - q2)) / denom;
    if (l < nb && (tid & 15) == 0) rec[place] = a0 + a1 * rs + a2 * (rs * rs);
}

// Smoothing: a block has 32 wall points; its warps form the products of SURF_ROWS terms of each in shared
// memory, the next round's weights already on their way, and warp 0 adds them in the reference's order.
// The weights are a table, so the first round's are loaded before the wait.
constexpr int SURF_ROWS = 64, SURF_B_THREADS = 256;
__global__ void __launch_bounds__(SURF_B_THREADS) surface_b(const __grid_constant__ SurfaceTables t, double* rec) {
    __shared__ double prod[SURF_ROWS][32];
    constexpr int R = SURF_ROWS * 32 / SURF_B_THREADS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nb = t.nb;
    const int i = blockIdx.x * 32 + lane;
    double w[R];
    auto weights = [&](int j0) {
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int j = j0 + u * (SURF_B_THREADS / 32) + warp;
            w[u] = i < nb && j < nb ? __ldg(t.W + (size_t)j * nb + i) : 0.0;
        }
    };
    weights(0);
    const double sumw = i < nb ? __ldg(t.sumw + i) : 1.0;
    wait_prior_grid();
    double s = 0.0;
    for (int j0 = 0; j0 < nb; j0 += SURF_ROWS) {
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int q = u * (SURF_B_THREADS / 32) + warp;
            prod[q][lane] = j0 + q < nb ? w[u] * rec[j0 + q] : 0.0;
        }
        __syncthreads();
        weights(j0 + SURF_ROWS);
        if (warp == 0) {
            const int m = min(SURF_ROWS, nb - j0);
#pragma unroll 16
            for (int q = 0; q < m; ++q) s = s + prod[q][lane];
        }
        __syncthreads();
    }
    if (warp == 0 && i < nb) rec[nb + i] = s / sumw;
}

template <class T>
int launch_surface(const StepParams<T>& p, const SurfaceTables& t, double* rec, double* prec, cudaStream_t s) {
    if (t.nb <= 0) return 0;
    const unsigned ga = (unsigned)((t.nb + SURF_THREADS / 16 - 1) / (SURF_THREADS / 16)) + 1, gb = (unsigned)((t.nb + 31) / 32);
    return launch_after_prior(surface_a<T>, ga, SURF_THREADS, 0, s, p, t, rec, prec) == cudaSuccess &&
                   launch_after_prior(surface_b, gb, SURF_B_THREADS, 0, s, t, rec) == cudaSuccess
               ? 0
               : -1;
}

}  // namespace surf
}  // namespace mrlbm
