// adjoint.cuh -- discrete adjoint of the FP64 step for the gradient of time-averaged drag.
//
// State of step n: the post-collision field F^n (the buffer a step writes).  Step n maps
// F^{n-1} to F^n node by node: node x gathers its inputs g_x from F^{n-1} (pull streaming),
// and its local map C_x gives the nine outputs F^n(x, :).  With J = (1/T) sum_{n in window}
// D^n, D^n the net drag of step n (a function of the wall nodes' inputs and outputs), the
// adjoint field lambda^n = dJ/dF^n obeys
//     lambda^{n-1}(slot) = sum over the consumers x of the slot of (dC_x/dg_x)^T lambda^n(x)
//                          + w_n dD^n/dF^{n-1}(slot),      w_n = 1/T inside the window,
// and the parameter gradients collect (dC_x/dtheta)^T lambda^n(x).  One adjoint step is one
// launch with three kinds of blocks, each node's contribution added atomically to
// lambda^{n-1} at the slots it pulled (a slot can feed several nodes: stencils, the outlet
// copy, corner wraps):
//   * bulk nodes (fluid and solid, not edge nodes, not curved-wall nodes): reverse mode
//     written out by hand: reconstruction -> collision -> moments (adjoint_bulk_node);
//   * edge nodes (inlet column i = 1, outlet column i = nx, and with no-slip reference walls
//     rows 1 and ny): one thread per (node, input), the node's
//     local map evaluated on dual numbers carrying the derivative along that input, then
//     contracted with lambda^n (the transposed Jacobian column); the inlet's extra input is
//     u_in(j), whose column gives the inlet-profile gradient;
//   * curved-wall nodes, their drag contribution in the same pass: reverse mode by hand (adjoint_wall);
//     with the unrotated closure on dual numbers like the edge nodes, over the node's 9 own inputs and
//     the 72 inputs of its 8 bilinear stencil nodes.
// The local maps below restate the FP64 step's arithmetic (step_fp64.cuh) for a generic
// scalar; they cover every closure of the FP64 step: the curved-wall closures (rotated
// strong, weak and rho_eq, unrotated with Cramer's rule, none) with or without velocity and
// moment extrapolation; inlet and outlet edge closures and no-slip
// reference walls, each in its apply_bc and apply_bc_incomp form; free-slip or y-periodic top
// and bottom; the incomp_bulk collision.
#pragma once
#include "adjoint.h"
#include "step_fp64.cuh"

namespace mrlbm {
namespace adj {

// Populations of node (i, j) as FP64 f: FP64 storage as is, FP32 storage holds f - w_k.
template <class T>
__device__ __forceinline__ double to_f(const StepParams<T>& p, int k, T v) {
    return sizeof(T) == 8 ? (double)v : (double)p.w[k] + (double)v;
}

template <class T>
__device__ __forceinline__ void gather_d(const StepParams<T>& p, int i, int j, double f[Q]) {
    T g[Q];
    gather(p, i, j, g);
#pragma unroll
    for (int k = 0; k < Q; ++k) f[k] = to_f(p, k, g[k]);
}

template <class T>
__device__ __forceinline__ void edge_gather_d(const StepParams<T>& p, int i, int j, double f[Q]) {
    T g[Q];
    edge_gather(p, i, j, g);
#pragma unroll
    for (int k = 0; k < Q; ++k) f[k] = to_f(p, k, g[k]);
}

// ---- dual numbers (value, derivative along one input) -----------------------------------
struct Dual {
    double v, d;
    __device__ Dual() : v(0.0), d(0.0) {}
    __device__ Dual(double a) : v(a), d(0.0) {}
    __device__ Dual(double a, double b) : v(a), d(b) {}
};
__device__ __forceinline__ Dual operator+(Dual a, Dual b) { return Dual(a.v + b.v, a.d + b.d); }
__device__ __forceinline__ Dual operator-(Dual a, Dual b) { return Dual(a.v - b.v, a.d - b.d); }
__device__ __forceinline__ Dual operator-(Dual a) { return Dual(-a.v, -a.d); }
__device__ __forceinline__ Dual operator*(Dual a, Dual b) { return Dual(a.v * b.v, a.d * b.v + a.v * b.d); }
// (one division each: a division is some 40 instructions, and the edge nodes' maps divide seven times in a
// row.  The gradient over 400 steps of 512 x 128: 7.79 ms, with two divisions 8.11)
__device__ __forceinline__ Dual operator/(Dual a, Dual b) {
    const double r = 1.0 / b.v, q = quotient(a.v, b.v, r);
    return Dual(q, quotient(a.d - q * b.d, b.v, r));
}
__device__ __forceinline__ Dual operator+(Dual a, double b) { return Dual(a.v + b, a.d); }
__device__ __forceinline__ Dual operator+(double a, Dual b) { return Dual(a + b.v, b.d); }
__device__ __forceinline__ Dual operator-(Dual a, double b) { return Dual(a.v - b, a.d); }
__device__ __forceinline__ Dual operator-(double a, Dual b) { return Dual(a - b.v, -b.d); }
__device__ __forceinline__ Dual operator*(Dual a, double b) { return Dual(a.v * b, a.d * b); }
__device__ __forceinline__ Dual operator*(double a, Dual b) { return Dual(a * b.v, a * b.d); }
__device__ __forceinline__ Dual operator/(Dual a, double b) {
    const double r = 1.0 / b;
    return Dual(quotient(a.v, b, r), quotient(a.d, b, r));
}
__device__ __forceinline__ Dual operator/(double a, Dual b) {
    const double r = 1.0 / b.v, q = quotient(a, b.v, r);
    return Dual(q, quotient(-q * b.d, b.v, r));
}

template <class S>
struct MacS { S rho, ux, uy, mxx, myy, mxy; };

template <class S>
__device__ __forceinline__ MacS<S> moments_s(const S f[Q], double hm, double hp) {
    MacS<S> m;
    S r = f[0];
    for (int k = 1; k < Q; ++k) r = r + f[k];
    const S inv = 1.0 / r;
    const S sx = ((((f[1] - f[3]) + f[5]) - f[6]) - f[7]) + f[8];
    const S sy = ((((f[2] - f[4]) + f[5]) + f[6]) - f[7]) - f[8];
    S sxx = f[0] * hm, syy = f[0] * hm;
#pragma unroll
    for (int k = 1; k < Q; ++k) {
        sxx = sxx + f[k] * (ex(k) != 0 ? hp : hm);
        syy = syy + f[k] * (ey(k) != 0 ? hp : hm);
    }
    const S sxy = ((f[5] - f[6]) + f[7]) - f[8];
    m.rho = r;
    m.ux = sx * inv;
    m.uy = sy * inv;
    m.mxx = sxx * inv;
    m.myy = syy * inv;
    m.mxy = sxy * inv;
    return m;
}

// Collision (2d_mrlbm.f90:407-415, incomp_bulk 419-428) and Hermite reconstruction
// (2d_mrlbm.f90:445-457).
template <class P, class S>
__device__ __forceinline__ void collide_s(const P& p, const MacS<S>& m, S fo[Q]) {
    const double om = p.omega, om1 = p.omega1;
    S mxx = om1 * m.mxx + om * m.ux * m.ux;
    S myy = om1 * m.myy + om * m.uy * m.uy;
    const S mxy = om1 * m.mxy + om * m.ux * m.uy;
    if (p.incomp_bulk) {
        const S t = 0.5 * (((mxx + myy) - m.ux * m.ux) - m.uy * m.uy);
        mxx = mxx - t;
        myy = myy - t;
    }
    const S a = 4.5 * mxx, b = 4.5 * myy, c = 9.0 * mxy;
    const S am = a * p.hm, ap = a * p.hp, bm = b * p.hm, bp = b * p.hp;
    const S t1 = 3.0 * m.ux, t2 = 3.0 * m.uy, t5 = 3.0 * (m.ux + m.uy), t8 = 3.0 * (m.ux - m.uy);
    const S w0 = p.w[0] * m.rho, w1 = p.w[1] * m.rho, w5 = p.w[5] * m.rho;
    fo[0] = w0 * ((1.0 + am) + bm);
    fo[1] = w1 * (((1.0 + t1) + ap) + bm);
    fo[2] = w1 * (((1.0 + t2) + am) + bp);
    fo[3] = w1 * (((1.0 - t1) + ap) + bm);
    fo[4] = w1 * (((1.0 - t2) + am) + bp);
    fo[5] = w5 * ((((1.0 + t5) + ap) + bp) + c);
    fo[6] = w5 * ((((1.0 - t8) + ap) + bp) - c);
    fo[7] = w5 * ((((1.0 - t5) + ap) + bp) + c);
    fo[8] = w5 * ((((1.0 + t8) + ap) + bp) - c);
}

// Sums over an incoming mask normalised by rho_I (apply_bc prologue, 2d_mrlbm.f90:1249-1269).
template <class S>
__device__ __forceinline__ void incoming_s(const S f[Q], int mask, double hm, double hp, S& rhoI, S& mxxI, S& myyI,
                                           S& mxyI) {
    S r = 0.0, a = 0.0, b = 0.0, c = 0.0;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        if (!((mask >> k) & 1)) continue;
        r = r + f[k];
        a = a + f[k] * (ex(k) != 0 ? hp : hm);
        b = b + f[k] * (ey(k) != 0 ? hp : hm);
        const int hxy = ex(k) * ey(k);
        if (hxy > 0) c = c + f[k];
        if (hxy < 0) c = c - f[k];
    }
    rhoI = r;
    const S inv = 1.0 / r;
    mxxI = a * inv;
    myyI = b * inv;
    mxyI = c * inv;
}

// Domain-edge node (i, j): moments, Dirichlet values and the apply_bc / apply_bc_incomp closure
// (2d_mrlbm.f90:249-272, 1237-1494): inlet column i = 1, outlet column i = nx (fn: the inputs
// of node (nx - 1, j), whose moments it copies), and with no-slip reference walls rows 1 and
// ny, whose closure wins at the corners.
template <class P, class S>
__device__ __forceinline__ void edge_map(const P& p, int i, int j, const S f[Q], const S fn[Q], S uin, S fo[Q]) {
    const bool outlet = i == p.L.nx, inlet = i == 1;
    const bool top = p.walls_ref && j == p.L.ny, bottom = p.walls_ref && j == 1;
    const double hm = p.hm, hp = p.hp, om = p.omega;
    MacS<S> m = moments_s(f, hm, hp);
    if (outlet) {
        S r = fn[0];
        for (int k = 1; k < Q; ++k) r = r + fn[k];
        const S inv = 1.0 / r;
        m.rho = r;
        m.ux = (((((fn[1] - fn[3]) + fn[5]) - fn[6]) - fn[7]) + fn[8]) * inv;
        m.uy = (((((fn[2] - fn[4]) + fn[5]) + fn[6]) - fn[7]) - fn[8]) * inv;
    }
    if (inlet) {
        m.ux = uin;
        m.uy = S(p.vinlet);
    }
    S rhoI, mxxI, myyI, mxyI;
    if (top || bottom) {
        m.ux = S(0.0);
        m.uy = S(0.0);
        incoming_s(f, top ? fp64::M_TOP : fp64::M_BOTTOM, hm, hp, rhoI, mxxI, myyI, mxyI);
        if (!p.incomp_bc) {
            m.rho = 3.0 * rhoI * (4.0 + 3.0 * (1.0 - om) * myyI) / (9.0 + om);
            const S rp = m.rho;
            m.mxx = 6.0 * rhoI * mxxI / (5.0 * rp);
            m.myy = (rp + 9.0 * rhoI * myyI) / (6.0 * rp);
            m.mxy = 2.0 * rhoI * mxyI / rp;
        } else {
            m.rho = 6.0 * rhoI / 5.0;
            m.mxx = S(0.0);
            m.myy = S(0.0);
            m.mxy = 5.0 * mxyI / 3.0;
        }
    } else if (inlet) {
        incoming_s(f, fp64::M_INLET, hm, hp, rhoI, mxxI, myyI, mxyI);
        if (!p.incomp_bc) {
            m.rho = (4.0 * rhoI + 3.0 * rhoI * mxxI) / (3.0 - 3.0 * m.ux);
            const S rp = m.rho;
            m.mxx = (rp + 9.0 * rhoI * mxxI + 3.0 * rp * m.ux) / (6.0 * rp);
            m.myy = 6.0 * rhoI * myyI / (5.0 * rp);
            m.mxy = 2.0 * rhoI * mxyI / rp;
        } else {
            m.rho = 6.0 * rhoI / ((5.0 - 3.0 * m.ux) - 3.0 * (m.ux * m.ux));
            const S rp = m.rho;
            m.mxx = m.ux * m.ux;
            m.myy = S(0.0);
            m.mxy = 2.0 * rhoI * mxyI / rp;
        }
    } else if (outlet) {
        incoming_s(f, fp64::M_OUTLET, hm, hp, rhoI, mxxI, myyI, mxyI);
        const S rp = m.rho;
        if (!p.incomp_bc) {
            m.mxx = (rp + 9.0 * rhoI * mxxI - 3.0 * rp * m.ux) / (6.0 * rp);
            m.myy = 6.0 * rhoI * myyI / (5.0 * rp);
        } else {
            m.mxx = m.ux * m.ux;
            m.myy = m.uy * m.uy;
        }
        m.mxy = (6.0 * rhoI * mxyI - rp * m.uy) / (3.0 * rp);
    }
    collide_s(p, m, fo);
}

// Edge node e of the adjoint's enumeration: column 1 (j = 1..ny), column nx, then, with
// no-slip reference walls, rows 1 and ny without the corners.
template <class P>
__device__ __forceinline__ void edge_node_ij(const P& p, int e, int& i, int& j) {
    const int nx = p.L.nx, ny = p.L.ny;
    if (e < ny) { i = 1; j = e + 1; }
    else if (e < 2 * ny) { i = nx; j = e - ny + 1; }
    else {
        const int q = e - 2 * ny, nr = nx - 2;
        i = 2 + (q < nr ? q : q - nr);
        j = q < nr ? 1 : ny;
    }
}

template <class P>
__device__ __forceinline__ double gf(const P& p, int field, int l) { return (double)__ldg(p.bgeo + (int64_t)field * p.nb + l); }
template <class P>
__device__ __forceinline__ int gi(const P& p, int field, int l) { return __ldg(p.bint + (int64_t)field * p.nb + l); }

// Rotated velocity and second moments of one bilinear stencil node (2d_mrlbm.f90:842-867).
template <class P, class S>
__device__ __forceinline__ void stencil_quad(const P& p, int l, int s, const S f[Q], S& u, S& v, S& mx, S& my) {
    const MacS<S> m = moments_s(f, p.hm, p.hp);
    const double c2 = gf(p, G_SCC + s, l), s2q = gf(p, G_SSS + s, l), sn2 = gf(p, G_SS2 + s, l);
    u = m.ux;
    v = m.uy;
    mx = m.mxx * c2 + m.myy * s2q + m.mxy * sn2;
    my = m.mxx * s2q + m.myy * c2 - m.mxy * sn2;
}

// Unrotated closure with Cramer's rule (2d_mrlbm.f90:1496-1633, 1974-2003) for a generic
// scalar, as closure_unrotated in step_fp64.cuh.
template <class P, class S>
__device__ __forceinline__ void closure_unrotated_s(const P& p, int l, const S f[Q], S ux, S uy, MacS<S>& m) {
    const int Is = gi(p, I_IS, l), Os = gi(p, I_OS, l);
    const double omega = p.omega, hm = p.hm, hp = p.hp;
    S rhoI = 0.0, mxxI = 0.0, myyI = 0.0, mxyI = 0.0, A_p = 0.0, E_p = 0.0, D_xx = 0.0, D_yy = 0.0, D_xy = 0.0;
    double B11 = 0, B22 = 0, B12 = 0, F11_xx = 0, F12_xx = 0, F22_xx = 0, F11_yy = 0, F12_yy = 0, F22_yy = 0;
    double F11_xy = 0, F12_xy = 0, F22_xy = 0;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const double hxx = ex(k) != 0 ? hp : hm, hyy = ey(k) != 0 ? hp : hm, hxy = (double)(ex(k) * ey(k));
        const double wk = p.w[k];
        const S A_i = wk * (1.0 + 3.0 * ux * (double)ex(k) + 3.0 * uy * (double)ey(k));
        const S E_i = wk * (1.0 + 3.0 * ux * (double)ex(k) + 3.0 * uy * (double)ey(k) + 4.5 * (ux * ux) * hxx +
                            4.5 * (uy * uy) * hyy + 9.0 * (ux * uy) * hxy);
        const double B11_i = 4.5 * wk * hxx, B22_i = 4.5 * wk * hyy, B12_i = 4.5 * wk * hxy;
        if ((Os >> k) & 1) { A_p = A_p + A_i; E_p = E_p + E_i; B11 += B11_i; B22 += B22_i; B12 += B12_i; }
        if ((Is >> k) & 1) {
            rhoI = rhoI + f[k];
            mxxI = mxxI + f[k] * hxx;
            myyI = myyI + f[k] * hyy;
            mxyI = mxyI + f[k] * hxy;
            D_xx = D_xx + A_i * hxx; D_yy = D_yy + A_i * hyy; D_xy = D_xy + A_i * hxy;
            F11_xx += B11_i * hxx; F22_xx += B22_i * hxx; F12_xx += B12_i * hxx;
            F11_yy += B11_i * hyy; F22_yy += B22_i * hyy; F12_yy += B12_i * hyy;
            F11_xy += B11_i * hxy; F22_xy += B22_i * hxy; F12_xy += B12_i * hxy;
        }
    }
    const S inv = 1.0 / rhoI;
    mxxI = mxxI * inv;
    myyI = myyI * inv;
    mxyI = mxyI * inv;
    const S G_p = (1.0 - omega) * A_p + omega * E_p;
    const double J11 = (1.0 - omega) * B11, J22 = (1.0 - omega) * B22, J12 = (1.0 - omega) * B12;
    const S a1 = J11 * mxxI - F11_xx, b1 = J22 * mxxI - F22_xx, c1 = 2.0 * (J12 * mxxI - F12_xx);
    const S a2 = J11 * myyI - F11_yy, b2 = J22 * myyI - F22_yy, c2 = 2.0 * (J12 * myyI - F12_yy);
    const S a3 = J11 * mxyI - F11_xy, b3 = J22 * mxyI - F22_xy, c3 = 2.0 * (J12 * mxyI - F12_xy);
    const S d1 = D_xx - G_p * mxxI, d2 = D_yy - G_p * myyI, d3 = D_xy - G_p * mxyI;
    const S denom = a3 * b2 * c1 - a2 * b3 * c1 - a3 * b1 * c2 + a1 * b3 * c2 + a2 * b1 * c3 - a1 * b2 * c3;
    const S Mxx = -((-b3 * c2 * d1 + b2 * c3 * d1 + b3 * c1 * d2 - b1 * c3 * d2 - b2 * c1 * d3 + b1 * c2 * d3) / denom);
    const S Myy = -((a3 * c2 * d1 - a2 * c3 * d1 - a3 * c1 * d2 + a1 * c3 * d2 + a2 * c1 * d3 - a1 * c2 * d3) / denom);
    const S Mxy = -((-a3 * b2 * d1 + a2 * b3 * d1 + a3 * b1 * d2 - a1 * b3 * d2 - a2 * b1 * d3 + a1 * b2 * d3) / denom);
    const S den = (1.0 - omega) * A_p + (1.0 - omega) * (Mxx * B11 + Myy * B22 + 2.0 * Mxy * B12) + omega * E_p;
    m.rho = rhoI / den;
    m.mxx = Mxx;
    m.myy = Myy;
    m.mxy = Mxy;
}

// Curved-wall node l with the unrotated closure, from its own inputs f and its 8 stencil nodes' (u, v):
// bilinear interpolation at reference points 2 and 3, extrapolation to the node, closure, collision
// (2d_mrlbm.f90:294-311, 768-819, 1496-1633, 407-457) and the node's drag term (2d_mrlbm.f90:558-591).
// The eight stencil nodes' u and v come as plain values (qd[kind][t]); the one stencil node s whose
// inputs carry the derivative (s < 0: none) comes as duals.  Each operand is formed where it is used,
// so no per-thread array of stencil duals exists.
template <class P, class S>
__device__ __forceinline__ void wall_map_unrotated(const P& p, int l, const S f[Q], const double (*qd)[8], int s, S us, S vs,
                                                   S fo[Q], S& drag) {
    auto val = [&](int kind, int t) -> S { return t == s ? (kind == 0 ? us : vs) : S(qd[kind][t]); };
    S u[2], v[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const double xd = gf(p, r == 0 ? G_XD2 : G_XD3, l), yd = gf(p, r == 0 ? G_YD2 : G_YD3, l);
        S row_u[2], row_v[2];
#pragma unroll
        for (int rr = 0; rr < 2; ++rr) {
            const int s0 = 4 * r + 2 * rr;
            row_u[rr] = (1.0 - xd) * val(0, s0) + xd * val(0, s0 + 1);
            row_v[rr] = (1.0 - xd) * val(1, s0) + xd * val(1, s0 + 1);
        }
        u[r] = (1.0 - yd) * row_u[0] + yd * row_u[1];
        v[r] = (1.0 - yd) * row_v[0] + yd * row_v[1];
    }
    const double t2 = gf(p, G_T2, l), t3 = gf(p, G_T3, l);
    MacS<S> m;
    m.ux = t2 * u[0] - t3 * u[1];
    m.uy = t2 * v[0] - t3 * v[1];
    closure_unrotated_s(p, l, f, m.ux, m.uy, m);
    collide_s(p, m, fo);
    const int Is = gi(p, I_IS, l), Os = gi(p, I_OS, l);
    S fxo = 0.0, fxi = 0.0;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        if (ex(k) == 0) continue;
        if ((Os >> k) & 1) fxo = fxo + fo[k] * (double)ex(k);
        if ((Is >> k) & 1) fxi = fxi + f[k] * (double)ex(k);
    }
    drag = fxi - fxo;
}

// ---- kernels ------------------------------------------------------------------------------

// Add c to lambda^{n-1} at the slot node (i, j) pulled for direction k (ghost slots hold
// constants and take nothing).
template <class P>
__device__ __forceinline__ void scatter(const P& p, const AdjArgs& a, int i, int j, int k, double c) {
    const SrcSlot sl = stream_source(p.L.nx, p.L.ny, i, j, k, p.xper, p.yper, p.freeslip);
    if (sl.i < 1 || sl.i > p.L.nx || sl.j < 1 || sl.j > p.L.ny) return;
    atomicAdd(a.lam_out + p.L.at(sl.i, sl.j, sl.k), c);
}

template <class P>
__device__ __forceinline__ void body_grad(const P& p, const AdjArgs& a, int i, int j, const double lam[Q]) {
    if (!a.grad_body) return;
    const int64_t n = (int64_t)(i - 1) + (int64_t)p.L.nx * (j - 1), N = (int64_t)p.L.nx * p.L.ny;
    double gx = 0.0, gy = 0.0;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        gx += 3.0 * p.w[k] * ex(k) * lam[k];
        gy += 3.0 * p.w[k] * ey(k) * lam[k];
    }
    a.grad_body[n] += gx;
    a.grad_body[N + n] += gy;
}

// Bulk node, reverse mode by hand.  Forward: rho = sum g, u = j / rho, m = Pi / rho,
// m' = (1 - w) m + w u u, fo_k = w_k rho A_k with A_k = 1 + 3 c.u + 4.5 m'_xx Hxx
// + 4.5 m'_yy Hyy + 9 m'_xy Hxy.  Every load the node needs (its inputs, lambda^n, the
// body-gradient sums) is issued before the first use, so a node waits for memory once.
template <class P>
__device__ __forceinline__ void adjoint_bulk(const P& p, const AdjArgs& a, int t) {
    const int nx = p.L.nx, ny = p.L.ny;
    if (t >= nx * ny) return;
    const int j = 1 + t / nx, i = t - (j - 1) * nx + 1;
    if (!p.xper && (i == 1 || i == nx)) return;            // edge columns: adjoint_edge
    if (p.walls_ref && (j == 1 || j == ny)) return;        // no-slip wall rows: adjoint_edge
    const int cls = node_class(p, i, j);
    if (cls >= 0) return;                                  // curved-wall node: adjoint_wall
    const int64_t own = p.L.at(i, j, 0), plane = p.L.plane;
    double g[Q], lam[Q];
    gather_d(p, i, j, g);
#pragma unroll
    for (int k = 0; k < Q; ++k) lam[k] = __ldcg(a.lam_in + own + k * plane);
    const int64_t n = (int64_t)(i - 1) + (int64_t)nx * (j - 1), N = (int64_t)nx * ny;
    const bool bg = p.body && a.grad_body;
    double gbx = 0.0, gby = 0.0;
    if (bg) {
        gbx = a.grad_body[n];
        gby = a.grad_body[N + n];
    }
    // the buffer becomes step n-2's target: cleared where some of the nine nodes that pull these slots add to it,
    // left where all of them store (a fifth of the node's traffic)
    const bool keep = i > 2 && i < nx - 2 && j > 2 && j < ny - 1 &&
                      (i < a.sx0 - 1 || i > a.sx1 + 1 || j < a.sy0 - 1 || j > a.sy1 + 1);
    if (!keep) {
#pragma unroll
        for (int k = 0; k < Q; ++k) a.lam_in[own + k * plane] = 0.0;
    }
    const fp64::Mac m = fp64::moments(g, p.hm, p.hp);
    const bool u_zero = cls == CLS_SOLID && p.zero_solid_u;
    const double ux = u_zero ? 0.0 : m.ux, uy = u_zero ? 0.0 : m.uy;
    const double om = p.omega, om1 = p.omega1;
    double mxx = om1 * m.mxx + om * ux * ux, myy = om1 * m.myy + om * uy * uy;
    const double mxy = om1 * m.mxy + om * ux * uy;
    if (p.incomp_bulk) {                                   // m'' = m' - t I, t = (tr m' - |u|^2) / 2
        const double t = 0.5 * (((mxx + myy) - ux * ux) - uy * uy);
        mxx -= t;
        myy -= t;
    }
    double rb = 0.0, uxb = 0.0, uyb = 0.0, mxxb = 0.0, myyb = 0.0, mxyb = 0.0;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const double hxx = ex(k) != 0 ? p.hp : p.hm, hyy = ey(k) != 0 ? p.hp : p.hm, hxy = (double)(ex(k) * ey(k));
        const double A = 1.0 + 3.0 * (ex(k) * ux + ey(k) * uy) + 4.5 * mxx * hxx + 4.5 * myy * hyy + 9.0 * mxy * hxy;
        rb += lam[k] * p.w[k] * A;
        const double Ab = lam[k] * p.w[k] * m.rho;
        uxb += 3.0 * ex(k) * Ab;
        uyb += 3.0 * ey(k) * Ab;
        mxxb += 4.5 * hxx * Ab;
        myyb += 4.5 * hyy * Ab;
        mxyb += 9.0 * hxy * Ab;
    }
    if (p.incomp_bulk) {
        const double tb = -(mxxb + myyb);
        mxxb += 0.5 * tb;
        myyb += 0.5 * tb;
        uxb -= tb * ux;
        uyb -= tb * uy;
    }
    // collision: m' = (1 - w) m + w u u
    uxb += om * (2.0 * ux * mxxb + uy * mxyb);
    uyb += om * (2.0 * uy * myyb + ux * mxyb);
    mxxb *= om1;
    myyb *= om1;
    mxyb *= om1;
    if (u_zero) { uxb = 0.0; uyb = 0.0; }
    const double inv = 1.0 / m.rho;
    double mu[Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const double hxx = ex(k) != 0 ? p.hp : p.hm, hyy = ey(k) != 0 ? p.hp : p.hm, hxy = (double)(ex(k) * ey(k));
        mu[k] = rb + inv * (uxb * (ex(k) - m.ux) + uyb * (ey(k) - m.uy) + mxxb * (hxx - m.mxx) + myyb * (hyy - m.myy) +
                            mxyb * (hxy - m.mxy));
    }
    const bool shared = i == nx - 1 || (i >= a.sx0 && i <= a.sx1 && j >= a.sy0 && j <= a.sy1);
    if (!shared && is_interior(p, i, j)) {
        // the nine source slots are this node's alone: plain stores into the zeroed buffer
        double* d = a.lam_out + own;
#pragma unroll
        for (int k = 0; k < Q; ++k) d[k * plane - ey(k) * (int64_t)p.L.pitch - ex(k)] = mu[k];
    } else {
#pragma unroll
        for (int k = 0; k < Q; ++k) scatter(p, a, i, j, k, mu[k]);
    }
    if (bg) {
        double gx = 0.0, gy = 0.0;
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            gx += 3.0 * p.w[k] * ex(k) * lam[k];
            gy += 3.0 * p.w[k] * ey(k) * lam[k];
        }
        a.grad_body[n] = gbx + gx;
        a.grad_body[N + n] = gby + gy;
    }
}

// Edge block b: 7 nodes of edge_node_ij x 18 threads, thread q of a node for its input q: own inputs
// 0..8; at the outlet the copied neighbour's inputs 9..17; at the inlet q = 9 is u_in(j).  Every load
// (the nodes' lambda^n, staged once and cleared for reuse, and each thread's inputs) is issued before
// the first use: with the staging ahead of the gathers and two divisions per dual quotient these blocks
// were the last of a step to end, 7.4 of its 8.4 us on 512 x 128 (the gradient over 400 steps 9.1 ms;
// with this, and without the clearing of what adjoint_bulk stores outright, 8.1).
template <class P>
__device__ __forceinline__ void adjoint_edge_block(const P& p, const AdjArgs& a, int b) {
    __shared__ double lams[7][Q];
    const int t = threadIdx.x, nx = p.L.nx;
    double* clear = nullptr;
    double lv = 0.0;
    if (t < 7 * Q && 7 * b + t / Q < a.n_edge) {
        int i, j;
        edge_node_ij(p, 7 * b + t / Q, i, j);
        clear = a.lam_in + p.L.at(i, j, t % Q);
        lv = *clear;
    }
    const int e = 7 * b + t / 18, q = t % 18;
    int i = 0, j = 0;
    bool on = t < 7 * 18 && e < a.n_edge;
    if (on) edge_node_ij(p, e, i, j);
    const bool inlet = i == 1, outlet = i == nx;
    on = on && (outlet || q < 9 || (inlet && q == 9));
    double g[Q] = {}, gn[Q] = {}, u0 = 0.0;
    if (on) {
        edge_gather_d(p, i, j, g);
        if (outlet) edge_gather_d(p, nx - 1, j, gn);
        u0 = p.u_in ? (double)p.u_in[j - 1] : (double)p.uinlet;
    }
    if (clear) {
        lams[t / Q][t % Q] = lv;
        *clear = 0.0;
    }
    __syncthreads();
    if (!on) return;
    const double* lam = lams[t / 18];
    Dual f[Q], fn[Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        f[k] = Dual(g[k], q == k ? 1.0 : 0.0);
        fn[k] = Dual(gn[k], (outlet && q == 9 + k) ? 1.0 : 0.0);
    }
    const Dual uin(u0, (inlet && q == 9) ? 1.0 : 0.0);
    Dual fo[Q];
    edge_map(p, i, j, f, fn, uin, fo);
    double c = 0.0;
#pragma unroll
    for (int k = 0; k < Q; ++k) c += lam[k] * fo[k].d;
    if (q < 9) scatter(p, a, i, j, q, c);
    else if (outlet) scatter(p, a, nx - 1, j, q - 9, c);
    else if (a.grad_uin) a.grad_uin[j - 1] += c;
    if (q == 0 && p.body) body_grad(p, a, i, j, lam);
}

// Curved-wall node l with the unrotated closure, one block: the block stages the node's 81 inputs (9 own, 9 for each
// of its 8 stencil nodes) and the stencil quantities in shared memory; thread q < 81 then runs
// the node's map with the derivative along input q (only its stencil node's quantities carry
// a derivative) and scatters the contracted column.
template <class P>
__device__ __forceinline__ void adjoint_wall_unrotated(const P& p, const AdjArgs& a, int l) {
    __shared__ double in[81], lam[Q], qd[4][8];
    __shared__ int slot[81];
    const int q = threadIdx.x;
    const int i = gi(p, I_NODEI, l), j = gi(p, I_NODEJ, l);
    if (q < 81) {
        int ni = i, nj = j, k = q;
        if (q >= 9) {
            const int s = (q - 9) / Q;
            ni = gi(p, I_SI + s, l);
            nj = gi(p, I_SJ + s, l);
            k = (q - 9) % Q;
        }
        const SrcSlot sl = stream_source(p.L.nx, p.L.ny, ni, nj, k, p.xper, p.yper, p.freeslip);
        const int64_t at = p.L.at(sl.i, sl.j, sl.k);
        in[q] = to_f(p, k, __ldg(p.src + at));
        const bool ghost = sl.i < 1 || sl.i > p.L.nx || sl.j < 1 || sl.j > p.L.ny;
        slot[q] = ghost ? -1 : (int)at;
    } else if (q < 81 + Q) {
        const int64_t at = p.L.at(i, j, q - 81);
        lam[q - 81] = a.lam_in[at];
        a.lam_in[at] = 0.0;                      // read once, into shared memory
    }
    __syncthreads();
    if (q < 8) {
        double f[Q], u, v, mx, my;
#pragma unroll
        for (int k = 0; k < Q; ++k) f[k] = in[9 + Q * q + k];
        stencil_quad(p, l, q, f, u, v, mx, my);
        qd[0][q] = u; qd[1][q] = v; qd[2][q] = mx; qd[3][q] = my;
    }
    __syncthreads();
    if (q >= 81) return;
    Dual f[Q];
#pragma unroll
    for (int k = 0; k < Q; ++k) f[k] = Dual(in[k], q == k ? 1.0 : 0.0);
    int s = -1;                                          // the stencil node input q belongs to
    Dual us(0.0), vs(0.0), mxs(0.0), mys(0.0);
    if (q >= 9) {
        s = (q - 9) / Q;
        const int kk = (q - 9) % Q;
        Dual g[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) g[k] = Dual(in[9 + Q * s + k], k == kk ? 1.0 : 0.0);
        stencil_quad(p, l, s, g, us, vs, mxs, mys);    // only stencil s depends on input q
    }
    Dual fo[Q], drag;
    wall_map_unrotated(p, l, f, qd, s, us, vs, fo, drag);
    double c = a.wJ * drag.d;
#pragma unroll
    for (int k = 0; k < Q; ++k) c += lam[k] * fo[k].d;
    if (slot[q] >= 0) atomicAdd(a.lam_out + slot[q], c);
}

// Sum over the 16 lanes of a node, in every lane.
__device__ __forceinline__ double sum16(double v) {
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d, 16);
    return v;
}

// Curved-wall nodes with a rotated closure (strong, weak, rho_eq) or none: reverse mode by hand, 16
// lanes per node as in the forward step's wall blocks (fp64::wall_block, whose quantities it names
// alike).  Lane s (and s + 8) holds stencil node s, lane k < 9 direction k; b after a name is the
// derivative of J by it.  Forward: extrapolated (ux, uy, X, Y) = sum_s kappa_s (stencil quantities),
// closure (rho, Z), moments rotated back, collision, fo_k, drag.  Then the same backwards; the sums
// over the directions are shuffles.  Every table value is loaded before the wait.  With dual numbers a
// block ran the map once for each of the node's 81 inputs: 12 of an adjoint step's 20 us on
// 512 x 128 (the gradient over 400 steps 11.2 ms, with this form 9.4; the sums in another order,
// 5e-15 of the largest entry apart).
template <int CL, class P>
__device__ __forceinline__ void adjoint_wall(const P& p, const AdjArgs& a, int block) {
    const int tid = threadIdx.x, lane = tid & 15, nb = p.nb;
    const int l = block * (int)(blockDim.x >> 4) + (tid >> 4);
    const bool active = l < nb;
    const int lt = active ? l : 0;
    auto G = [&](int field) { return gf(p, field, lt); };
    const int k = min(lane, Q - 1), s = lane & 7, r = s >> 2;
    const bool dir = active && lane < Q;
    const int i = gi(p, I_NODEI, lt), j = gi(p, I_NODEJ, lt), si = gi(p, I_SI + s, lt), sj = gi(p, I_SJ + s, lt);
    const double in = (gi(p, I_IS, lt) >> k) & 1, out = (gi(p, I_OS, lt) >> k) & 1;
    const double scc = G(G_SCC + s), sss = G(G_SSS + s), ss2 = G(G_SS2 + s);
    const double xd = G(r == 0 ? G_XD2 : G_XD3), yd = G(r == 0 ? G_YD2 : G_YD3);
    const double kappa = (r == 0 ? G(G_T2) : -G(G_T3)) * ((s & 1) ? xd : 1.0 - xd) * ((s & 2) ? yd : 1.0 - yd);
    const double c = G(G_CTH), sn = G(G_STH), s2 = G(G_S2TH), c2 = G(G_C2TH), cc = G(G_CC), ss = G(G_SS);
    const double cxp = G(G_CXP + k), cyp = G(G_CYP + k), hxx = G(G_HXXP + k), hyy = G(G_HYYP + k), hxy = G(G_HXYP + k);
    const double exk = ex(k), eyk = ey(k), Hx = exk != 0.0 ? (double)p.hp : (double)p.hm, Hy = eyk != 0.0 ? (double)p.hp : (double)p.hm;
    const double w = lane < Q ? (double)(k == 0 ? p.w[0] : k < 5 ? p.w[1] : p.w[5]) : 0.0;     // lanes past the directions add nothing
    constexpr bool none = CL == CLOSURE_NONE, strong = CL == CLOSURE_STRONG, weak = CL == CLOSURE_WEAK;
    const double om = p.omega, om1 = p.omega1;         // om1: the collision's, an FP32 handle's rounded to FP32
    const double beta = strong ? 1.0 - om : 1.0;       // the closure's
    // The closure's constant sums.  An FP32 handle's table has them rounded to FP32, and L11, L22 and L12 below take
    // them from one another (which put gradients 1e-8 to 5e-8 of the largest entry off): there they are summed from the node's entries,
    // like every other sum of the adjoint in FP64.
    double B11 = 0.0, B22 = 0.0, B12 = 0.0, F11 = 0.0, F22 = 0.0, F12 = 0.0;
    if constexpr (!none) {
        if constexpr (sizeof(typename P::Real) == 8) {
            B11 = G(G_B11); B22 = G(G_B22); B12 = G(G_B12);
            F11 = G(G_F11); F22 = G(G_F22); F12 = G(G_F12);
        } else {
            const double b = 4.5 * w, sum = strong ? out : in;
            B11 = sum16(sum * b * hxx); B22 = sum16(sum * b * hyy); B12 = sum16(sum * b * hxy);
            F11 = sum16(in * b * hxx * hxy); F22 = sum16(in * b * hyy * hxy); F12 = sum16(in * b * hxy * hxy);
        }
    }
    wait_prior_grid();

    const int64_t own = p.L.at(i, j, k), src = p.L.at(i - ex(k), j - ey(k), k);     // wall nodes are interior nodes
    double f = 0.0, lam = 0.0;
    fp64::Mac q{};
    double qs[Q];
#pragma unroll
    for (int t = 0; t < Q; ++t) qs[t] = (double)p.w[t];
    if (active) {
        typename P::Real g[Q];
        gather_interior(p, si, sj, g);
        if (lane < Q) {
            f = to_f(p, k, __ldg(p.src + src));
            lam = a.lam_in[own];
        }
#pragma unroll
        for (int t = 0; t < Q; ++t) qs[t] = to_f(p, t, g[t]);
    }
    if (dir) a.lam_in[own] = 0.0;
    q = fp64::moments(qs, p.hm, p.hp);                                               // stencil node s
    const double xs = q.mxx * scc + q.myy * sss + q.mxy * ss2, ys = q.mxx * sss + q.myy * scc - q.mxy * ss2;
    const double half = lane < 8 ? 1.0 : 0.0;                                          // each stencil node once
    double ux = sum16(half * kappa * q.ux), uy = sum16(half * kappa * q.uy);
    double X = sum16(half * kappa * xs), Y = sum16(half * kappa * ys);
    if (!p.mom_interp) X = Y = 0.0;
    // the node's own moments, where something of them survives
    MacS<double> m0{1.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    double inv0 = 1.0;
    if (none || !p.vel_interp) {
        m0.rho = sum16(f);
        inv0 = 1.0 / m0.rho;
        m0.ux = sum16(f * exk) * inv0;
        m0.uy = sum16(f * eyk) * inv0;
        m0.mxx = sum16(f * Hx) * inv0;
        m0.myy = sum16(f * Hy) * inv0;
        m0.mxy = sum16(f * exk * eyk) * inv0;
    }
    if (!p.vel_interp) { ux = m0.ux; uy = m0.uy; }
    const double up = ux * c + uy * sn, vp = uy * c - ux * sn;
    double rho, mxx, myy, mxy;
    double A_p = 0.0, E_p = 0.0, rhoI = 1.0, mI = 0.0, D = 0.0, Z = 0.0, Pp = 0.0, den = 1.0, L11 = 0.0, L22 = 0.0, L12 = 1.0;
    if constexpr (none) {
        rho = m0.rho; mxx = m0.mxx; myy = m0.myy; mxy = m0.mxy;
    } else {
        const double A = w * (1.0 + 3.0 * up * cxp + 3.0 * vp * cyp);
        const double E = A + w * (4.5 * up * up * hxx + 4.5 * vp * vp * hyy + 9.0 * up * vp * hxy);
        rhoI = sum16(in * f);
        mI = sum16(in * f * hxy) / rhoI;
        D = sum16(in * A * hxy);
        if (strong || weak) A_p = sum16((strong ? out : in) * A);
        if (!weak) E_p = sum16((strong ? out : in) * E);
        if constexpr (strong || weak) {
            Pp = strong ? beta * A_p + om * E_p : A_p;
            L11 = beta * B11 * mI - F11;
            L22 = beta * B22 * mI - F22;
            L12 = 2.0 * (beta * B12 * mI - F12);
            Z = (D - Pp * mI - X * L11 - Y * L22) / L12;
            den = Pp + beta * (X * B11 + Y * B22 + 2.0 * Z * B12);
        } else {
            L11 = F11; L22 = F22; L12 = 2.0 * F12;
            Z = (E_p * mI - D - X * L11 - Y * L22) / L12;
            den = E_p;
        }
        rho = rhoI / den;
        mxx = X * cc + Y * ss - Z * s2;
        myy = X * ss + Y * cc + Z * s2;
        mxy = (X - Y) * 0.5 * s2 + Z * c2;
    }
    // collision and reconstruction of direction k
    double xx = om1 * mxx + om * ux * ux, yy = om1 * myy + om * uy * uy;
    const double xy = om1 * mxy + om * ux * uy;
    if (p.incomp_bulk) {
        const double t = 0.5 * (((xx + yy) - ux * ux) - uy * uy);
        xx -= t;
        yy -= t;
    }
    const double Phi = 1.0 + 3.0 * (exk * ux + eyk * uy) + 4.5 * xx * Hx + 4.5 * yy * Hy + 9.0 * xy * exk * eyk;

    // ---- backwards: fo_k = w rho Phi, drag = sum_in f e_x - sum_out fo e_x
    const double lw = (lam - a.wJ * out * exk) * w, lr = lw * rho;
    double rb = sum16(lw * Phi), uxb = sum16(3.0 * exk * lr), uyb = sum16(3.0 * eyk * lr);
    double xxb = sum16(4.5 * Hx * lr), yyb = sum16(4.5 * Hy * lr);
    const double xyb = sum16(9.0 * exk * eyk * lr);
    if (p.incomp_bulk) {
        const double tb = -(xxb + yyb);
        xxb += 0.5 * tb;
        yyb += 0.5 * tb;
        uxb -= tb * ux;
        uyb -= tb * uy;
    }
    uxb += om * (2.0 * ux * xxb + uy * xyb);
    uyb += om * (2.0 * uy * yyb + ux * xyb);
    const double mxxb = om1 * xxb, myyb = om1 * yyb, mxyb = om1 * xyb;
    double fb = a.wJ * in * exk, Xb = 0.0, Yb = 0.0;
    if constexpr (!none) {
        Xb = mxxb * cc + myyb * ss + 0.5 * mxyb * s2;
        Yb = mxxb * ss + myyb * cc - 0.5 * mxyb * s2;
        double Zb = (myyb - mxxb) * s2 + mxyb * c2;
        double rhoIb = rb / den;
        const double denb = -rb * rho / den;
        double mIb, Db, Ab, Eb;                        // Ab, Eb: by this direction's A and E
        if constexpr (strong || weak) {
            Xb += denb * beta * B11;
            Yb += denb * beta * B22;
            Zb += 2.0 * denb * beta * B12;
            const double t = Zb / L12;
            Xb -= t * L11;
            Yb -= t * L22;
            mIb = -beta * t * (X * B11 + Y * B22 + 2.0 * Z * B12) - t * Pp;
            const double Pb = denb - t * mI;
            Db = t;
            Ab = in * Db * hxy + (strong ? out * beta * Pb : in * Pb);
            Eb = strong ? out * om * Pb : 0.0;
        } else {
            const double t = Zb / L12;
            Xb -= t * L11;
            Yb -= t * L22;
            mIb = t * E_p;
            Db = -t;
            Ab = in * Db * hxy;
            Eb = in * (denb + t * mI);
        }
        rhoIb -= mIb * mI / rhoI;
        fb += in * (rhoIb + mIb / rhoI * hxy);
        const double both = 3.0 * w * (Ab + Eb), e9 = 9.0 * w * Eb;
        const double upb = sum16(both * cxp + e9 * (up * hxx + vp * hxy)), vpb = sum16(both * cyp + e9 * (vp * hyy + up * hxy));
        uxb += upb * c - vpb * sn;
        uyb += upb * sn + vpb * c;
    }
    if (none || !p.vel_interp) {                       // through the node's own moments
        double t = 0.0;
        if (none) t += rb + inv0 * (mxxb * (Hx - m0.mxx) + myyb * (Hy - m0.myy) + mxyb * (exk * eyk - m0.mxy));
        if (!p.vel_interp) t += inv0 * (uxb * (exk - m0.ux) + uyb * (eyk - m0.uy));
        fb += t;
    }
    if (dir) atomicAdd(a.lam_out + src, fb);
    // through the stencil nodes
    const double kv = p.vel_interp ? kappa : 0.0, km = !none && p.mom_interp ? kappa : 0.0;
    if (active && lane < 8 && (kv != 0.0 || km != 0.0)) {
        const double inv = 1.0 / q.rho, ub = kv * uxb * inv, vb = kv * uyb * inv;
        const double ax = km * (Xb * scc + Yb * sss) * inv, ay = km * (Xb * sss + Yb * scc) * inv, axy = km * (Xb - Yb) * ss2 * inv;
        double* d = a.lam_out + p.L.at(si, sj, 0);
#pragma unroll
        for (int t = 0; t < Q; ++t) {
            const double hx = ex(t) != 0 ? (double)p.hp : (double)p.hm, hy = ey(t) != 0 ? (double)p.hp : (double)p.hm;
            atomicAdd(d + t * p.L.plane - ey(t) * (int64_t)p.L.pitch - ex(t),
                      ub * (ex(t) - q.ux) + vb * (ey(t) - q.uy) + ax * (hx - q.mxx) + ay * (hy - q.myy) + axy * (ex(t) * ey(t) - q.mxy));
        }
    }
}

// Wall blocks of 128 threads: a node each with the unrotated closure, eight nodes otherwise.
__host__ __device__ inline int adjoint_wall_blocks(int closure, int nb) {
    return closure == CLOSURE_UNROTATED ? nb : (nb + 7) / 8;
}

// One adjoint step as two launches, ordered like the forward step's (step_common.cuh): the
// wall and edge blocks [nb wall blocks][edge blocks, 7 nodes x 18 inputs each], whose dual-number
// maps get the registers they need, then the bulk blocks (128 nodes each), which start once the
// first launch has waited for the previous step and run beside it; the last bulk block to finish
// waits for the first launch, so the step completes as a whole.
template <class P, int CL>
__global__ void __launch_bounds__(128, 3) adjoint_aux(const __grid_constant__ P p, const __grid_constant__ AdjArgs a) {
    const int b = (int)blockIdx.x, nw = adjoint_wall_blocks(CL, p.nb);
    if (b < nw) {
        if constexpr (CL == CLOSURE_UNROTATED) {
            wait_prior_grid();
            adjoint_wall_unrotated(p, a, b);
        } else {
            adjoint_wall<CL>(p, a, b);
        }
        return;
    }
    wait_prior_grid();
    adjoint_edge_block(p, a, b - nw);
}

template <class P>
__global__ void __launch_bounds__(128, 4) adjoint_bulk_step(const __grid_constant__ P p, const __grid_constant__ AdjArgs a) {
    bulk_begin();
    adjoint_bulk(p, a, (int)blockIdx.x * 128 + (int)threadIdx.x);
    if (threadIdx.x == 0 && atomicAdd(a.done, 1u) == gridDim.x - 1) {
        *a.done = 0u;
        asm volatile("griddepcontrol.wait;" ::: "memory");
    }
}

}  // namespace adj
}  // namespace mrlbm
