// step_fp64.cuh -- FP64 fused time step, arithmetic in the reference's exact order.
//
// One launch advances one time step of 2d_mrlbm.f90:231-535.  State between launches is
// the post-collision population field fout (plus a ghost ring for populations the
// reference never overwrites).  Three kinds of work make a step up:
//   * wall blocks: 16 lanes per curved-wall node (wall_block).  They pull the node's populations and
//     those of its 8 bilinear-stencil nodes from the previous fout, recompute the stencil moments,
//     extrapolate velocity and rotated moments, run the regularized closure, collide, store, and leave
//     the momentum-exchange force of the node for the step's record;
//   * edge blocks: one thread per domain-edge node, Dirichlet values and regularized edge closures;
//   * bulk tiles: pull-stream, moments, moment-space collision, Hermite reconstruction, coalesced
//     store.  Wall and edge nodes are skipped; solid nodes are ordinary nodes, as in the reference.
// Every expression follows the reference's operation order (sums from k = 0 upwards,
// products left to right); the translation unit is compiled with -fmad=false, so each
// node's result is bit-identical to the reference's FP64 arithmetic.
#pragma once
#include <cuda_runtime.h>
#include "step_common.cuh"

namespace mrlbm {
namespace fp64 {

using P = StepParams<double>;

struct Mac { double rho, ux, uy, mxx, myy, mxy; };

// Macroscopic variables, 2d_mrlbm.f90:235-242.
__device__ __forceinline__ Mac moments(const double f[Q], double hm, double hp) {
    Mac m;
    double s = f[0];
    s = s + f[1]; s = s + f[2]; s = s + f[3]; s = s + f[4];
    s = s + f[5]; s = s + f[6]; s = s + f[7]; s = s + f[8];
    m.rho = s;
    const double inv_rho = 1.0 / s;
    const double sx = ((((f[1] - f[3]) + f[5]) - f[6]) - f[7]) + f[8];
    const double sy = ((((f[2] - f[4]) + f[5]) + f[6]) - f[7]) - f[8];
    double sxx = f[0] * hm;
    sxx = sxx + f[1] * hp; sxx = sxx + f[2] * hm; sxx = sxx + f[3] * hp; sxx = sxx + f[4] * hm;
    sxx = sxx + f[5] * hp; sxx = sxx + f[6] * hp; sxx = sxx + f[7] * hp; sxx = sxx + f[8] * hp;
    double syy = f[0] * hm;
    syy = syy + f[1] * hm; syy = syy + f[2] * hp; syy = syy + f[3] * hm; syy = syy + f[4] * hp;
    syy = syy + f[5] * hp; syy = syy + f[6] * hp; syy = syy + f[7] * hp; syy = syy + f[8] * hp;
    const double sxy = ((f[5] - f[6]) + f[7]) - f[8];
    m.ux = sx * inv_rho;
    m.uy = sy * inv_rho;
    m.mxx = sxx * inv_rho;
    m.myy = syy * inv_rho;
    m.mxy = sxy * inv_rho;
    return m;
}

// rho, ux, uy only (outlet copy source and stencil velocities).
__device__ __forceinline__ void moments_u(const double f[Q], double& rho, double& ux, double& uy) {
    double s = f[0];
    s = s + f[1]; s = s + f[2]; s = s + f[3]; s = s + f[4];
    s = s + f[5]; s = s + f[6]; s = s + f[7]; s = s + f[8];
    rho = s;
    const double inv_rho = 1.0 / s;
    ux = (((((f[1] - f[3]) + f[5]) - f[6]) - f[7]) + f[8]) * inv_rho;
    uy = (((((f[2] - f[4]) + f[5]) + f[6]) - f[7]) - f[8]) * inv_rho;
}

// Hxx_k and Hyy_k as values hm / hp.
__device__ __forceinline__ double hxx_of(int k, double hm, double hp) { return ex(k) != 0 ? hp : hm; }
__device__ __forceinline__ double hyy_of(int k, double hm, double hp) { return ey(k) != 0 ? hp : hm; }

// Sums over a fixed incoming mask, normalised by rho_I (prologue of apply_bc,
// 2d_mrlbm.f90:1249-1269).
template <int MASK>
__device__ __forceinline__ void incoming(const double f[Q], double hm, double hp, double& rhoI, double& mxxI,
                                         double& myyI, double& mxyI) {
    bool first = true;
    double r = 0.0, a = 0.0, b = 0.0, c = 0.0;
    bool cfirst = true;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        if (!((MASK >> k) & 1)) continue;
        if (first) {
            r = f[k];
            a = f[k] * hxx_of(k, hm, hp);
            b = f[k] * hyy_of(k, hm, hp);
            first = false;
        } else {
            r = r + f[k];
            a = a + f[k] * hxx_of(k, hm, hp);
            b = b + f[k] * hyy_of(k, hm, hp);
        }
        const int hxy = ex(k) * ey(k);
        if (hxy != 0) {
            if (cfirst) { c = hxy > 0 ? f[k] : -f[k]; cfirst = false; }
            else c = hxy > 0 ? c + f[k] : c - f[k];
        }
    }
    rhoI = r;
    const double inv = 1.0 / rhoI;
    mxxI = a * inv;
    myyI = b * inv;
    mxyI = c * inv;
}

// Masks (bit k = population k) of apply_bc's Is vectors (2d_mrlbm.f90:1254, 1283, 1311, 1339).
constexpr int M_OUTLET = (1 << 0) | (1 << 1) | (1 << 2) | (1 << 4) | (1 << 5) | (1 << 8);
constexpr int M_INLET = (1 << 0) | (1 << 2) | (1 << 3) | (1 << 4) | (1 << 6) | (1 << 7);
constexpr int M_TOP = (1 << 0) | (1 << 1) | (1 << 2) | (1 << 3) | (1 << 5) | (1 << 6);
constexpr int M_BOTTOM = (1 << 0) | (1 << 1) | (1 << 3) | (1 << 4) | (1 << 7) | (1 << 8);

// Edge nodes (fn: the populations of node (nx - 1, j) at the outlet, whose moments it copies): Dirichlet
// values (2d_mrlbm.f90:249-272) then the regularized closure the
// reference applies last at this node (apply_bc / apply_bc_incomp, 2d_mrlbm.f90:313-351).
__device__ __forceinline__ void edge_node(const P& p, int i, int j, const double f[Q], const double fn[Q], Mac& m) {
    const int nx = p.L.nx, ny = p.L.ny;
    const bool outlet = !p.xper && !p.halo_r && i == nx;
    const bool inlet = !p.xper && !p.halo_l && i == 1;
    const bool top = p.walls_ref && j == ny;
    const bool bottom = p.walls_ref && j == 1;
    if (outlet) moments_u(fn, m.rho, m.ux, m.uy);
    if (inlet) {
        m.ux = p.u_in ? p.u_in[j - 1] : p.uinlet;
        m.uy = p.vinlet;
    }
    if (top || bottom) { m.ux = 0.0; m.uy = 0.0; }
    const double hm = p.hm, hp = p.hp, omega = p.omega;
    double rhoI, mxxI, myyI, mxyI;
    if (top || bottom) {
        if (top) incoming<M_TOP>(f, hm, hp, rhoI, mxxI, myyI, mxyI);
        else incoming<M_BOTTOM>(f, hm, hp, rhoI, mxxI, myyI, mxyI);
        if (!p.incomp_bc) {
            m.rho = 3.0 * rhoI * (4.0 + 3.0 * (1.0 - omega) * myyI) / (9.0 + omega);
            const double rp = m.rho;
            m.mxx = 6.0 * rhoI * mxxI / (5.0 * rp);
            m.myy = (rp + 9.0 * rhoI * myyI) / (6.0 * rp);
            m.mxy = 2.0 * rhoI * mxyI / rp;
        } else {
            m.rho = 6.0 * rhoI / 5.0;
            m.mxx = 0.0;
            m.myy = 0.0;
            m.mxy = 5.0 * mxyI / 3.0;
        }
    } else if (inlet) {
        incoming<M_INLET>(f, hm, hp, rhoI, mxxI, myyI, mxyI);
        if (!p.incomp_bc) {
            m.rho = (4.0 * rhoI + 3.0 * rhoI * mxxI) / (3.0 - 3.0 * m.ux);
            const double rp = m.rho;
            m.mxx = (rp + 9.0 * rhoI * mxxI + 3.0 * rp * m.ux) / (6.0 * rp);
            m.myy = 6.0 * rhoI * myyI / (5.0 * rp);
            m.mxy = 2.0 * rhoI * mxyI / rp;
        } else {
            m.rho = 6.0 * rhoI / (5.0 - 3.0 * m.ux - 3.0 * (m.ux * m.ux));
            const double rp = m.rho;
            m.mxx = m.ux * m.ux;
            m.myy = 0.0;
            m.mxy = 2.0 * rhoI * mxyI / rp;
        }
    } else if (outlet) {
        incoming<M_OUTLET>(f, hm, hp, rhoI, mxxI, myyI, mxyI);
        const double rp = m.rho;
        if (!p.incomp_bc) {
            m.mxx = (rp + 9.0 * rhoI * mxxI - 3.0 * rp * m.ux) / (6.0 * rp);
            m.myy = 6.0 * rhoI * myyI / (5.0 * rp);
            m.mxy = (6.0 * rhoI * mxyI - rp * m.uy) / (3.0 * rp);
        } else {
            m.mxx = m.ux * m.ux;
            m.myy = m.uy * m.uy;
            m.mxy = (6.0 * rhoI * mxyI - rp * m.uy) / (3.0 * rp);
        }
    }
}

// Moment-space collision (2d_mrlbm.f90:407-415, 419-428) and Hermite reconstruction
// (2d_mrlbm.f90:445-457), per direction in the reference's left-to-right order.
__device__ __forceinline__ void collide(const P& p, const Mac& m, double fo[Q]) {
    const double om = p.omega, om1 = p.omega1;
    double mxx = om1 * m.mxx + om * m.ux * m.ux;
    double myy = om1 * m.myy + om * m.uy * m.uy;
    double mxy = om1 * m.mxy + om * m.ux * m.uy;
    if (p.incomp_bulk) {
        const double t = 0.50 * (mxx + myy - m.ux * m.ux - m.uy * m.uy);
        mxx = mxx - t;
        myy = myy - t;
    }
    const double a = 4.50 * mxx, b = 4.50 * myy, c = 9.00 * mxy;
    const double am = a * p.hm, ap = a * p.hp, bm = b * p.hm, bp = b * p.hp;
    const double t1 = 3.0 * m.ux, t2 = 3.0 * m.uy;
    const double t5 = 3.0 * (m.ux + m.uy), t8 = 3.0 * (m.ux - m.uy);
    const double w0 = p.w[0] * m.rho, w1 = p.w[1] * m.rho, w5 = p.w[5] * m.rho;
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

// Post-boundary-condition macroscopic values of a non-cylinder node.
__device__ __forceinline__ Mac node_macro(const P& p, int i, int j, const double f[Q]) {
    Mac m = moments(f, p.hm, p.hp);
    if (!is_interior(p, i, j)) {
        double fn[Q];
        edge_gather(p, max(i - 1, 1), j, fn);           // the outlet's neighbour
        edge_node(p, i, j, f, fn, m);
    }
    return m;
}

// ---------------------------------------------------------------------------------------
// Curved-wall boundary node (2d_mrlbm.f90:294-311 and the routines they call).

// Velocity and rotated second moments (2d_mrlbm.f90:842-867) of one bilinear stencil node.
__device__ __forceinline__ void stencil_node(const P& p, int si, int sj, double cc, double ss, double s2, double& ux,
                                             double& uy, double& mx, double& my) {
    double f[Q];
    gather_written(p, si, sj, f);                   // stencil nodes are interior fluid nodes (checked at setup)
    const Mac m = moments(f, p.hm, p.hp);
    ux = m.ux;
    uy = m.uy;
    mx = m.mxx * cc + m.myy * ss + m.mxy * s2;
    my = m.mxx * ss + m.myy * cc - m.mxy * s2;
}

// Unrotated closure with Cramer's rule, 2d_mrlbm.f90:1496-1633 and 1974-2003.
static __device__ __noinline__ void closure_unrotated(const P& p, const BTab<double>& tb, int li, const double f[Q], double uxp,
                                                      double uyp, Mac& m) {
    const int Is = tb.gi(I_IS, li), Os = tb.gi(I_OS, li);
    const double omega = p.omega, hm = p.hm, hp = p.hp;
    double rhoI = 0, mxxI = 0, myyI = 0, mxyI = 0, A_p = 0, E_p = 0, B11 = 0, B22 = 0, B12 = 0;
    double D_xx = 0, D_yy = 0, D_xy = 0, F11_xx = 0, F12_xx = 0, F22_xx = 0, F11_yy = 0, F12_yy = 0, F22_yy = 0;
    double F11_xy = 0, F12_xy = 0, F22_xy = 0;
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const double hxx = hxx_of(k, hm, hp), hyy = hyy_of(k, hm, hp), hxy = (double)(ex(k) * ey(k));
        const double wk = p.w[k];
        const double A_i = wk * (1.0 + 3.0 * uxp * (double)ex(k) + 3.0 * uyp * (double)ey(k));
        const double E_i = wk * (1.0 + 3.0 * uxp * (double)ex(k) + 3.0 * uyp * (double)ey(k) + 4.50 * (uxp * uxp) * hxx +
                                 4.50 * (uyp * uyp) * hyy + 9.0 * (uxp * uyp) * hxy);
        const double B11_i = 4.50 * wk * hxx, B22_i = 4.50 * wk * hyy, B12_i = 4.50 * wk * hxy;
        if ((Os >> k) & 1) { A_p = A_p + A_i; E_p = E_p + E_i; B11 = B11 + B11_i; B22 = B22 + B22_i; B12 = B12 + B12_i; }
        if ((Is >> k) & 1) {
            rhoI = rhoI + f[k];
            mxxI = mxxI + f[k] * hxx;
            myyI = myyI + f[k] * hyy;
            mxyI = mxyI + f[k] * hxy;
            D_xx = D_xx + A_i * hxx; D_yy = D_yy + A_i * hyy; D_xy = D_xy + A_i * hxy;
            F11_xx = F11_xx + B11_i * hxx; F22_xx = F22_xx + B22_i * hxx; F12_xx = F12_xx + B12_i * hxx;
            F11_yy = F11_yy + B11_i * hyy; F22_yy = F22_yy + B22_i * hyy; F12_yy = F12_yy + B12_i * hyy;
            F11_xy = F11_xy + B11_i * hxy; F22_xy = F22_xy + B22_i * hxy; F12_xy = F12_xy + B12_i * hxy;
        }
    }
    const double inv = 1.0 / rhoI;
    mxxI = mxxI * inv;
    myyI = myyI * inv;
    mxyI = mxyI * inv;
    const double G_p = (1.0 - omega) * A_p + omega * E_p;
    const double J11 = (1.0 - omega) * B11, J22 = (1.0 - omega) * B22, J12 = (1.0 - omega) * B12;
    const double a1 = J11 * mxxI - F11_xx, b1 = J22 * mxxI - F22_xx, c1 = 2.0 * (J12 * mxxI - F12_xx);
    const double a2 = J11 * myyI - F11_yy, b2 = J22 * myyI - F22_yy, c2 = 2.0 * (J12 * myyI - F12_yy);
    const double a3 = J11 * mxyI - F11_xy, b3 = J22 * mxyI - F22_xy, c3 = 2.0 * (J12 * mxyI - F12_xy);
    const double d1 = D_xx - G_p * mxxI, d2 = D_yy - G_p * myyI, d3 = D_xy - G_p * mxyI;
    const double denom = a3 * b2 * c1 - a2 * b3 * c1 - a3 * b1 * c2 + a1 * b3 * c2 + a2 * b1 * c3 - a1 * b2 * c3;
    const double Mxx = -((-b3 * c2 * d1 + b2 * c3 * d1 + b3 * c1 * d2 - b1 * c3 * d2 - b2 * c1 * d3 + b1 * c2 * d3) / denom);
    const double Myy = -((a3 * c2 * d1 - a2 * c3 * d1 - a3 * c1 * d2 + a1 * c3 * d2 + a2 * c1 * d3 - a1 * c2 * d3) / denom);
    const double Mxy = -((-a3 * b2 * d1 + a2 * b3 * d1 + a3 * b1 * d2 - a1 * b3 * d2 - a2 * b1 * d3 + a1 * b2 * d3) / denom);
    const double den = (1.0 - omega) * A_p + (1.0 - omega) * (Mxx * B11 + Myy * B22 + 2.0 * Mxy * B12) + omega * E_p;
    m.rho = rhoI / den;
    m.mxx = Mxx;
    m.myy = Myy;
    m.mxy = Mxy;
}

// One direction's constants: velocity components, H_xx and H_yy values, weight.
struct Dir { double x, y, hx, hy, w; };

// Collision and reconstruction of one direction: collide's expressions with this direction's signs
// (3 (x u + y v) is its +-t1 .. +-t8, x y its +-c; products with 0 and +-1 are exact, and adding a zero
// where a direction has no such term changes no bit).  No branch depends on the direction: with the
// nine cases spelled out the lanes of a node took them one after another (1900 cycles of 6400).
__device__ __forceinline__ double collide_dir(const P& p, const Mac& m, const Dir& e) {
    const double om = p.omega, om1 = p.omega1;
    double mxx = om1 * m.mxx + om * m.ux * m.ux;
    double myy = om1 * m.myy + om * m.uy * m.uy;
    const double mxy = om1 * m.mxy + om * m.ux * m.uy;
    if (p.incomp_bulk) {
        const double t = 0.50 * (mxx + myy - m.ux * m.ux - m.uy * m.uy);
        mxx = mxx - t;
        myy = myy - t;
    }
    const double a = 4.50 * mxx, b = 4.50 * myy, c = 9.00 * mxy;
    const double t = 3.0 * (e.x * m.ux + e.y * m.uy);
    return (e.w * m.rho) * ((((1.0 + t) + a * e.hx) + b * e.hy) + (e.x * e.y) * c);
}

// Wall block: curved-wall nodes (2d_mrlbm.f90:294-311 and the routines it calls) by 16 lanes each.  Lane s
// (and s + 8, the same) pulls stencil node s; the bilinear interpolation is completed by shuffles in the
// reference's order; then lane k < 9 carries direction k: its population, its terms of the closure's
// sums, its outgoing population and its part of the force.  The sums of nine run over the directions in
// order, one lane per sum, from terms staged in shared memory; what a rotated closure sums over the
// geometry alone comes from the table.  Every table value is loaded before the wait for the previous
// step.  Compared with one lane running a node's closure after the shuffles this is a fifth of the
// instructions on the critical path of every step that is not bound by the bulk: a 400 x 100 wall
// block took 6.5 us of a 7.1 us step.
template <bool FULL, bool WAIT>
__device__ __forceinline__ void wall_block(const P& p, unsigned char* smem, int bb) {
    const int tid = threadIdx.x, lane = tid & 15, li = tid >> 4, per = (int)(blockDim.x >> 4);
    const int l = bb * per + li, nb = p.nb;
    const bool active = l < nb;
    const int lt = active ? l : 0;
    auto G = [&](int field) { return p.bgeo[field * nb + lt]; };
    auto I = [&](int field) { return p.bint[field * nb + lt]; };
    const int k = min(lane, Q - 1), s = lane & 7, r = s >> 2;      // direction; stencil node, reference point 2 + r
    const bool dir = lane < Q;
    const int ekx = ex(k), eky = ey(k);
    const Dir e{(double)ekx, (double)eky, ekx != 0 ? p.hp : p.hm, eky != 0 ? p.hp : p.hm, k == 0 ? p.w[0] : k < 5 ? p.w[1] : p.w[5]};
    const int closure = p.closure;
    const bool rotated = closure != CLOSURE_UNROTATED;
    const bool interp = !rotated || p.vel_interp || p.mom_interp;
    const int ni = I(I_NODEI), nj = I(I_NODEJ);
    const bool in = (I(I_IS) >> k) & 1, out = (I(I_OS) >> k) & 1;
    const int si = I(I_SI + s), sj = I(I_SJ + s);
    const double cc = G(G_SCC + s), ss = G(G_SSS + s), s2 = G(G_SS2 + s);
    const double xd = G(r == 0 ? G_XD2 : G_XD3), yd = G(r == 0 ? G_YD2 : G_YD3);
    const double t1 = G(G_T1), t2 = G(G_T2), t3 = G(G_T3);
    const double cth = G(G_CTH), sth = G(G_STH), s2th = G(G_S2TH), c2th = G(G_C2TH), ccth = G(G_CC), ssth = G(G_SS);
    const double cxp = G(G_CXP + k), cyp = G(G_CYP + k), hxx = G(G_HXXP + k), hyy = G(G_HYYP + k), hxy = G(G_HXYP + k);
    const double B11 = G(G_B11), B22 = G(G_B22), B12 = G(G_B12), F11 = G(G_F11), F22 = G(G_F22), F12 = G(G_F12);
    const StepRec sr = step_rec(p);
    if (WAIT) wait_prior_grid();

    const unsigned all = 0xffffffffu;
    // the node's population of direction k (a wall node is an interior node)
    double fk = 0.0, ux = 0.0, uy = 0.0, mx = 0.0, my = 0.0;
    if (active) {
        fk = load_written(p.src + ((int64_t)k * p.L.plane + (int64_t)(nj - eky) * p.L.pitch + (ni - ekx) + p.L.off));
        if (interp) {
            stencil_node(p, si, sj, cc, ss, s2, ux, uy, mx, my);
            const double wx = (s & 1) ? xd : (1.0 - xd);
            ux = wx * ux; uy = wx * uy; mx = wx * mx; my = wx * my;
        }
    }
    // row sums (corner pairs 0+1, 2+3), then (1-yd)*a0 + yd*a1 at corners 0 (point 2) and 4 (point 3)
    auto bilinear = [&](double v) {
        v = v + __shfl_down_sync(all, v, 1, 8);
        const double v1 = __shfl_down_sync(all, v, 2, 8);
        return (1.0 - yd) * v + yd * v1;
    };
    ux = bilinear(ux); uy = bilinear(uy); mx = bilinear(mx); my = bilinear(my);
    // extrapolation to the node, wall value 0 (2d_mrlbm.f90:809-814, 919-924)
    auto extrapolate = [&](double v) {
        const double v2 = __shfl_sync(all, v, 0, 8), v3 = __shfl_sync(all, v, 4, 8);
        return t1 * 0.0 + t2 * v2 - t3 * v3;
    };
    double* sm = reinterpret_cast<double*>(smem) + li * WALL_TERMS * Q;          // [term][direction]
    double f[Q];
    Mac m{};
    if (closure == CLOSURE_NONE || !rotated || !p.vel_interp) {                  // the node's own moments
        if (dir) sm[k] = fk;
        __syncwarp();
#pragma unroll
        for (int q = 0; q < Q; ++q) f[q] = sm[q];
        __syncwarp();
        m = moments(f, p.hm, p.hp);
    }
    const double xu = extrapolate(ux), xv = extrapolate(uy), Xx = extrapolate(mx), Xy = extrapolate(my);
    if (!rotated || p.vel_interp) { m.ux = xu; m.uy = xv; }
    const double Mxx = rotated && p.mom_interp ? Xx : 0.0, Myy = rotated && p.mom_interp ? Xy : 0.0;
    if (!rotated) {
        const BTab<double> tb{p.bgeo, p.bint, nb};
        if (active && lane == 0) closure_unrotated(p, tb, l, f, m.ux, m.uy, m);
        m.rho = __shfl_sync(all, m.rho, 0, 16);
        m.mxx = __shfl_sync(all, m.mxx, 0, 16);
        m.myy = __shfl_sync(all, m.myy, 0, 16);
        m.mxy = __shfl_sync(all, m.mxy, 0, 16);
    } else if (closure != CLOSURE_NONE) {
        // numerical_boundary_cases_rotation (strong, 2d_mrlbm.f90:1635-1765), _weak (1767-1871), _rhoeq (1873-1972)
        const double uxp = m.ux * cth + m.uy * sth;                              // 2d_mrlbm.f90:304-305
        const double uyp = m.uy * cth - m.ux * sth;
        const double omega = p.omega, wk = e.w;
        const double A_i = wk * (1.0 + 3.0 * uxp * cxp + 3.0 * uyp * cyp);
        const double E_i = wk * (1.0 + 3.0 * uxp * cxp + 3.0 * uyp * cyp + 4.50 * (uxp * uxp) * hxx +
                                 4.50 * (uyp * uyp) * hyy + 9.0 * (uxp * uyp) * hxy);
        const bool strong = closure == CLOSURE_STRONG;
        if (dir) {
            sm[k] = (strong ? out : in) ? A_i : 0.0;
            sm[Q + k] = (strong ? out : in) ? E_i : 0.0;
            sm[2 * Q + k] = in ? fk : 0.0;
            sm[3 * Q + k] = in ? fk * hxy : 0.0;
            sm[4 * Q + k] = in ? A_i * hxy : 0.0;
        }
        __syncwarp();
        double sum = 0.0;
        const double* row = sm + min(lane, 4) * Q;
#pragma unroll
        for (int q = 0; q < Q; ++q) sum = sum + row[q];
        const double A_p = __shfl_sync(all, sum, 0, 16), E_p = __shfl_sync(all, sum, 1, 16), rhoI = __shfl_sync(all, sum, 2, 16);
        double mxyI = __shfl_sync(all, sum, 3, 16);
        const double D_xy = __shfl_sync(all, sum, 4, 16);
        const double inv = 1.0 / rhoI;
        mxyI = mxyI * inv;
        double Mxy, rhop;
        if (strong) {
            const double G_p = (1.0 - omega) * A_p + omega * E_p;
            const double J11 = (1.0 - omega) * B11, J22 = (1.0 - omega) * B22, J12 = (1.0 - omega) * B12;
            const double L11 = J11 * mxyI - F11, L22 = J22 * mxyI - F22, L12 = 2.0 * (J12 * mxyI - F12);
            const double R = D_xy - G_p * mxyI;
            Mxy = (R - Mxx * L11 - Myy * L22) / L12;
            const double den = (1.0 - omega) * A_p + (1.0 - omega) * (Mxx * B11 + Myy * B22 + 2.0 * Mxy * B12) + omega * E_p;
            rhop = rhoI / den;
        } else if (closure == CLOSURE_WEAK) {
            const double L11 = B11 * mxyI - F11, L22 = B22 * mxyI - F22, L12 = 2.0 * (B12 * mxyI - F12);
            const double R = D_xy - A_p * mxyI;
            Mxy = (R - Mxx * L11 - Myy * L22) / L12;
            const double den = A_p + (Mxx * B11 + Myy * B22 + 2.0 * Mxy * B12);
            rhop = rhoI / den;
        } else {  // CLOSURE_RHOEQ
            const double L11 = F11, L22 = F22, L12 = 2.0 * F12;
            const double R = E_p * mxyI - D_xy;
            Mxy = (R - Mxx * L11 - Myy * L22) / L12;
            rhop = rhoI / E_p;
        }
        m.rho = rhop;
        m.mxx = Mxx * ccth + Myy * ssth - Mxy * s2th;
        m.myy = Mxx * ssth + Myy * ccth + Mxy * s2th;
        m.mxy = (Mxx - Myy) * 0.50 * s2th + Mxy * c2th;
    }
    const double fo = collide_dir(p, m, e);
    if (active && dir) p.dst[(int64_t)k * p.L.plane + (int64_t)nj * p.L.pitch + ni + p.L.off] = fo;
    // momentum-exchange force (evaluate_forces, 2d_mrlbm.f90:558-591): lanes 0 and 1 sum the outgoing
    // populations' x and y, lanes 2 and 3 the incoming ones'
    __syncwarp();
    if (dir) {
        sm[k] = out ? fo * e.x : 0.0;
        sm[Q + k] = out ? fo * e.y : 0.0;
        sm[2 * Q + k] = in ? fk * e.x : 0.0;
        sm[3 * Q + k] = in ? fk * e.y : 0.0;
    }
    __syncwarp();
    double sum = 0.0;
    const double* row = sm + (lane & 3) * Q;
#pragma unroll
    for (int q = 0; q < Q; ++q) sum = sum + row[q];
    const double F = __shfl_down_sync(all, sum, 2, 16) - sum;
    if (active && lane < 2) {
        if (sr.do_stats) p.partials[lane * nb + l] = F;
        if (p.node_force) p.node_force[2 * l + lane] = F;
    }
    if (active && lane == 0) {
        if (!(m.rho > 0.0)) flag_bad_density(p);
        if (FULL && p.macro) store_macro(p, ni, nj, m.rho, m.ux, m.uy, m.mxx, m.myy, m.mxy);
        if (FULL && p.fstat) accumulate_fields(p, ni, nj, m.rho, m.ux, m.uy);
    }
}

// Edge nodes (first/last row or column): own gather, Dirichlet values and closures.  Inline,
// so the populations stay in registers and the gathers of a node overlap (edge blocks are a
// branch of their own, so the bulk path's registers are not affected).
template <bool FULL>
__device__ __forceinline__ double edge_bulk_node(const P& p, int i, int j, int cls) {
    double f[Q], fn[Q];
    edge_gather(p, i, j, f);
    if (i == p.L.nx && !p.halo_r) edge_gather(p, i - 1, j, fn);       // the outlet's neighbour, in the same round trip
    Mac m = moments(f, p.hm, p.hp);
    edge_node(p, i, j, f, fn, m);
    if ((cls == CLS_SOLID && p.zero_solid_u) || cls == CLS_SOLID_ZERO) { m.ux = 0.0; m.uy = 0.0; }
    if (!(m.rho > 0.0)) flag_bad_density(p);
    if (FULL && p.macro) store_macro(p, i, j, m.rho, m.ux, m.uy, m.mxx, m.myy, m.mxy);
    if (FULL && p.fstat) accumulate_fields(p, i, j, m.rho, m.ux, m.uy);
    double fo[Q];
    collide(p, m, fo);
    if (FULL && p.body) add_body_force(p, i, j, fo);
    store(p, i, j, fo);
    return m.rho;
}

// Bulk node (fluid or solid).
// Interior fluid or solid node: populations already gathered.
template <bool FULL>
__device__ __forceinline__ void compute(const P& p, int i, int j, int cls, const double f[Q], double fo[Q]) {
    FieldPre pre;
    if (FULL && p.fstat) fields_load(p, i, j, pre);
    Mac m = moments(f, p.hm, p.hp);
    if ((cls == CLS_SOLID && p.zero_solid_u) || cls == CLS_SOLID_ZERO) { m.ux = 0.0; m.uy = 0.0; }
    if (!(m.rho > 0.0)) flag_bad_density(p);
    if (FULL && p.macro) store_macro(p, i, j, m.rho, m.ux, m.uy, m.mxx, m.myy, m.mxy);
    if (FULL && p.fstat) fields_store(p, i, j, pre, m.rho, m.ux, m.uy);
    collide(p, m, fo);
    if (FULL && p.body) add_body_force(p, i, j, fo);
}

template <bool FULL>
__device__ __forceinline__ void finish(const P& p, int i, int j, int cls, const double f[Q]) {
    double fo[Q];
    compute<FULL>(p, i, j, cls, f, fo);
    store(p, i, j, fo);
}

// FULL: the node paths include the optional per-node work (field statistics, macroscopic
// output, body force), each behind its run-time switch.  The lean instantiation leaves it
// out; the launchers pick it when all three are off, which keeps the registers and the
// branches of that work out of the common step.
template <bool FULL>
struct PhysicsT {
    using P = StepParams<double>;
    using T = double;
    static __device__ __forceinline__ void compute(const P& p, int i, int j, int cls, const T f[Q], T fo[Q]) {
        fp64::compute<FULL>(p, i, j, cls, f, fo);
    }
    static __device__ __forceinline__ void finish(const P& p, int i, int j, int cls, const T f[Q]) {
        fp64::finish<FULL>(p, i, j, cls, f);
    }
    // Plain interior nodes (no wall, edge or solid handling), n at a time: populations f[k][.] in,
    // g[k][.] out, the macroscopic values returned in m.
    using M = Mac;
    template <int N>
    static __device__ __forceinline__ void plain(const P& p, const T (&f)[Q][N], T (&g)[Q][N], M (&m)[N]) {
#pragma unroll
        for (int n = 0; n < N; ++n) {
            T a[Q], o[Q];
#pragma unroll
            for (int k = 0; k < Q; ++k) a[k] = f[k][n];
            m[n] = moments(a, p.hm, p.hp);
            collide(p, m[n], o);
#pragma unroll
            for (int k = 0; k < Q; ++k) g[k][n] = o[k];
        }
    }
    static __device__ __forceinline__ double rho_of(const M& m) { return m.rho; }
    static __device__ __forceinline__ double edge_bulk_node(const P& p, int i, int j, int cls) {
        return fp64::edge_bulk_node<FULL>(p, i, j, cls);
    }
    static constexpr int WALL_LANES = 16;
    template <bool WAIT>
    static __device__ __forceinline__ void wall_block(const P& p, unsigned char* smem, int bb) {
        fp64::wall_block<FULL, WAIT>(p, smem, bb);
        if (!p.defer) force_tail<PhysicsT>(p, step_rec(p), smem);
    }
    // (registers of the kernels that carry the 8-lane wall path; no FP64 kernel does)
    static constexpr int WIDE_REGS = 0;
    static constexpr bool FUSED_AUX = false;         // the wall closures get a launch of their own
};
using Physics = PhysicsT<true>;
using PhysicsLean = PhysicsT<false>;

}  // namespace fp64
}  // namespace mrlbm
