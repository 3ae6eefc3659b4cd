// sgs.cuh -- the dynamic mixed-scale subgrid model of the uniform cavity
// (compute_dynamic_sgs, src/uniform/solver.rs:562-828; box_filter / ddx /
// ddy / lilly_coefficient :1195-1261), evaluated on the GPU before the
// collision of a step, on the REF state (post-stream populations and
// fields).  The octree runs the same kernels on each level
// (compute_dynamic_sgs_level, src/octree/smag.rs:144-416: the same
// algorithm with the level's tau, nu and alpha in its own lattice units).
//
// One thread per node, every quantity in FP64 whatever the storage format (the
// reference's arithmetic); a launch covers gridDim.z grids of one shape (the two
// blocks of an octree level).  Three kernels for any test-filter width:
//   k_sgs_b  test-filter boxes of u_x, u_y, T (at the node and at the four
//            neighbours its central differences read, each box summed in
//            the reference's window order) and of the five products
//            (Leonard terms at the test level); grid-level S~ and |S~| from
//            pi_neq (the collision's formula), test-level S-bar and
//            temperature gradients by central differences, similarity scales
//            qsm^1/2 and Phi_sm^1/2, |T~|, |T-bar|;
//   k_sgs_c  box of qsm^1/2 and Phi_sm^1/2, the interpolated mixed forms
//            (a^alpha b^(1-alpha)), Germano tensors M and L, Lilly numerators
//            and denominators;
//   k_sgs_d  box of the numerators and denominators (regularisation),
//            Lilly coefficients clamped to [0, 0.04], nu_t and alpha_t bounded
//            below by the TRT floor, written for the collision.
// The default width of two nodes (eta_test = 2) has its windows unrolled
// (WIDTH 2).  The uniform solver then runs the first two parts as one kernel
// (k_sgs_bc2) and the third inside the collision (k_sgs_collide2).
// Sums run in the reference's order (box windows row by row).  In FP64 everything
// but the roots and the a^alpha powers is then bit-identical.  The roots are
// sqrt_nr's, within one ulp and rounded as sqrt() but for rare arguments; the
// powers CUDA's pow, within 2 ulp of the reference's, or, at the default alpha =
// 1/2, one such root of the product a b (zero where that product underflows: a
// mixed form below 2^-537, lost beside any viscosity).
#pragma once

#include "kernels.cuh"

namespace cav {

constexpr double C_DYN_MAX = 0.04;       // src/uniform/solver.rs:25
constexpr double TAU_TRT_FLOOR = 0.505;  // src/uniform/solver.rs:31

// Work planes (FP64, ny x pitch each).
enum SgsPlane {
    S_UBX, S_UBY, S_TB, S_LXX, S_LXY, S_LYY, S_LTX, S_LTY,             // k_sgs_a
    S_SHXX, S_SHXY, S_SHYY, S_SMH, S_SBXX, S_SBXY, S_SBYY, S_SMB,    // k_sgs_b
    S_GTX, S_GTY, S_GBX, S_GBY, S_QSM, S_PHI, S_TMH, S_TMB,          // k_sgs_b
    S_NUMV, S_DENV, S_NUMK, S_DENK, S_NUMIX, S_KAPMIX,               // k_sgs_c
    S_CNU, S_CK,                                                     // k_sgs_d
    S_NPLANES
};

// One grid's inputs and outputs; a launch takes two (blockIdx.z).
template <class St>
struct SgsGrid {
    const St* pops;                    // REF populations
    const typename Fmt<St>::A* rho;    // fields (rho stored minus sp.rho_off)
    const typename Fmt<St>::A* ux;
    const typename Fmt<St>::A* uy;
    const typename Fmt<St>::A* tt;
    double* W;                          // S_NPLANES work planes
    typename Fmt<St>::A* nut;           // nu_t_pre out
    typename Fmt<St>::A* at;            // alpha_t_pre out
};
template <class St>
struct SgsGrids {
    SgsGrid<St> g[2];
    // (selects: an indexed parameter would be copied to local memory)
    __device__ __forceinline__ SgsGrid<St> at(int z) const { return z == 0 ? g[0] : g[1]; }
};

struct SgsParams {
    int width = 2;           // box width in nodes: max(round(eta_test), 1)
    double dtest = 2.0;      // test filter width eta * dx (dx = 1)
    double alpha_exp = 0.5;  // smag_alpha
    double tau_s = 0.5;      // uniform: 0.5 + 3 max(nu_eff, 0.002/3), as in the collision;
                             // octree level: 0.5 + 3 nu of the level
    double nu_mol = 0.0, alpha_mol = 0.0, nu_sm_min = -0.1;
    double rho_off = 0.0;    // added to the stored density (1 when the format stores rho - 1)
};

struct Window {
    int x0, x1, y0, y1;
    double cnt;
};

// box_filter's window (src/uniform/solver.rs:1204-1227): `width` nodes
// starting (width - 1) / 2 before the node, clamped to the grid.
__device__ __forceinline__ Window box_window(const Geom& G, int ix, int iy, int width) {
    const int hl = (width - 1) / 2;
    Window w;
    w.y0 = iy - hl < 0 ? 0 : iy - hl;
    w.y1 = iy + width - hl < G.ny ? iy + width - hl : G.ny;
    w.x0 = ix - hl < 0 ? 0 : ix - hl;
    w.x1 = ix + width - hl < G.nx ? ix + width - hl : G.nx;
    w.cnt = double((w.y1 - w.y0) * (w.x1 - w.x0));
    return w;
}

// ddx / ddy (src/uniform/solver.rs:1229-1245): central, clamped at the walls.
template <class A>
__device__ __forceinline__ double ddx_f(const A* __restrict__ p, const Geom& G, int ix, int iy) {
    const int xm = ix == 0 ? 0 : ix - 1, xp = ix + 1 >= G.nx ? G.nx - 1 : ix + 1;
    return 0.5 * (double(p[iy * G.pitch + xp]) - double(p[iy * G.pitch + xm]));
}
template <class A>
__device__ __forceinline__ double ddy_f(const A* __restrict__ p, const Geom& G, int ix, int iy) {
    const int ym = iy == 0 ? 0 : iy - 1, yp = iy + 1 >= G.ny ? G.ny - 1 : iy + 1;
    return 0.5 * (double(p[yp * G.pitch + ix]) - double(p[ym * G.pitch + ix]));
}

// lilly_coefficient (src/uniform/solver.rs:1250-1261).
__host__ __device__ __forceinline__ double lilly_coefficient(double num, double den) {
    if (!isfinite(den) || !isfinite(num) || den <= 0.0) return 0.0;
    const double c = 0.5 * num / den;
    if (!isfinite(c)) return 0.0;
    return c < 0.0 ? 0.0 : (c > C_DYN_MAX ? C_DYN_MAX : c);
}

// Test-filter box of u_x, u_y, T at (x, y): box_filter's window and order.
template <class A>
__device__ __forceinline__ void box3(const A* __restrict__ ux, const A* __restrict__ uy, const A* __restrict__ tt,
                                     const Geom& G, int x, int y, int width, double& bu, double& bv, double& bt) {
    const Window w = box_window(G, x, y, width);
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int yy = w.y0; yy < w.y1; ++yy)
        for (int xx = w.x0; xx < w.x1; ++xx) {
            const int k = yy * G.pitch + xx;
            s0 += double(ux[k]);
            s1 += double(uy[k]);
            s2 += double(tt[k]);
        }
    bu = s0 / w.cnt;
    bv = s1 / w.cnt;
    bt = s2 / w.cnt;
}

// What the first part of the model (k_sgs_b) gives for a node.
struct SgsB {
    double ubx, uby, tb, l[5];                                   // boxes of u_x, u_y, T and of the five products
    double shxx, shxy, shyy, smh, sxx, sxy, syy, smb;            // grid- and test-level strain
    double gtx, gty, gbx, gby, qsm, phi, tmh, tmb;
};

// Grid-level S~ and |S~| of a node from pi_neq, the collision's formula.
template <class St>
__device__ __forceinline__ void sgs_strain(const SgsGrid<St>& io, const Geom& G, int ix, int iy, double ux_k,
                                           double uy_k, const SgsParams& sp, SgsB& o) {
    constexpr bool SH = Fmt<St>::SHIFT;
    const double rho_k = double(io.rho[iy * G.pitch + ix]) + sp.rho_off;
    double pi_xx = 0.0, pi_xy = 0.0, pi_yy = 0.0;
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        const double fi = double(ldp(io.pops, G, i, iy, ix)) + (SH ? WD(i) : 0.0);
        const double fneq = fi - feq_full<double>(i, rho_k, ux_k, uy_k);
        if (CX(i) != 0) pi_xx += fneq;
        if (CX(i) * CY(i) != 0) pi_xy += CX(i) * CY(i) > 0 ? fneq : -fneq;
        if (CY(i) != 0) pi_yy += fneq;
    }
    const double rho_m = rho_k > 1e-12 ? rho_k : 1e-12;
    const double denom = 2.0 * CS2 * sp.tau_s * rho_m;
    const double pi2 = pi_xx * pi_xx + 2.0 * pi_xy * pi_xy + pi_yy * pi_yy;
    const double inv = rcp_rn(denom);
    o.shxx = quot_rn(-pi_xx, denom, inv);
    o.shxy = quot_rn(-pi_xy, denom, inv);
    o.shyy = quot_rn(-pi_yy, denom, inv);
    o.smh = quot_rn(sqrt_nr(pi2), denom, inv);
}

// qsm^1/2 and Phi_sm^1/2 of a node from its fields and boxes.
__device__ __forceinline__ void sgs_small(double u, double v, double t, double ub, double vb, double tb, double& q,
                                          double& phi) {
    const double du = u - ub, dv = v - vb;
    const double r = sqrt_nr(0.5 * (du * du + dv * dv));
    q = r / 2.0;
    phi = 0.5 * fabs(t - tb) * r;
}

// |T~| and |T-bar| from the gradients and strains.
__device__ __forceinline__ void sgs_flux(SgsB& o) {
    const double th_x = o.gtx * o.shxx + o.gty * o.shxy;
    const double th_y = o.gtx * o.shxy + o.gty * o.shyy;
    o.tmh = sqrt_nr(2.0 * (th_x * th_x + th_y * th_y));
    const double tb_x = o.gbx * o.sxx + o.gby * o.sxy;
    const double tb_y = o.gbx * o.sxy + o.gby * o.syy;
    o.tmb = sqrt_nr(2.0 * (tb_x * tb_x + tb_y * tb_y));
}

// The first part for any test-filter width.
template <class St>
__device__ __forceinline__ void sgs_node_b(const SgsGrid<St>& io, const Geom& G, int ix, int iy, const SgsParams& sp,
                                           SgsB& o) {
    using A = typename Fmt<St>::A;
    const A* ux = io.ux;
    const A* uy = io.uy;
    const A* tt = io.tt;
    const int k = iy * G.pitch + ix;
    // test-filter boxes at the node and at the neighbours of its central
    // differences (ddx / ddy clamp at the walls), and the Leonard boxes
    const int xm = ix == 0 ? 0 : ix - 1, xp = ix + 1 >= G.nx ? G.nx - 1 : ix + 1;
    const int ym = iy == 0 ? 0 : iy - 1, yp = iy + 1 >= G.ny ? G.ny - 1 : iy + 1;
    double ubx_xm, uby_xm, tb_xm, ubx_xp, uby_xp, tb_xp, ubx_ym, uby_ym, tb_ym, ubx_yp, uby_yp, tb_yp;
    box3<A>(ux, uy, tt, G, ix, iy, sp.width, o.ubx, o.uby, o.tb);
    box3<A>(ux, uy, tt, G, xm, iy, sp.width, ubx_xm, uby_xm, tb_xm);
    box3<A>(ux, uy, tt, G, xp, iy, sp.width, ubx_xp, uby_xp, tb_xp);
    box3<A>(ux, uy, tt, G, ix, ym, sp.width, ubx_ym, uby_ym, tb_ym);
    box3<A>(ux, uy, tt, G, ix, yp, sp.width, ubx_yp, uby_yp, tb_yp);
    const Window w = box_window(G, ix, iy, sp.width);
    double l[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int yy = w.y0; yy < w.y1; ++yy)
        for (int xx = w.x0; xx < w.x1; ++xx) {
            const int kk = yy * G.pitch + xx;
            const double u = ux[kk], v = uy[kk], t = tt[kk];
            l[0] += u * u;
            l[1] += u * v;
            l[2] += v * v;
            l[3] += u * t;
            l[4] += v * t;
        }
#pragma unroll
    for (int p = 0; p < 5; ++p) o.l[p] = l[p] / w.cnt;
    const double ux_k = ux[k], uy_k = uy[k], t_k = tt[k];
    sgs_strain<St>(io, G, ix, iy, ux_k, uy_k, sp, o);
    // ddx / ddy of the boxed fields (src/uniform/solver.rs:1229-1245)
    o.sxx = 0.5 * (ubx_xp - ubx_xm);
    o.syy = 0.5 * (uby_yp - uby_ym);
    o.sxy = 0.5 * (0.5 * (uby_xp - uby_xm) + 0.5 * (ubx_yp - ubx_ym));
    o.smb = sqrt_nr(o.sxx * o.sxx + 2.0 * o.sxy * o.sxy + o.syy * o.syy);
    o.gtx = ddx_f(tt, G, ix, iy);
    o.gty = ddy_f(tt, G, ix, iy);
    o.gbx = 0.5 * (tb_xp - tb_xm);
    o.gby = 0.5 * (tb_yp - tb_ym);
    sgs_small(ux_k, uy_k, t_k, o.ubx, o.uby, o.tb, o.qsm, o.phi);
    sgs_flux(o);
}

// The first part for the test filter of two nodes: the box of a node covers it
// and its upper neighbours in x and y, cut at the grid's edge, its count (1, 2
// or 4) divided out exactly by a multiplication.  The boxes a node needs -- its
// own, those of the four neighbours that its central differences read (the
// clamped ones are its own) and that of the diagonal one of its window -- all
// come from 13 nodes, kept in registers.  WINDOW: also the boxes of qsm^1/2
// and Phi_sm^1/2 at the node (from the four nodes of its window).
template <class St, bool WINDOW>
__device__ __forceinline__ void sgs_node_b2(const SgsGrid<St>& io, const Geom& G, int ix, int iy, const SgsParams& sp,
                                            SgsB& o, double& qbar_h, double& phibar_h) {
    const int k = iy * G.pitch + ix;
    // offsets of columns ix - 1 .. ix + 2 and rows iy - 1 .. iy + 2, kept in
    // the grid (values taken from a clamped place are not used)
    const bool x0 = ix == 0, y0 = iy == 0;
    const bool x1 = ix + 1 < G.nx, y1 = iy + 1 < G.ny, x2 = ix + 2 < G.nx, y2 = iy + 2 < G.ny;
    const int ox[4] = {x0 ? 0 : -1, 0, x1 ? 1 : 0, x2 ? 2 : 0};
    const int oy[4] = {y0 ? 0 : -G.pitch, 0, y1 ? G.pitch : 0, y2 ? 2 * G.pitch : 0};
    // the box's mean of four values in window order; vx / vy: the second
    // column / row is in the grid
    auto box = [](double a, double b, double c, double d, bool vx, bool vy) {
        const double s = ((a + (vx ? b : 0.0)) + (vy ? c : 0.0)) + (vx && vy ? d : 0.0);
        return s * ((vx ? 0.5 : 1.0) * (vy ? 0.5 : 1.0));
    };
    struct Boxes {
        double c, w, e, s, n, ne;
    };
    double uv[4][4], vv[4][4], tv[4][4];  // [row][column]; the corners no box reads stay unused
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if ((j == 0 && (i == 0 || i == 3)) || (j == 3 && i == 0)) continue;
            const int kk = k + oy[j] + ox[i];
            uv[j][i] = io.ux[kk];
            vv[j][i] = io.uy[kk];
            tv[j][i] = io.tt[kk];
        }
    auto boxes = [&](const double (&p)[4][4]) {
        Boxes b;
        b.c = box(p[1][1], p[1][2], p[2][1], p[2][2], x1, y1);
        const double w = box(p[1][0], p[1][1], p[2][0], p[2][1], true, y1);
        const double e = box(p[1][2], p[1][3], p[2][2], p[2][3], x2, y1);
        const double s = box(p[0][1], p[0][2], p[1][1], p[1][2], x1, true);
        const double n = box(p[2][1], p[2][2], p[3][1], p[3][2], x1, y2);
        b.ne = box(p[2][2], p[2][3], p[3][2], p[3][3], x2, y2);
        b.w = x0 ? b.c : w;
        b.e = x1 ? e : b.c;
        b.s = y0 ? b.c : s;
        b.n = y1 ? n : b.c;
        return b;
    };
    const Boxes bu = boxes(uv), bv = boxes(vv), bt = boxes(tv);
    o.ubx = bu.c;
    o.uby = bv.c;
    o.tb = bt.c;
    auto box_prod = [&](const double (&p)[4][4], const double (&q)[4][4]) {
        return box(p[1][1] * q[1][1], p[1][2] * q[1][2], p[2][1] * q[2][1], p[2][2] * q[2][2], x1, y1);
    };
    o.l[0] = box_prod(uv, uv);
    o.l[1] = box_prod(uv, vv);
    o.l[2] = box_prod(vv, vv);
    o.l[3] = box_prod(uv, tv);
    o.l[4] = box_prod(vv, tv);
    const double t_k = tv[1][1];
    sgs_strain<St>(io, G, ix, iy, uv[1][1], vv[1][1], sp, o);
    o.sxx = 0.5 * (bu.e - bu.w);
    o.syy = 0.5 * (bv.n - bv.s);
    o.sxy = 0.5 * (0.5 * (bv.e - bv.w) + 0.5 * (bu.n - bu.s));
    o.smb = sqrt_nr(o.sxx * o.sxx + 2.0 * o.sxy * o.sxy + o.syy * o.syy);
    o.gtx = 0.5 * ((x1 ? tv[1][2] : t_k) - (x0 ? t_k : tv[1][0]));
    o.gty = 0.5 * ((y1 ? tv[2][1] : t_k) - (y0 ? t_k : tv[0][1]));
    o.gbx = 0.5 * (bt.e - bt.w);
    o.gby = 0.5 * (bt.n - bt.s);
    sgs_small(uv[1][1], vv[1][1], t_k, bu.c, bv.c, bt.c, o.qsm, o.phi);
    if constexpr (WINDOW) {
        double q1, q2, q3, p1, p2, p3;
        sgs_small(uv[1][2], vv[1][2], tv[1][2], bu.e, bv.e, bt.e, q1, p1);
        sgs_small(uv[2][1], vv[2][1], tv[2][1], bu.n, bv.n, bt.n, q2, p2);
        sgs_small(uv[2][2], vv[2][2], tv[2][2], bu.ne, bv.ne, bt.ne, q3, p3);
        qbar_h = box(o.qsm, q1, q2, q3, x1, y1);
        phibar_h = box(o.phi, p1, p2, p3, x1, y1);
    }
    sgs_flux(o);
}

template <class St, int WIDTH>
__global__ void __launch_bounds__(128) k_sgs_b(SgsGrids<St> S, Geom G, SgsParams sp) {
    pdl_wait();
    const int ix = blockIdx.x * blockDim.x + threadIdx.x;
    const int iy = blockIdx.y * blockDim.y + threadIdx.y;
    if (ix >= G.nx || iy >= G.ny) return;
    const SgsGrid<St> io = S.at(blockIdx.z);
    SgsB o;
    if constexpr (WIDTH == 2) {
        double qb, pb;
        sgs_node_b2<St, false>(io, G, ix, iy, sp, o, qb, pb);
    } else {
        sgs_node_b<St>(io, G, ix, iy, sp, o);
    }
    const long long P = G.plane;
    double* __restrict__ w = io.W + iy * G.pitch + ix;
    w[S_UBX * P] = o.ubx;
    w[S_UBY * P] = o.uby;
    w[S_TB * P] = o.tb;
#pragma unroll
    for (int p = 0; p < 5; ++p) w[(S_LXX + p) * P] = o.l[p];
    w[S_SHXX * P] = o.shxx;
    w[S_SHXY * P] = o.shxy;
    w[S_SHYY * P] = o.shyy;
    w[S_SMH * P] = o.smh;
    w[S_SBXX * P] = o.sxx;
    w[S_SBXY * P] = o.sxy;
    w[S_SBYY * P] = o.syy;
    w[S_SMB * P] = o.smb;
    w[S_GTX * P] = o.gtx;
    w[S_GTY * P] = o.gty;
    w[S_GBX * P] = o.gbx;
    w[S_GBY * P] = o.gby;
    w[S_QSM * P] = o.qsm;
    w[S_PHI * P] = o.phi;
    w[S_TMH * P] = o.tmh;
    w[S_TMB * P] = o.tmb;
}

// a^alpha b^(1 - alpha) of the mixed forms.  HALF: alpha = 1/2, as one square
// root (B200, us per step with eight pow / with four roots: 64 x 256 11.5 / 7.5, 128 x
// 512 17.7 / 12.5).
template <bool HALF>
__device__ __forceinline__ double sgs_mix(double a, double b, double ae) {
    if constexpr (HALF)
        return sqrt_nr(a * b);
    else
        return pow(a, ae) * pow(b, 1.0 - ae);
}

// The second part: mixed forms, Germano tensors, Lilly numerators and
// denominators of a node.
template <bool HALF>
__device__ __forceinline__ void sgs_node_c(const SgsB& o, double qbar_h, double phibar_h, const SgsParams& sp,
                                           double* __restrict__ w, long long P) {
    const double ae = sp.alpha_exp, dx = 1.0, dtest = sp.dtest, delta_t = 1.0;
    const double nu_mix_t = sgs_mix<HALF>(dtest * dtest * o.smb, dtest * qbar_h, ae);
    const double nu_mix_g = sgs_mix<HALF>(dx * dx * o.smh, dx * o.qsm, ae);
    const double kap_mix_t =
        sgs_mix<HALF>(dtest * dtest * dtest / delta_t * o.tmb, dtest / delta_t * phibar_h, ae);
    const double kap_mix_g = sgs_mix<HALF>(dx * dx * dx / delta_t * o.tmh, dx / delta_t * o.phi, ae);
    const double mxx = nu_mix_t * o.sxx - nu_mix_g * o.shxx;
    const double mxy = nu_mix_t * o.sxy - nu_mix_g * o.shxy;
    const double myy = nu_mix_t * o.syy - nu_mix_g * o.shyy;
    const double mx = kap_mix_t * o.gbx - kap_mix_g * o.gtx;
    const double my = kap_mix_t * o.gby - kap_mix_g * o.gty;
    const double lxx = o.l[0] - o.ubx * o.ubx;
    const double lxy = o.l[1] - o.ubx * o.uby;
    const double lyy = o.l[2] - o.uby * o.uby;
    const double lkk3 = quot_rn(lxx + lyy, 3.0, 1.0 / 3.0);
    const double ldxx = lxx - lkk3, ldyy = lyy - lkk3;
    const double ljx = o.l[3] - o.ubx * o.tb;
    const double ljy = o.l[4] - o.uby * o.tb;
    w[S_NUMV * P] = ldxx * mxx + 2.0 * lxy * mxy + ldyy * myy;
    w[S_DENV * P] = mxx * mxx + 2.0 * mxy * mxy + myy * myy;
    w[S_NUMK * P] = ljx * mx + ljy * my;
    w[S_DENK * P] = mx * mx + my * my;
    w[S_NUMIX * P] = nu_mix_g;
    w[S_KAPMIX * P] = kap_mix_g;
}

// Box of plane p at a node, in window order.
template <int WIDTH>
__device__ __forceinline__ double sgs_box(const double* __restrict__ p, const Geom& G, int ix, int iy, int width) {
    if constexpr (WIDTH == 2) {
        const bool vx = ix + 1 < G.nx, vy = iy + 1 < G.ny;
        const int kx = vx ? 1 : 0, ky = vy ? G.pitch : 0;
        const double* __restrict__ w = p + (iy * G.pitch + ix);
        const double a = w[0], b = w[kx], c = w[ky], d = w[kx + ky];
        const double s = ((a + (vx ? b : 0.0)) + (vy ? c : 0.0)) + (vx && vy ? d : 0.0);
        return s * ((vx ? 0.5 : 1.0) * (vy ? 0.5 : 1.0));
    } else {
        const Window w = box_window(G, ix, iy, width);
        double s = 0.0;
        for (int yy = w.y0; yy < w.y1; ++yy)
            for (int xx = w.x0; xx < w.x1; ++xx) s += p[yy * G.pitch + xx];
        return s / w.cnt;
    }
}

template <class St, int WIDTH, bool HALF>
__global__ void __launch_bounds__(128) k_sgs_c(SgsGrids<St> S, Geom G, SgsParams sp) {
    pdl_wait();
    const int ix = blockIdx.x * blockDim.x + threadIdx.x;
    const int iy = blockIdx.y * blockDim.y + threadIdx.y;
    if (ix >= G.nx || iy >= G.ny) return;
    double* __restrict__ W = S.at(blockIdx.z).W;
    const long long P = G.plane;
    double* __restrict__ w = W + iy * G.pitch + ix;
    SgsB o;
    o.ubx = w[S_UBX * P];
    o.uby = w[S_UBY * P];
    o.tb = w[S_TB * P];
#pragma unroll
    for (int p = 0; p < 5; ++p) o.l[p] = w[(S_LXX + p) * P];
    o.shxx = w[S_SHXX * P];
    o.shxy = w[S_SHXY * P];
    o.shyy = w[S_SHYY * P];
    o.smh = w[S_SMH * P];
    o.sxx = w[S_SBXX * P];
    o.sxy = w[S_SBXY * P];
    o.syy = w[S_SBYY * P];
    o.smb = w[S_SMB * P];
    o.gtx = w[S_GTX * P];
    o.gty = w[S_GTY * P];
    o.gbx = w[S_GBX * P];
    o.gby = w[S_GBY * P];
    o.qsm = w[S_QSM * P];
    o.phi = w[S_PHI * P];
    o.tmh = w[S_TMH * P];
    o.tmb = w[S_TMB * P];
    const double qbar_h = sgs_box<WIDTH>(W + S_QSM * P, G, ix, iy, sp.width);
    const double phibar_h = sgs_box<WIDTH>(W + S_PHI * P, G, ix, iy, sp.width);
    sgs_node_c<HALF>(o, qbar_h, phibar_h, sp, w, P);
}

// k_sgs_b and k_sgs_c in one for the test filter of two nodes: a node forms
// qsm^1/2 and Phi_sm^1/2 of its window itself (three more square roots), so only
// the six results go through memory and one launch is saved.  Held to 128 registers,
// four CTAs per SM: with 138 the step on 128 x 512 took 14.8 us instead of 12.4.
template <class St, bool HALF>
__global__ void __launch_bounds__(128, 4) k_sgs_bc2(SgsGrids<St> S, Geom G, SgsParams sp) {
    pdl_wait();
    const int ix = blockIdx.x * blockDim.x + threadIdx.x;
    const int iy = blockIdx.y * blockDim.y + threadIdx.y;
    if (ix >= G.nx || iy >= G.ny) return;
    const SgsGrid<St> io = S.at(blockIdx.z);
    SgsB o;
    double qbar_h, phibar_h;
    sgs_node_b2<St, true>(io, G, ix, iy, sp, o, qbar_h, phibar_h);
    sgs_node_c<HALF>(o, qbar_h, phibar_h, sp, io.W + iy * G.pitch + ix, G.plane);
}

// The third part of a node: regularised Lilly coefficients, nu_t and alpha_t.
template <int WIDTH>
__device__ __forceinline__ void sgs_node_d(double* __restrict__ W, const Geom& G, int ix, int iy, const SgsParams& sp,
                                           double& nut, double& at_out) {
    const long long P = G.plane;
    const int k = iy * G.pitch + ix;
    double s[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) s[p] = sgs_box<WIDTH>(W + (S_NUMV + p) * P, G, ix, iy, sp.width);
    const double cnu = lilly_coefficient(s[0], s[1]);
    const double ck = lilly_coefficient(s[2], s[3]);
    W[S_CNU * P + k] = cnu;
    W[S_CK * P + k] = ck;
    const double margin = (TAU_TRT_FLOOR - 0.5) / 3.0;
    const double nt = cnu * W[S_NUMIX * P + k];
    const double nu_t_min = fmax(sp.nu_sm_min * sp.nu_mol, margin - sp.nu_mol);
    nut = nt < nu_t_min ? nu_t_min : nt;
    const double at = ck * W[S_KAPMIX * P + k];
    const double alpha_t_min = fmax(sp.nu_sm_min * sp.alpha_mol, margin - sp.alpha_mol);
    at_out = at < alpha_t_min ? alpha_t_min : at;
}

template <class St, int WIDTH>
__global__ void __launch_bounds__(128) k_sgs_d(SgsGrids<St> S, Geom G, SgsParams sp) {
    using A = typename Fmt<St>::A;
    pdl_wait();
    const int ix = blockIdx.x * blockDim.x + threadIdx.x;
    const int iy = blockIdx.y * blockDim.y + threadIdx.y;
    if (ix >= G.nx || iy >= G.ny) return;
    const SgsGrid<St> io = S.at(blockIdx.z);
    const int k = iy * G.pitch + ix;
    double nut, at;
    sgs_node_d<WIDTH>(io.W, G, ix, iy, sp, nut, at);
    io.nut[k] = A(nut);
    io.at[k] = A(at);
}

// The last part of the model (width 2) and the collision of the node that it is for
// (k_collide_ref with the node's nu_t / alpha_t).
template <class St>
__global__ void __launch_bounds__(128) k_sgs_collide2(const St* __restrict__ src, St* __restrict__ dst,
                                                      const typename Fmt<St>::A* __restrict__ rho,
                                                      const typename Fmt<St>::A* __restrict__ ux,
                                                      const typename Fmt<St>::A* __restrict__ uy,
                                                      const typename Fmt<St>::A* __restrict__ tt,
                                                      typename Fmt<St>::A* __restrict__ fy,
                                                      typename Fmt<St>::A* __restrict__ nut, double* __restrict__ W,
                                                      Geom G, SgsParams sp, StepScalars<typename Fmt<St>::A> c) {
    using A = typename Fmt<St>::A;
    pdl_wait();
    const int ix = blockIdx.x * blockDim.x + threadIdx.x;
    const int iy = blockIdx.y * blockDim.y + threadIdx.y;
    if (ix >= G.nx || iy >= G.ny) return;
    double nt, at;
    sgs_node_d<2>(W, G, ix, iy, sp, nt, at);
    const A nt_a = A(nt), at_a = A(at);
    collide_ref_node<St>(src, dst, rho, ux, uy, tt, fy, nut, G, ix, iy, c, &nt_a, &at_a);
}

// Mean and max of the Lilly coefficients (cs_dyn_mean / _max, kappa_dyn_mean
// / _max): one CTA, sums in a fixed order.
static __global__ void __launch_bounds__(256) k_sgs_stats(const double* __restrict__ W, Geom G,
                                                          double* __restrict__ out) {
    const long long P = G.plane;
    __shared__ double sh[4][256];
    double s0 = 0.0, m0 = 0.0, s1 = 0.0, m1 = 0.0;
    const int n = G.nx * G.ny;
    for (int j = threadIdx.x; j < n; j += 256) {
        const int k = (j / G.nx) * G.pitch + (j % G.nx);
        const double a = W[S_CNU * P + k], b = W[S_CK * P + k];
        s0 += a;
        m0 = fmax(m0, a);
        s1 += b;
        m1 = fmax(m1, b);
    }
    sh[0][threadIdx.x] = s0;
    sh[1][threadIdx.x] = m0;
    sh[2][threadIdx.x] = s1;
    sh[3][threadIdx.x] = m1;
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0, c = 0.0, d = 0.0;
        for (int t = 0; t < 256; ++t) {
            a += sh[0][t];
            b = fmax(b, sh[1][t]);
            c += sh[2][t];
            d = fmax(d, sh[3][t]);
        }
        out[0] = a / double(n);
        out[1] = b;
        out[2] = c / double(n);
        out[3] = d;
    }
}

}  // namespace cav
