// smf_slot_parity.cuh -- the PARITY predictor-corrector on a slot mesh (AMR
// meshes, meshes given cell by cell) with four threads per cell, with the
// operations of k_grad, k_stage1 and k_stage2 (smf_struct.cuh) bit for bit.
//
// The one-thread-per-cell kernels hold eight slots' geometry in registers (218
// and 110) and walk the slots one after another: at 56 k cells 436 blocks leave
// 6-10 % of the warps resident, each a chain of eight Riemann problems, 36 + 17
// + 44 us.  Here lane s of a cell's four lanes takes slots s and s + 4 (the
// second halves of split sides, mostly undefined): the face geometry, then the
// predictor's and the corrector's fluxes; the gradients go one field per lane.
// What the lanes exchange goes through shared memory within the warp, and the
// sums over the slots keep the slot order, one component per lane.
#pragma once

#include "smf_struct.cuh"

namespace zg {
namespace slotpar {

constexpr int BLOCK = 128, CELLS = BLOCK / 4;
constexpr int ROW = CELLS + 4;  // shared-memory rows: a half-warp's 4 cells x 4 slots hit 16 different banks

// p_from_q of the state whose components the cell's four lanes hold.
__device__ __forceinline__ Prim prim_of_lanes(double mine, const EosD &eos) {
    const int l0 = (threadIdx.x & 31) & ~3;
    Cons q;
    q.r = __shfl_sync(0xffffffffu, mine, l0);
    q.mu = __shfl_sync(0xffffffffu, mine, l0 + 1);
    q.mv = __shfl_sync(0xffffffffu, mine, l0 + 2);
    q.E = __shfl_sync(0xffffffffu, mine, l0 + 3);
    return p_from_q(q, eos);
}
__device__ __forceinline__ double component(const Cons &q, int s) {
    return s == 0 ? q.r : (s == 1 ? q.mu : (s == 2 ? q.mv : q.E));
}
// The field of lane s (lane 0 also writes the energy).
__device__ __forceinline__ void store_lane(const PrimPtr &z, int ic, int s, const Prim &n) {
    if (s == 0) {
        z.r[ic] = n.r;
        z.e[ic] = n.e;
    } else if (s == 1) {
        z.u[ic] = n.u;
    } else if (s == 2) {
        z.v[ic] = n.v;
    } else {
        z.p[ic] = n.p;
    }
}

struct GradShm {
    // per cell and slot: weight, neighbour offset, normal projection, normal,
    // face centre from the cell centre, flux area; flag and neighbour
    double w[8][ROW], rx[8][ROW], ry[8][ROW], nxx[8][ROW], nyy[8][ROW], nx[8][ROW], ny[8][ROW];
    int flag[8][ROW], nb[8][ROW];
};
struct FluxShm {
    double g[8][ROW];     // gradients of the four fields: x, then y
    double f[4][8][ROW];  // face fluxes times area
    bool on[8][ROW];
};

// Limited gradients of z (k_grad), and with STAGE1 the half step of the same
// state (k_stage1; a.z is z).
template <bool STAGE1>
__global__ void __launch_bounds__(BLOCK, STAGE1 ? 4 : 5) k_grad4(SmfArgs a, PrimPtr z) {
    __shared__ GradShm G;
    __shared__ FluxShm X;
    const int t = threadIdx.x, cl = t >> 2, s = t & 3;
    const int ic0 = blockIdx.x * CELLS + cl;
    const bool live = ic0 < SlotAcc::n(a);
    const int ic = live ? ic0 : SlotAcc::n(a) - 1;  // whole warps stay for the exchanges
    const SlotAcc c(a, ic);
    const double pcx = c.cx(), pcy = c.cy();
    const Prim zc = load_prim(z, ic);
    // ---- geometry of slots s and s + 4 -----------------------------------------
    double fdx[2], fdy[2], area[2], fnx[2], fny[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int q = s + 4 * h;
        const FaceG g = c.face(q);
        G.flag[q][cl] = g.flag;
        if (g.flag == BC_UNDEFINED) continue;
        double ncx, ncy;
        neib_center(c, g, q, pcx, pcy, ncx, ncy);
        const double rx = ncx - pcx, ry = ncy - pcy;
        const double d = rx * g.nx + ry * g.ny;
        const double nxx = d * g.nx, nyy = d * g.ny;
        G.w[q][cl] = g.area / cube_rn(sqrt(nxx * nxx + nyy * nyy));
        G.rx[q][cl] = rx;
        G.ry[q][cl] = ry;
        G.nxx[q][cl] = nxx;
        G.nyy[q][cl] = nyy;
        G.nx[q][cl] = g.nx;
        G.ny[q][cl] = g.ny;
        G.nb[q][cl] = g.nb;
        fnx[h] = g.nx;
        fny[h] = g.ny;
        fdx[h] = g.fcx - pcx;
        fdy[h] = g.fcy - pcy;
        area[h] = STAGE1 ? c.flux_area(g, q) : 0.0;
    }
    __syncwarp();
    // ---- the gradient of field s -------------------------------------------------
    const double *zf = s == 0 ? z.r : (s == 1 ? z.u : (s == 2 ? z.v : z.p));
    const double zk = s == 0 ? zc.r : (s == 1 ? zc.u : (s == 2 ? zc.v : zc.p));
    double A00 = 0.0, A01 = 0.0, A10 = 0.0, A11 = 0.0, Fx = 0.0, Fy = 0.0, dn[8];
    unsigned on = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int flag = G.flag[q][cl];
        if (flag == BC_UNDEFINED) continue;
        on |= 1u << q;
        const double w = G.w[q][cl], nxx = G.nxx[q][cl], nyy = G.nyy[q][cl], rx = G.rx[q][cl], ry = G.ry[q][cl];
        double zn;
        if (!is_boundary(flag)) {
            zn = zf[G.nb[q][cl]];
        } else {
            const Prim b = boundary_value(zc, G.nx[q][cl], G.ny[q][cl], flag);
            zn = s == 0 ? b.r : (s == 1 ? b.u : (s == 2 ? b.v : b.p));
        }
        const double wdx = w * nxx, wdy = w * nyy;
        A00 += wdx * rx;
        A01 += wdx * ry;
        A10 += wdy * rx;
        A11 += wdy * ry;
        const double dF = zn - zk;
        dn[q] = dF;
        Fx += w * dF * nxx;
        Fy += w * dF * nyy;
    }
    if (fabs(A11) < 1e-8) A11 = 1.0;  // 1-D case (gradient.h:270-272)
    const double inv = 1.0 / (A11 * A00 + (-A01) * A10);
    const double B00 = A11 * inv, B01 = (-A01) * inv, B10 = (-A10) * inv, B11 = A00 * inv;
    const double g0x = B00 * Fx + B01 * Fy, g0y = B10 * Fx + B11 * Fy;
    double Lx = 0.0, Ly = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        if (!(on >> q & 1u)) continue;
        const double dF_p = dn[q];
        const double du_n = g0x * G.rx[q][cl] + g0y * G.ry[q][cl];
        const double dF_m = 2.0 * du_n - dF_p;
        const double dF_lim = limiter2(a.limiter, dF_m, dF_p) * dF_p;
        Lx += G.w[q][cl] * dF_lim * G.nxx[q][cl];
        Ly += G.w[q][cl] * dF_lim * G.nyy[q][cl];
    }
    const double gx = B00 * Lx + B01 * Ly, gy = B10 * Lx + B11 * Ly;
    if (live) {
        a.gx[s][ic] = gx;
        a.gy[s][ic] = gy;
    }
    if constexpr (STAGE1) {
        X.g[s][cl] = gx;
        X.g[4 + s][cl] = gy;
        __syncwarp();
        // ---- the predictor's fluxes of slots s and s + 4 (sm_fluid.cpp:176-253) ---
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int q = s + 4 * h;
            X.on[q][cl] = on >> q & 1u;
            if (!(on >> q & 1u)) continue;
            const double dx = fdx[h], dy = fdy[h];
            Prim zm;
            zm.r = zc.r + (X.g[0][cl] * dx + X.g[4][cl] * dy);
            zm.u = zc.u + (X.g[1][cl] * dx + X.g[5][cl] * dy);
            zm.v = zc.v + (X.g[2][cl] * dx + X.g[6][cl] * dy);
            zm.p = zc.p + (X.g[3][cl] * dx + X.g[7][cl] * dy);
            zm.e = a.eos.energy_rP(zm.r, zm.p);
            if (is_bad(zm, a.eos)) zm = zc;
            FaceG g;
            g.nx = fnx[h];
            g.ny = fny[h];
            double cs, sn;
            frame<SlotAcc>(g, cs, sn);
            rot_local(zm.u, zm.v, cs, sn);
            Cons lf = flux_from_p(zm);
            rot_global(lf.mu, lf.mv, cs, sn);
            X.f[0][q][cl] = lf.r * area[h];
            X.f[1][q][cl] = lf.mu * area[h];
            X.f[2][q][cl] = lf.mv * area[h];
            X.f[3][q][cl] = lf.E * area[h];
        }
        __syncwarp();
        // ---- component s of the half step ---------------------------------------
        double F = 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (X.on[q][cl]) F += X.f[s][q][cl];
        const double dt = finalize_dt(a);
        double mine = component(q_from_p(zc), s);
        mine -= (0.5 * dt / c.flux_vol()) * F;
        if (c.axial() && s == 2) {  // sm_fluid.cpp:242-245
            const double coeff = c.vol() / c.flux_vol();
            mine += 0.5 * coeff * zc.p * dt;
        }
        Prim h = prim_of_lanes(mine, a.eos);
        if (is_bad(h, a.eos) || a.wait_in[ic] > 0) h = zc;
        if (live) store_lane(a.zhalf, ic, s, h);
    }
}

// The corrector (k_stage2, sm_fluid.cpp:255-366), and the next step's dt where
// dt_next is set.
template <int FX>
__global__ void __launch_bounds__(BLOCK, 4) k_stage2_4(SmfArgs a, double *dt_next) {
    __shared__ double f[4][8][ROW];
    __shared__ bool on[8][ROW];
    const int t = threadIdx.x, cl = t >> 2, s = t & 3;
    const int ic0 = blockIdx.x * CELLS + cl;
    const bool live = ic0 < SlotAcc::n(a);
    const int ic = live ? ic0 : SlotAcc::n(a) - 1;
    const SlotAcc c(a, ic);
    const double dt = finalize_dt(a), pcx = c.cx(), pcy = c.cy();
    const Prim zch = load_prim(a.zhalf, ic);
    const int wc = a.wait_in[ic];
#pragma unroll 1
    for (int q = s; q < 8; q += 4) {
        const FaceG g = c.face(q);
        on[q][cl] = g.flag != BC_UNDEFINED;
        if (g.flag == BC_UNDEFINED) continue;
        const Cons lf = corrector_face<FX>(a, a.zhalf, a.wait_in, c, q, g, zch, pcx, pcy, wc);
        f[0][q][cl] = lf.r;
        f[1][q][cl] = lf.mu;
        f[2][q][cl] = lf.mv;
        f[3][q][cl] = lf.E;
    }
    __syncwarp();
    const Prim zc = load_prim(a.z, ic);
    double F = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q)
        if (on[q][cl]) F += f[s][q][cl];
    double mine = component(q_from_p(zc), s);
    mine -= (dt / c.flux_vol()) * F;
    if (c.axial() && s == 2) {  // sm_fluid.cpp:347-350, with the half-step pressure
        const double coeff = c.vol() / c.flux_vol();
        mine += coeff * zch.p * dt;
    }
    Prim n = prim_of_lanes(mine, a.eos);
    int wn = wc;
    if (is_bad(n, a.eos)) {
        n = zc;
        wn = 3;
    } else if (wn > 0) {
        --wn;
    }
    if (live) {
        store_lane(a.znext, ic, s, n);
        if (s == 0) a.wait_out[ic] = wn;
    }
    if (dt_next) commit_cfl_min<BLOCK>(a, cfl_bits(a, c.dinc(), n.r, n.u, n.v, n.p), dt_next);
}

inline unsigned blocks(const SmfArgs &a) { return (unsigned)((a.smesh.n + CELLS - 1) / CELLS); }

}  // namespace slotpar
}  // namespace zg
