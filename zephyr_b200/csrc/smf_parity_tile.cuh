// smf_parity_tile.cuh -- the PARITY step of a structured rectangle as ONE
// kernel per stage for the HLLC and HLL fluxes: a tile of cells with its halo
// in shared memory, limited gradients, predictor, every face once, update and
// the next step's dt, with the operations of the gather kernels of
// smf_struct.cuh bit for bit (signs of exact zeros aside, as there).
//
// What allows a face to be evaluated once although the reference evaluates it
// from both of its cells and the two results differ in their last bits:
//  * the reconstruction of a cell at a face does not depend on the side that
//    asks for it (except across a periodic seam, where the asking cell's
//    mirror geometry enters: the tile's edge faces use those offsets);
//  * seen from the high cell B the frame is reversed, and every quantity of
//    HLLC up to the contact speed is the exact negative or the exact copy of
//    the low cell's; the contact speed's numerator is summed in another order,
//    and so are the five terms of the flux.  `hllc_both` forms the shared part
//    once and these parts twice.  HLL is exactly antisymmetric.
// The least-squares geometry of an axis-aligned rectangle is a table per axis
// (the reference's expressions, filled on the host without contraction); the
// products with the zero components of the normals are left out: they are
// exact zeros unless a value is not finite, and then the cell or the face
// takes the reference's full expressions (`odd_cell`, `odd_face`).
//
// What bounded the gather kernels (1031 x 517, second order, 237 us of kernels,
// 224 us a step): 142 and 104 registers (18-23 % of the warps resident, issue
// slots 37-41 % used) and the second evaluation of faces and of geometry
// quotients.  One kernel 144 us; with zero numerators kept out of the divisions
// (div_z) 104 us.  Tiles of 12 rows at two blocks per SM (72 registers): 6 rows
// at 2, 3 and 4 blocks took 200, 171 and 186 us, 12 rows at one block 203.
// The first-order step stays in the gather kernel: its four evaluations of HLLC
// per cell cost no more than this form's two double ones with the tile's halo
// (1850 against 1425 instructions a cell).
// This file is compiled with -fmad=false.
#pragma once

#include <type_traits>

#include "smf_struct.cuh"

namespace zg {
namespace ptile {

struct Args {
    SmfArgs a;
    Axis x, y;
    PrimPtr zin, zout;      // source and result of the stage
    const double *dt_in;    // this step's dt
    double *dt_next;        // the next step's (last stage; null: not asked for)
};

// Physical flux along an axis of a state with normal velocity n, tangential t
// (models.cpp:131-137).
struct F4 {
    double r, n, t, E;
};
__device__ __forceinline__ F4 flux_n(double r, double n, double t, double p, double e) {
    F4 f;
    const double rn = r * n;
    f.r = rn;
    f.n = rn * n + p;
    f.t = rn * t;
    f.E = (r * (e + 0.5 * (n * n + t * t)) + p) * n;
    return f;
}

// A face state: density, normal and tangential velocity (axis directions),
// pressure, energy.
struct FState {
    double r, n, t, p, e;
};

// Values that are not finite: both views of the face with the reference's
// rotations (rotate.cpp:7-77).  Out of line, practically never called.
static __device__ __noinline__ void odd_face(FState A, FState B, int axis, bool hll_flux, EosD eos, F4 &lo, F4 &hi) {
    Cons out[2];
#pragma unroll 1
    for (int view = 0; view < 2; ++view) {
        // from the low cell: normal +axis; from the high cell: -axis
        const double cs = axis == 0 ? (view == 0 ? 1.0 : -1.0) : (view == 0 ? 0.0 : -0.0);
        const double sn = axis == 0 ? (view == 0 ? 0.0 : -0.0) : (view == 0 ? 1.0 : -1.0);
        const FState &a = view == 0 ? A : B, &b = view == 0 ? B : A;
        Prim zm{a.r, axis == 0 ? a.n : a.t, axis == 0 ? a.t : a.n, a.p, a.e};
        Prim zp{b.r, axis == 0 ? b.n : b.t, axis == 0 ? b.t : b.n, b.p, b.e};
        rot_local(zm.u, zm.v, cs, sn);
        rot_local(zp.u, zp.v, cs, sn);
        Cons lf = hll_flux ? hll(zm, zp, eos) : hllc(zm, zp, eos);
        rot_global(lf.mu, lf.mv, cs, sn);
        out[view] = lf;
    }
    lo = axis == 0 ? F4{out[0].r, out[0].mu, out[0].mv, out[0].E} : F4{out[0].r, out[0].mv, out[0].mu, out[0].E};
    hi = axis == 0 ? F4{-out[1].r, -out[1].mu, -out[1].mv, -out[1].E}
                   : F4{-out[1].r, -out[1].mv, -out[1].mu, -out[1].E};
}

// hll.cpp:23-57; exactly antisymmetric, so one value serves both cells.
// put(view, flux) takes the flux of the low cell's view (0) and the negated one
// of the high cell's (1).  False: a value is not finite, nothing was put.
template <class Put>
__device__ __forceinline__ bool hll_both(const FState &A, const FState &B, const EosD &eos, Put &&put) {
    const double cA = eos.sound_speed_rP(A.r, A.p), cB = eos.sound_speed_rP(B.r, B.p);
    if (!(fabs(cA + cB + A.n + B.n) + (fabs(A.t) + fabs(B.t)) < CUDART_INF)) return false;
    const double SL = smin(A.n - cA, smin(B.n - cB, 0.0));
    const double SR = smax(A.n + cA, smax(B.n + cB, 0.0));
    const F4 fA = flux_n(A.r, A.n, A.t, A.p, A.e), fB = flux_n(B.r, B.n, B.t, B.p, B.e);
    const double EA = A.r * (A.e + 0.5 * (A.n * A.n + A.t * A.t)), EB = B.r * (B.e + 0.5 * (B.n * B.n + B.t * B.t));
    const double SLR = SL * SR, den = SR - SL;
    F4 o;
    o.r = (SR * fA.r - SL * fB.r + SLR * (B.r - A.r)) / den;
    o.n = (SR * fA.n - SL * fB.n + SLR * (B.r * B.n - A.r * A.n)) / den;
    o.t = (SR * fA.t - SL * fB.t + SLR * (B.r * B.t - A.r * A.t)) / den;
    o.E = (SR * fA.E - SL * fB.E + SLR * (EB - EA)) / den;
    put(0, o);
    put(1, o);
    return true;
}

// hllc.cpp:23-83 seen from the low cell and, negated, from the high cell, in
// axis directions; as hll_both.
template <class Put>
__device__ __forceinline__ bool hllc_both(const FState &A, const FState &B, const EosD &eos, Put &&put) {
    const double cA = eos.sound_speed_rP(A.r, A.p), cB = eos.sound_speed_rP(B.r, B.p);
    const double SL = smin(A.n - cA, B.n - cB), SR = smax(A.n + cA, B.n + cB);
    // (both sides' own values: the minimum of a number and a NaN is the first)
    if (!(fabs(cA + cB + A.n + B.n) + (fabs(A.t) + fabs(B.t)) < CUDART_INF)) return false;
    if (SL >= 0.0 || SR <= 0.0) {  // each cell tests its own side first
        const F4 fA = flux_n(A.r, A.n, A.t, A.p, A.e), fB = flux_n(B.r, B.n, B.t, B.p, B.e);
        put(0, SL >= 0.0 ? fA : fB);
        put(1, SR <= 0.0 ? fB : fA);
        return true;
    }
    const double aL = A.r * (SL - A.n), aR = B.r * (SR - B.n);
    const double d = A.p - B.p, X = aR * B.n, Y = aL * A.n, den = aR - aL;
    const double EA = A.e + 0.5 * (A.n * A.n + A.t * A.t), EB = B.e + 0.5 * (B.n * B.n + B.t * B.t);
    const double pA = A.p / aL, pB = B.p / aR;
    const double rnA = A.r * A.n, rtA = A.r * A.t, rEA = A.r * EA;
    const double rnB = B.r * B.n, rtB = B.r * B.t, rEB = B.r * EB;
#pragma unroll 1
    for (int view = 0; view < 2; ++view) {
        const double SC = div_z(view == 0 ? (d + X) - Y : (d - Y) + X, den);
        const double rsL = aL / (SL - SC), rsR = aR / (SR - SC);
        const double EsL = EA + (SC - A.n) * (SC + pA), EsR = EB + (SC - B.n) * (SC + pB);
        const double aSC = fabs(SC);
        // 0.5 (F_L + F_R + first outer wave + contact + second outer wave)
        auto sum = [&](double s, double qL, double qsL, double qR, double qsR) {
            const double wl = SL * (qsL - qL), wr = SR * (qsR - qR), wc = aSC * (qsL - qsR);
            return 0.5 * (s + (view == 0 ? wl : wr) + wc + (view == 0 ? wr : wl));
        };
        put(view, F4{sum(rnA + rnB, A.r, rsL, B.r, rsR), sum((rnA * A.n + A.p) + (rnB * B.n + B.p), rnA, rsL * SC, rnB, rsR * SC),
                     sum(rnA * A.t + rnB * B.t, rtA, rsL * A.t, rtB, rsR * B.t),
                     sum((rEA + A.p) * A.n + (rEB + B.p) * B.n, rEA, rsL * EsL, rEB, rsR * EsR)});
    }
    return true;
}

// Cell ic's limited gradients and half step with the reference's full
// expressions, for cells with a value that is not finite in reach.  Out of
// line, practically never called.
static __device__ __noinline__ void odd_cell(const SmfArgs &a, PrimPtr z, int ic, bool waiting, double dt, double gx[4],
                                             double gy[4], Prim &h) {
    StructAcc c(a, ic);
    const Prim zc = load_prim(z, ic);
    lsm_limited(c, z, a.limiter, zc, gx, gy);
    h = zc;
    if (waiting) return;
    Cons q = q_from_p(zc), F{0.0, 0.0, 0.0, 0.0};
    for (int s = 0; s < 4; ++s) {
        const FaceG g = c.face(s);
        const double dx = g.fcx - c.cx(), dy = g.fcy - c.cy();
        Prim zm{zc.r + (gx[0] * dx + gy[0] * dy), zc.u + (gx[1] * dx + gy[1] * dy), zc.v + (gx[2] * dx + gy[2] * dy),
                zc.p + (gx[3] * dx + gy[3] * dy), 0.0};
        zm.e = a.eos.energy_rP(zm.r, zm.p);
        if (is_bad(zm, a.eos)) zm = zc;
        rot_local(zm.u, zm.v, g.nx, g.ny);
        Cons lf = flux_from_p(zm);
        rot_global(lf.mu, lf.mv, g.nx, g.ny);
        add_area(F, lf, g.area);
    }
    update(q, 0.5 * dt / c.vol(), F);
    const Prim n = p_from_q(q, a.eos);
    if (!is_bad(n, a.eos)) h = n;
}

// is_bad without integer classification: comparisons with a NaN are false.
__device__ __forceinline__ bool bad(double r, double p, double e, double pmin) {
    return !(r > 0.0 && r < CUDART_INF && p >= pmin && p < CUDART_INF && fabs(e) < CUDART_INF);
}

template <int MODE, int TH>
struct Layout {
    static constexpr int H = 2;                               // halo of the staged state
    static constexpr int ZR = TH + 2 * H, ZC = 30 + 2 * H;    // staged rows and columns
    static constexpr int GR = TH + 2, NT = 32 * GR;           // cells with a face of the tile; the block
    static constexpr size_t al(size_t x) { return (x + 15) / 16 * 16; }
    static constexpr size_t z_bytes = al(sizeof(double) * 5 * ZR * ZC);
    static constexpr size_t f_bytes = al(sizeof(double) * 8 * (2 * TH + 1) * 32);
    // the predictor-corrector's faces read no staged state, so the fluxes
    // may overwrite it (the conserved state is taken from memory)
    static constexpr size_t off_f = MODE == PC ? 0 : z_bytes;
    static constexpr size_t off_v = MODE == PC ? (z_bytes > f_bytes ? z_bytes : f_bytes) : z_bytes + f_bytes;
    // values of a G cell at its low faces, x then y
    static constexpr size_t v_bytes = al(sizeof(double) * 10 * GR * 32);
    static constexpr size_t off_h = off_v + v_bytes;
    static constexpr size_t h_bytes = MODE == PC ? al(sizeof(double) * 5 * GR * 32) : 0;
    static constexpr size_t off_w = off_h + h_bytes;
    static constexpr size_t w_bytes = MODE == PC ? al(GR * 32) : 0;
    static constexpr size_t off_red = off_w + w_bytes;
    static constexpr size_t bytes = off_red + al(8 + 4 * GR);
};

// x wrapped into [0, n).
__device__ __forceinline__ int wrap(int x, int n) {
    if (x < 0) x += n;
    if (x >= n) x -= n;
    return x >= 0 && x < n ? x : (x % n + n) % n;
}

// One block's tile.  INTERIOR: the staged region lies inside the mesh, so the
// boundary selects and the wrapping drop out.
// (i0, j0): its first row and column.
template <int MODE, int LIM, bool HLL, int TH, bool INTERIOR>
__device__ __forceinline__ void tile(const Args &A, int i0, int j0) {
    using L = Layout<MODE, TH>;
    constexpr int ZR = L::ZR, ZC = L::ZC, GR = L::GR, NT = L::NT, HALO = L::H;
    extern __shared__ __align__(16) unsigned char smem[];
    double(*Z)[ZR][ZC] = reinterpret_cast<double(*)[ZR][ZC]>(smem);
    // face fluxes seen from the low cell (0-3) and the high cell (4-7): +x
    // faces of rows 0 .. TH, +y faces of rows 1 .. TH
    double(*FX)[TH + 1][32] = reinterpret_cast<double(*)[TH + 1][32]>(smem + L::off_f);
    double(*FY)[TH][32] = reinterpret_cast<double(*)[TH][32]>(smem + L::off_f + sizeof(double) * 8 * (TH + 1) * 32);
    double(*V)[GR][32] = reinterpret_cast<double(*)[GR][32]>(smem + L::off_v);
    double(*Hs)[GR][32] = reinterpret_cast<double(*)[GR][32]>(smem + L::off_h);
    unsigned char(*wt)[32] = reinterpret_cast<unsigned char(*)[32]>(smem + L::off_w);
    double *red = reinterpret_cast<double *>(smem + L::off_red);
    const SmfArgs &a = A.a;
    const StructMesh &m = a.mesh;
    const EosD &eos = a.eos;
    const int l = threadIdx.x, r = threadIdx.y, tid = r * 32 + l;

    // ---- stage the state ------------------------------------------------------
    if (INTERIOR) {
        const double *p0 = A.zin.r, *p1 = A.zin.u, *p2 = A.zin.v, *p3 = A.zin.p, *p4 = A.zin.e;
        for (int zr = r; zr < ZR; zr += GR) {
            int g = (i0 + zr - HALO) * m.ny + j0 - HALO + l;
#pragma unroll
            for (int zc = l; zc < ZC; zc += 32, g += 32) {
                Z[0][zr][zc] = p0[g];
                Z[1][zr][zc] = p1[g];
                Z[2][zr][zc] = p2[g];
                Z[3][zr][zc] = p3[g];
                Z[4][zr][zc] = p4[g];
            }
        }
    } else {
        for (int k = tid; k < ZR * ZC; k += NT) {
            const int zr = k / ZC, zc = k - zr * ZC;
            int gi = i0 + zr - HALO, gj = j0 + zc - HALO;
            // past a side without a neighbour any cell will do: it is not used
            gi = m.xper ? wrap(gi, m.nx) : min(max(gi, 0), m.nx - 1);
            gj = m.yper ? wrap(gj, m.ny) : min(max(gj, 0), m.ny - 1);
            const int g = gi * m.ny + gj;
            Z[0][zr][zc] = A.zin.r[g];
            Z[1][zr][zc] = A.zin.u[g];
            Z[2][zr][zc] = A.zin.v[g];
            Z[3][zr][zc] = A.zin.p[g];
            Z[4][zr][zc] = A.zin.e[g];
        }
    }
    if (tid == 0) red[0] = *A.dt_in / m.vol;
    __syncthreads();
    const double coef = red[0];

    // the thread's cell (r, l) of the G region: row i0 - 1 + r, column j0 - 1 + l
    const int iu = i0 - 1 + r, ju = j0 - 1 + l;
    const bool inx = INTERIOR || m.xper || (iu >= 0 && iu < m.nx), iny = INTERIOR || m.yper || (ju >= 0 && ju < m.ny);
    const int gi = INTERIOR || !m.xper ? iu : wrap(iu, m.nx), gj = INTERIOR || !m.yper ? ju : wrap(ju, m.ny);
    const int zr = r - 1 + HALO, zc = l - 1 + HALO;
    double xh[5] = {}, yh[5] = {};  // the cell's values at its high faces
    bool waiting = false;

    {
        // ---- limited gradients, half step, values at the four faces --------------
        double gx[4], gy[4], h[5];
        bool odd = false;
        if (inx && iny) {
            const bool bl = !INTERIOR && !m.xper && gi == 0, bh = !INTERIOR && !m.xper && gi == m.nx - 1;
            const bool bb = !INTERIOR && !m.yper && gj == 0, bt = !INTERIOR && !m.yper && gj == m.ny - 1;
            const double wl = A.x.wl[gi], rl = A.x.rl[gi], wh = A.x.wh[gi], rh = A.x.rh[gi];
            const double vl = A.y.wl[gj], sl = A.y.rl[gj], vh = A.y.wh[gj], sh = A.y.rh[gj];
            double B00, B11;
            {
                const double A00 = A.x.A[gi];
                double A11 = A.y.A[gj];
                if (fabs(A11) < 1e-8) A11 = 1.0;  // 1-D case (gradient.h:270-272)
                const double inv = 1.0 / (A11 * A00);
                B00 = A11 * inv;
                B11 = A00 * inv;
            }
            if (MODE == PC) waiting = a.wait_in[gi * m.ny + gj] > 0;
            double chk = 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double c = Z[q][zr][zc];
                // a boundary slot takes the reflected own value (sm_fluid.cpp:69-79)
                const double nL = bl ? (q == 1 && m.bc[0] == BC_WALL ? -c : c) : Z[q][zr - 1][zc];
                const double nR = bh ? (q == 1 && m.bc[1] == BC_WALL ? -c : c) : Z[q][zr + 1][zc];
                const double nB = bb ? (q == 2 && m.bc[2] == BC_WALL ? -c : c) : Z[q][zr][zc - 1];
                const double nT = bt ? (q == 2 && m.bc[3] == BC_WALL ? -c : c) : Z[q][zr][zc + 1];
                const double dL = nL - c, dR = nR - c, dB = nB - c, dT = nT - c;
                const double g0x = B00 * (wl * dL * rl + wh * dR * rh), g0y = B11 * (vl * dB * sl + vh * dT * sh);
                auto lim = [&](double g0, double rr, double dF) {
                    const double dFm = 2.0 * (g0 * rr) - dF;
                    return limiter2(LIM >= 0 ? LIM : a.limiter, dFm, dF) * dF;
                };
                gx[q] = B00 * (wl * lim(g0x, rl, dL) * rl + wh * lim(g0x, rh, dR) * rh);
                gy[q] = B11 * (vl * lim(g0y, sl, dB) * sl + vh * lim(g0y, sh, dT) * sh);
                chk += fabs(gx[q]) + fabs(gy[q]);
                h[q] = c;
            }
            h[4] = Z[4][zr][zc];
            odd = !(chk < CUDART_INF);
            if (MODE == PC && !waiting) {
                // predictor (sm_fluid.cpp:176-253)
                const Prim z{h[0], h[1], h[2], h[3], h[4]};
                const double mx = A.x.om[gi], my = A.y.om[gj];
                double F[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const double dx = s == 0 ? A.x.ol[gi] : (s == 1 ? A.x.oh[gi] : mx);
                    const double dy = s == 2 ? A.y.ol[gj] : (s == 3 ? A.y.oh[gj] : my);
                    double fr = z.r + (gx[0] * dx + gy[0] * dy), fu = z.u + (gx[1] * dx + gy[1] * dy);
                    double fv = z.v + (gx[2] * dx + gy[2] * dy), fp = z.p + (gx[3] * dx + gy[3] * dy);
                    double fe = eos.energy_rP(fr, fp);
                    if (bad(fr, fp, fe, eos.pmin)) fr = z.r, fu = z.u, fv = z.v, fp = z.p, fe = z.e;
                    const F4 f = s < 2 ? flux_n(fr, fu, fv, fp, fe) : flux_n(fr, fv, fu, fp, fe);
                    const double w = (s & 1) ? (s < 2 ? m.hy : m.hx) : -(s < 2 ? m.hy : m.hx);
                    F[0] += f.r * w;
                    F[1] += (s < 2 ? f.n : f.t) * w;
                    F[2] += (s < 2 ? f.t : f.n) * w;
                    F[3] += f.E * w;
                }
                Cons q = q_from_p(z);
                update(q, 0.5 * coef, Cons{F[0], F[1], F[2], F[3]});
                const Prim n = p_from_q(q, eos);
                if (!bad(n.r, n.p, n.e, eos.pmin)) h[0] = n.r, h[1] = n.u, h[2] = n.v, h[3] = n.p, h[4] = n.e;
            }
        }
        if (__syncthreads_or(odd)) {  // (the staged state is read above, and overwritten below)
            if (odd) {
                Prim hp{};
                odd_cell(a, A.zin, gi * m.ny + gj, MODE != PC || waiting, *A.dt_in, gx, gy, hp);
                h[0] = hp.r, h[1] = hp.u, h[2] = hp.v, h[3] = hp.p, h[4] = hp.e;
            }
        }
        if (inx && iny) {
            if (MODE == PC) {
                wt[r][l] = waiting;
#pragma unroll
                for (int q = 0; q < 5; ++q) Hs[q][r][l] = h[q];
            }
            // past a periodic seam the offset from the mirrored centre
            const double oxl = !INTERIOR && iu >= m.nx ? A.x.seam_hi : A.x.ol[gi];
            const double oxh = !INTERIOR && iu < 0 ? A.x.seam_lo : A.x.oh[gi];
            const double oyl = !INTERIOR && ju >= m.ny ? A.y.seam_hi : A.y.ol[gj];
            const double oyh = !INTERIOR && ju < 0 ? A.y.seam_lo : A.y.oh[gj];
            const double mx = A.x.om[gi], my = A.y.om[gj];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const double dx = s == 0 ? oxl : (s == 1 ? oxh : mx), dy = s == 2 ? oyl : (s == 3 ? oyh : my);
                double o[5];
#pragma unroll
                for (int q = 0; q < 4; ++q) o[q] = h[q] + (gx[q] * dx + gy[q] * dy);
                o[4] = eos.energy_rP(o[0], o[3]);
                if (bad(o[0], o[3], o[4], eos.pmin)) {
#pragma unroll
                    for (int q = 0; q < 5; ++q) o[q] = h[q];
                }
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    if (s == 0) V[q][r][l] = o[q];
                    else if (s == 1) xh[q] = o[q];
                    else if (s == 2) V[5 + q][r][l] = o[q];
                    else yh[q] = o[q];
                }
            }
        }
        __syncthreads();
    }

    // ---- the faces of the tile's cells, each once --------------------------------
    // the face's two states in axis directions; false: no face of a cell
    auto states = [&](auto axc, FState &a_, FState &b_, bool &robust) {
        constexpr int AX = decltype(axc)::value;
        const int r2 = r + (AX == 0), l2 = l + (AX == 1);
        // the low cell's row / column along the axis, and the mesh's extent
        const int ua = AX == 0 ? iu : ju, n = AX == 0 ? m.nx : m.ny;
        const bool per = INTERIOR || (AX == 0 ? m.xper : m.yper);
        const bool inA = per || ua >= 0, inB = per || ua + 1 < n;
        double va[5], vb[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            va[q] = AX == 0 ? xh[q] : yh[q];
            vb[q] = V[5 * AX + q][r2][l2];
        }
        robust = MODE == PC && ((inA && waiting) || (inB && wt[r2][l2]));
        if (robust) {  // isolated cells: without reconstruction
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                if (inA) va[q] = Hs[q][r][l];
                if (inB) vb[q] = Hs[q][r2][l2];
            }
        }
        a_ = AX == 0 ? FState{va[0], va[1], va[2], va[3], va[4]} : FState{va[0], va[2], va[1], va[3], va[4]};
        b_ = AX == 0 ? FState{vb[0], vb[1], vb[2], vb[3], vb[4]} : FState{vb[0], vb[2], vb[1], vb[3], vb[4]};
        if (!inA) {  // the mirror of the only cell's value (sm_fluid.cpp:69-79)
            a_ = b_;
            if (m.bc[2 * AX] == BC_WALL) a_.n = -a_.n;
        }
        if (!inB) {
            b_ = a_;
            if (m.bc[2 * AX + 1] == BC_WALL) b_.n = -b_.n;
        }
    };
    // (a face outside the mesh on the other axis, or past both ends of its
    // own, belongs to no cell)
    const bool fx = r <= TH && l >= 1 && l <= 30 && iny && (INTERIOR || iu < m.nx);
    const bool fy = r >= 1 && r <= TH && l <= 30 && inx && (INTERIOR || ju < m.ny);
    auto put_x = [&](int view, const F4 &f) {
        FX[4 * view][r][l] = f.r;
        FX[4 * view + 1][r][l] = f.n;
        FX[4 * view + 2][r][l] = f.t;
        FX[4 * view + 3][r][l] = f.E;
    };
    auto put_y = [&](int view, const F4 &f) {
        FY[4 * view][r - 1][l] = f.r;
        FY[4 * view + 1][r - 1][l] = f.t;
        FY[4 * view + 2][r - 1][l] = f.n;
        FY[4 * view + 3][r - 1][l] = f.E;
    };
    auto both = [&](const FState &a_, const FState &b_, bool robust, auto &&put) {
        if (HLL || robust) return hll_both(a_, b_, eos, put);
        return hllc_both(a_, b_, eos, put);
    };
    bool odd_x = false, odd_y = false;
    if (fx) {
        FState a_, b_;
        bool robust;
        states(std::integral_constant<int, 0>{}, a_, b_, robust);
        odd_x = !both(a_, b_, robust, put_x);
    }
    if (fy) {
        FState a_, b_;
        bool robust;
        states(std::integral_constant<int, 1>{}, a_, b_, robust);
        odd_y = !both(a_, b_, robust, put_y);
    }
    if (__syncthreads_or(odd_x || odd_y)) {
        FState a_, b_;
        F4 lo, hi;
        bool robust;
        if (odd_x) {
            states(std::integral_constant<int, 0>{}, a_, b_, robust);
            odd_face(a_, b_, 0, HLL || robust, eos, lo, hi);
            put_x(0, lo);
            put_x(1, hi);
        }
        if (odd_y) {
            states(std::integral_constant<int, 1>{}, a_, b_, robust);
            odd_face(a_, b_, 1, HLL || robust, eos, lo, hi);
            put_y(0, lo);
            put_y(1, hi);
        }
        __syncthreads();
    }

    // ---- update --------------------------------------------------------------------
    float low = INFINITY;  // lower bound of the cell's CFL term (0: none; infinite: no cell)
    Prim n{};
    const bool mine = r >= 1 && r <= TH && l >= 1 && l <= 30 && (INTERIOR || (iu < m.nx && ju < m.ny));
    if (mine) {
        const int ic = iu * m.ny + ju;
        double F[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            F[q] = ((0.0 - FX[4 + q][r - 1][l] * m.hy) + FX[q][r][l] * m.hy - FY[4 + q][r - 1][l - 1] * m.hx) +
                   FY[q][r - 1][l] * m.hx;
        Prim zo;
        if constexpr (MODE == PC) zo = load_prim(a.z, ic);
        else zo = Prim{Z[0][zr][zc], Z[1][zr][zc], Z[2][zr][zc], Z[3][zr][zc], Z[4][zr][zc]};
        Cons q = q_from_p(zo);
        update(q, coef, Cons{F[0], F[1], F[2], F[3]});
        if (MODE == HEUN_B) {
            const Cons q0 = q_from_p(load_prim(a.z, ic));
            q.r = 0.5 * (q0.r + q.r);
            q.mu = 0.5 * (q0.mu + q.mu);
            q.mv = 0.5 * (q0.mv + q.mv);
            q.E = 0.5 * (q0.E + q.E);
        }
        n = p_from_q(q, eos);
        if (MODE == PC) {
            int wn = a.wait_in[ic];
            if (bad(n.r, n.p, n.e, eos.pmin)) {
                n = zo;
                wn = 3;
            } else if (wn > 0) {
                --wn;
            }
            a.wait_out[ic] = wn;
        }
        store_prim(A.zout, ic, n);
        if (MODE != HEUN_A) {
            // lower bound of incircle / (|v| + c) in FP32, 2e-4 too small; 0
            // where FP32 cannot hold the squares, or for a NaN
            const float d = sqrtf((float)m.inc2min);
            const float c2 = __fdividef((float)(eos.gamma * (n.p + eos.P0)), (float)n.r);
            const float s = sqrtf(c2) + sqrtf((float)(n.u * n.u + n.v * n.v));
            const bool ok = d > 1e-15f && d < 1e15f && s > 1e-10f && s < 1e15f && n.r > 1e-30 && n.r < 1e30;
            low = ok ? __fdividef(d, s) * 0.9998f : 0.0f;
        }
    }
    if (MODE == HEUN_A || !A.dt_next) return;
    // The next step's dt (compute_dt, sm_fluid.cpp:104-116), k_dt's arithmetic;
    // the term is formed only where its lower bound does not exceed the
    // block's smallest (1.0005: a bound is at most 3e-4 below its term).
    float w = low > 0.0f ? low : INFINITY;
    for (int o = 16; o > 0; o >>= 1) w = fminf(w, __shfl_xor_sync(0xffffffffu, w, o));
    float *redf = reinterpret_cast<float *>(red + 1);
    if (l == 0) redf[r] = w;
    __syncthreads();
    float lim = redf[l < GR ? l : 0];
    for (int o = 16; o > 0; o >>= 1) lim = fminf(lim, __shfl_xor_sync(0xffffffffu, lim, o));
    const bool take = mine && low <= lim * 1.0005f;
    if (__any_sync(0xffffffffu, take)) {
        unsigned long long best = 0x7FEFFFFFFFFFFFFFull;
        if (take) best = cfl_bits(a, sqrt(smin(m.inc2x[iu], m.inc2y[ju])), n.r, n.u, n.v, n.p);
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
            best = t < best ? t : best;
        }
        if (l == 0) {
            atomicMin(a.dmin_bits, best);
            __threadfence();
        }
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        const unsigned int ticket = atomicAdd(a.dt_ticket, 1u);
        if (ticket == gridDim.x * (unsigned)((m.nx + TH - 1) / TH) - 1) {  // no block waits for another
            const unsigned long long bits = atomicMin(a.dmin_bits, 0x7FEFFFFFFFFFFFFFull);
            *A.dt_next = smin(a.CFL * __longlong_as_double((long long)bits), a.max_dt);
            *a.dmin_bits = 0x7FEFFFFFFFFFFFFFull;
            *a.dt_ticket = 0u;
            __threadfence();
        }
    }
}

template <int MODE, int LIM, bool HLL, int TH, int MINB>
__global__ void __launch_bounds__(32 * (TH + 2), MINB) k_tile(const __grid_constant__ Args A) {
    after_previous();
    constexpr int H = Layout<MODE, TH>::H;
    const int i0 = (blockIdx.z * gridDim.y + blockIdx.y) * TH, j0 = blockIdx.x * 30;
    if (i0 >= A.a.mesh.nx) return;
    // (a limiter chosen at run time: one copy of its code)
    if constexpr (LIM >= 0) {
        if (i0 >= H && i0 + TH + H <= A.a.mesh.nx && j0 >= H && j0 + 30 + H <= A.a.mesh.ny) {
            tile<MODE, LIM, HLL, TH, true>(A, i0, j0);
            return;
        }
    }
    tile<MODE, LIM, HLL, TH, false>(A, i0, j0);
}

template <int MODE, int LIM, bool HLL, int TH, int MINB>
inline void launch(const Args &A, cudaStream_t s) {
    using L = Layout<MODE, TH>;
    static unsigned long long attr_set = 0;  // devices on which the attribute is set
    auto kern = k_tile<MODE, LIM, HLL, TH, MINB>;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 64 || !(attr_set >> dev & 1ull)) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::bytes);
        if (dev < 64) attr_set |= 1ull << dev;
    }
    const StructMesh &m = A.a.mesh;
    launch_after(kern, row_grid((m.ny + 29) / 30, (m.nx + TH - 1) / TH), dim3(32, TH + 2), L::bytes, s, A);
}

}  // namespace ptile
}  // namespace zg
