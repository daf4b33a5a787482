// smf_fused.cuh -- the whole second-order step of a structured rectangle in
// ONE kernel per stage: limited gradients, predictor, face-once corrector,
// update and the next step's CFL minimum, for a tile of cells held in shared
// memory.  Nothing but the state (and the isolation counters) crosses HBM:
// the gradients and the half-step state of the two-pass form (smf_tiled.cuh
// k_grad_predict -> k_faces) never leave the SM.
//
// Scheme: math/solver/sm_fluid.cpp:81-102 (compute_grad 116-125, fluxes_stage1
// 176-253, fluxes_stage2 255-366) in the precisions of the two-pass tiled
// kernels (FAST: FP64; MIXED: FP32 primitive states, gradients and fluxes
// with FP64 conserved sums, update, pressure recovery and dt).  The rectangle
// is uniform, so the least-squares geometry of gradient.h:226-282 reduces to
// per-axis constants: with cell size h along an axis and the differences
// dL = z_low - z, dR = z_high - z to the two neighbours (a boundary slot takes
// the reflected own value, sm_fluid.cpp:69-79), the unlimited slope is
// (dR - dL) / 2h, and the limited refit of gradient.h:412-474 becomes
//     g = (phi(-dL, dR) dR - phi(-dR, dL) dL) / 2h,
// because 2 g0 (dr . n) - dF equals -dR on the low face and -dL on the high
// one.  For van Albada 1 (limiter.cxx:69-82) both limiter values vanish
// unless dL dR < 0, and then g = -dL dR (dR - dL) / ((dL^2 + dR^2) h): one
// division per component instead of two.  Face centres sit at +-h/2 along
// the face normal.  These are the reference's formulas up to the rounding of
// the mesh coordinates, far inside the FAST form's 1e-12 per-step bound.
//
// Tile geometry (block = 32 x (TH + 2) threads, thread (l, r)):
//   interior cells  rows i0 .. i0 + TH - 1, columns j0 .. j0 + 29   (30 x TH)
//   G region        rows i0 - 1 .. i0 + TH, columns j0 - 1 .. j0 + 30: one
//                   cell per thread; gradients (and the half step) of every
//                   cell whose face touches an interior cell
//   Z region        rows i0 - 2 .. i0 + TH + 1, columns j0 - 2 .. j0 + 31:
//                   the state the G region's gradients read
// Phases, separated by block barriers:
//   0  stage Z from HBM (wrapped on periodic axes)
//   1  per G cell: limited gradient, for the predictor-corrector also the
//      half step (physical flux of the cell's own face values)
//   2  per thread: the +x face (G rows r | r + 1) and the +y face (G columns
//      l | l + 1) that bound an interior cell, each computed once
//   3  per interior cell: flux sum in the reference's slot order, update,
//      pressure recovery, isolation counters, CFL term, block minimum
#pragma once

#include <type_traits>

#include "smf_tiled.cuh"

namespace zg {
namespace tiled {

// Stage of the fused kernel.
enum : int { FUSED_PC = 1, FUSED_HEUN_A = 2, FUSED_HEUN_B = 3 };

// ---------------------------------------------------------------------------
// Reciprocals.  FP64: Newton-Raphson iteration for 1/x (y <- y + y (1 - x y),
// each step doubling the correct bits; e.g. P. Markstein, IBM J. Res. Dev.
// 34(1), 1990) from the hardware's approximate reciprocal (PTX
// rcp.approx.ftz.f64), two steps; within 2 ulp of 1/x for normal finite x.
// FP32 (MIXED, compiled with approximate division): 1 / x.
__device__ __forceinline__ double rcp_nr(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double e = fma(-x, y, 1.0);
    y = fma(y, e, y);
    e = fma(-x, y, 1.0);
    return fma(y, e, y);
}
__device__ __forceinline__ float rcp_r(float x) { return 1.0f / x; }
__device__ __forceinline__ double rcp_r(double x) { return rcp_nr(x); }

// A face state with its reciprocal density.
template <typename R>
struct FS {
    R r, u, v, p, e, ri;
};

// half: at the half step's faces
template <typename R>
__device__ __forceinline__ R energy_ri(const EosR<R> &eos, R P, R ri, R igm1, bool half = false) {
    if (eos.kind == EOS_IDEAL) return rmul(rmul(P, ri), igm1);
    const R s = half ? radd(P, rmul(eos.gamma, eos.P0)) : rfma(eos.gamma, eos.P0, P);
    return rfma(rmul(s, ri), igm1, eos.e0);
}

// models.cpp:58-63 (is_bad) without integer classification: every compare
// with a NaN is false, and the infinities fail the range tests.
template <typename R>
__device__ __forceinline__ bool bad_fs(const FS<R> &z, R pmin) {
    const R inf = R(INFINITY);
    const bool ok = z.r > R(0) && z.r < inf && z.p >= pmin && z.p < inf && z.e > -inf && z.e < inf;
    return !ok;
}

// is_bad of a reconstructed FP64 state (models.cpp:58-63): r and p finite, r
// positive, p not below the EoS's minimum; e = O(p / r) is then finite unless
// r is below p by the whole exponent range.
__device__ __forceinline__ bool bad_rp(double r, double p, double pmin) {
    return !(r > fabs(p) * 0x1p-997 && p >= pmin && fabs(r + p) < INFINITY);
}
template <typename R>
__device__ __forceinline__ bool bad_value(const FS<R> &z, R pmin) {
    if constexpr (sizeof(R) == 8) return bad_rp(z.r, z.p, pmin);
    else return bad_fs(z, pmin);
}

// phys flux along x of z (models.cpp:131-137 with the normal (1, 0))
// (k = |v|^2)
template <typename R>
__device__ __forceinline__ C4<R> flux_x(const FS<R> &z, R k) {
    const R ru = rmul(z.r, z.u), E = rfma(R(0.5), k, z.e);
    return C4<R>{ru, rfma(ru, z.u, z.p), rmul(ru, z.v), rmul(rfma(z.r, E, z.p), z.u)};
}
template <typename R>
__device__ __forceinline__ C4<R> flux_x(const FS<R> &z) {
    return flux_x(z, sq2(z.u, z.v));
}
template <typename R>
__device__ __forceinline__ R sound_ri(const FS<R> &z, const EosR<R> &eos) {
    return sqrt(rmul(rmul(eos.gamma, radd(z.p, eos.P0)), z.ri));
}

// HLLC (hllc.cpp:23-83) in the face frame.  hllc.cpp writes the flux in its
// symmetric form 1/2 (F_L + F_R + S_L (Q*_L - Q_L) + |S_C| (Q*_L - Q*_R) +
// S_R (Q*_R - Q_R)); through the Rankine-Hugoniot relations that define the
// star states this is the star flux on the side of the contact the face
// lies on: F_L + S_L (Q*_L - Q_L) for S_C >= 0, F_R + S_R (Q*_R - Q_R)
// otherwise.  The kernel evaluates that one side (the two forms agree to
// rounding), with the side's state chosen before the arithmetic so that a
// warp runs one path.
// VL, VR: |v|^2 of the left / right state as v^2 + u^2 (see hll_fs).
template <bool VL, bool VR, typename R>
__device__ __forceinline__ C4<R> hllc_fs(const FS<R> &L, const FS<R> &Rs, const EosR<R> &eos) {
    const R cL = sound_ri(L, eos), cR = sound_ri(Rs, eos);
    // (the states are finite here: a NaN ordering of std::min does not arise)
    const R SL = smin_t(rsub(L.u, cL), rsub(Rs.u, cR));
    const R SR = smax_t(radd(L.u, cL), radd(Rs.u, cR));
    if (SL >= R(0)) return flux_x(L, VL ? sq2(L.v, L.u) : sq2(L.u, L.v));
    if (SR <= R(0)) return flux_x(Rs, VR ? sq2(Rs.v, Rs.u) : sq2(Rs.u, Rs.v));
    const R aL = rmul(L.r, rsub(SL, L.u)), aR = rmul(Rs.r, rsub(SR, Rs.u));
    const R SC = rmul(rfma(-aL, L.u, rfma(aR, Rs.u, rsub(L.p, Rs.p))), rcp_r(rsub(aR, aL)));
    const bool left = SC >= R(0);
    FS<R> X;
    X.r = left ? L.r : Rs.r;
    X.u = left ? L.u : Rs.u;
    X.v = left ? L.v : Rs.v;
    X.p = left ? L.p : Rs.p;
    X.e = left ? L.e : Rs.e;
    const R SX = left ? SL : SR, aX = left ? aL : aR;
    const R rs = rmul(aX, rcp_r(rsub(SX, SC)));
    const R EX = rfma(R(0.5), sq2(X.u, X.v), X.e);
    const R Es = rfma(rsub(SC, X.u), rfma(X.p, rcp_r(aX), SC), EX);
    const R ru = rmul(X.r, X.u);
    const R rE = rmul(X.r, EX);
    C4<R> f;
    f.r = rfma(SX, rsub(rs, X.r), ru);
    f.mu = rfma(SX, rfma(rs, SC, -ru), rfma(ru, X.u, X.p));
    f.mv = rfma(ru, X.v, rmul(SX, rfma(rs, X.v, -rmul(X.r, X.v))));
    f.E = rfma(radd(rE, X.p), X.u, rmul(SX, rfma(rs, Es, -rE)));
    return f;
}

// The FP64 form of hllc_fs, in the marching kernel and in the tiles alike: the
// supersonic cases as a choice of the upwind side instead of early returns.
// VOTE: all lanes of the warp call it, and a warp without a subsonic face
// leaves the star state out.
template <bool VOTE>
__device__ __forceinline__ C4<double> hllc_d(const FS<double> &L, const FS<double> &Rs, const EosR<double> &eos) {
    const double cL = sound_ri(L, eos), cR = sound_ri(Rs, eos);
    // (no sum of a product among these: plain operators round the same, and leave
    // the compiler 1.3 % of a 2048^2 step)
    const double SL = smin_t(L.u - cL, Rs.u - cR), SR = smax_t(L.u + cL, Rs.u + cR);
    const double aL = L.r * (SL - L.u), aR = Rs.r * (SR - Rs.u);
    const double SC = rmul(rfma(-aL, L.u, rfma(aR, Rs.u, rsub(L.p, Rs.p))), rcp_nr(rsub(aR, aL)));
    const bool subsonic = SL < 0.0 && SR > 0.0;
    const bool left = subsonic ? SC >= 0.0 : SL >= 0.0;
    const double r = left ? L.r : Rs.r, u = left ? L.u : Rs.u, v = left ? L.v : Rs.v, p = left ? L.p : Rs.p;
    const double e = left ? L.e : Rs.e;
    const double ru = rmul(r, u), EX = rfma(0.5, sq2(u, v), e), rE = rmul(r, EX);
    C4<double> f{ru, rfma(ru, u, p), rmul(ru, v), rmul(radd(rE, p), u)};
    if (VOTE ? __any_sync(0xffffffffu, subsonic) : subsonic) {
        const double SX = left ? SL : SR, aX = left ? aL : aR;
        const double rs = rmul(aX, rcp_nr(rsub(SX, SC)));
        const double Es = rfma(rsub(SC, u), rfma(p, rcp_nr(aX), SC), EX);
        if (subsonic) {
            f.r = rfma(SX, rsub(rs, r), f.r);
            f.mu = rfma(SX, rfma(rs, SC, -ru), f.mu);
            f.mv = rfma(SX, rfma(rs, v, -rmul(r, v)), f.mv);
            f.E = rfma(SX, rfma(rs, Es, -rE), f.E);
        }
    }
    return f;
}

// HLL (hll.cpp:23-57) in the face frame (isolated cells, and the HLL method).
// VL, VR: |v|^2 of the left / right state as v^2 + u^2; Y: a y face's frame.
// Interior faces: VR = Y, VL = Y or Heun's first stage; boundary faces: both.
template <bool VL, bool VR, bool Y, typename R>
__device__ __forceinline__ C4<R> hll_fs(const FS<R> &L, const FS<R> &Rs, const EosR<R> &eos) {
    const R cL = sound_ri(L, eos), cR = sound_ri(Rs, eos);
    const R SL = smin_t(smin_t(rsub(L.u, cL), rsub(Rs.u, cR)), R(0));
    const R SR = smax_t(smax_t(radd(L.u, cL), radd(Rs.u, cR)), R(0));
    const R EL = rfma(R(0.5), VL ? sq2(L.v, L.u) : sq2(L.u, L.v), L.e);
    const R ER = rfma(R(0.5), VR ? sq2(Rs.v, Rs.u) : sq2(Rs.u, Rs.v), Rs.e);
    const R ruL = rmul(L.r, L.u), ruR = rmul(Rs.r, Rs.u), rvL = rmul(L.r, L.v), rvR = rmul(Rs.r, Rs.v);
    const R inv = rcp_r(rsub(SR, SL)), SLR = rmul(SL, SR);
    auto mean = [&](R fl, R fr, R dq) { return rmul(rfma(SLR, dq, rfma(SR, fl, -rmul(SL, fr))), inv); };
    C4<R> o;
    o.r = mean(ruL, ruR, rsub(Rs.r, L.r));
    o.mu = mean(rfma(ruL, L.u, L.p), rfma(ruR, Rs.u, Rs.p), rsub(ruR, ruL));
    o.mv = mean(rmul(ruL, L.v), rmul(ruR, Rs.v), Y ? rfma(-L.r, L.v, rvR) : rfma(Rs.r, Rs.v, -rvL));
    o.E = mean(rmul(rfma(L.r, EL, L.p), L.u), rmul(rfma(Rs.r, ER, Rs.p), Rs.u), rfma(Rs.r, ER, -rmul(L.r, EL)));
    return o;
}

// Limited slope of one component along one axis (see the header comment);
// inv2h = 1 / 2h, invh = 1 / h.
// A limiter chosen at run time is out of line: sixteen inlined copies of the
// switch outgrow the instruction cache (superbee 2nd order at 1400^2: 307 -> 219
// us a step).
template <typename R>
__device__ __noinline__ R limit_rt(int kind, R a, R b) {
    return lim2<R>(kind, a, b);
}
template <int LIM, typename R>
__device__ __forceinline__ R slope(int kind, R dL, R dR, R inv2h, R invh) {
    if (LIM == LIM_VANALBADA1) {
        const R p = rmul(dL, dR);
        if (p >= R(0)) return R(0);
        return rmul(rmul(rmul(-p, rsub(dR, dL)), rcp_r(sq2(dL, dR))), invh);
    }
    R a, b;
    if (LIM >= 0) {
        a = lim2<R>(LIM, -dL, dR);
        b = lim2<R>(LIM, -dR, dL);
    } else {
        a = limit_rt<R>(kind, -dL, dR);
        // van Albada 2 is symmetric in its arguments: one value (and one rounding) for both
        b = kind == LIM_VANALBADA2 ? a : limit_rt<R>(kind, -dR, dL);
    }
    if (LIM == LIM_MC || LIM == LIM_MINMOD) return rmul(rfma(-b, dL, rmul(a, dR)), inv2h);
    return rmul(rfma(a, dR, -rmul(b, dL)), inv2h);
}

// A cell's value at the face at `off` along an axis (FaceExtra::Direct,
// face_extra.h:121-184) with slopes g0-g3; low: an interior face on
// the cell's low side.
// The energy and 1 / r are the caller's.
template <typename R>
__device__ __forceinline__ FS<R> reconstruct(const FS<R> &z, R g0, R g1, R g2, R g3, R off, bool low) {
    const bool two = sizeof(R) == 4 && low;
    return FS<R>{rfma(g0, off, z.r), two ? radd(z.u, rmul(g1, off)) : rfma(g1, off, z.u),
                 two ? radd(z.v, rmul(g2, off)) : rfma(g2, off, z.v), rfma(g3, off, z.p), R(0), R(0)};
}
// Physical flux along an axis (ax: x) of a cell's value at its own face, for the
// half step (sm_fluid.cpp:176-253); the cell's own value where that is bad.
// rarely(bad, fix): runs fix where bad.
template <typename R, typename F>
__device__ __forceinline__ C4<R> half_flux(const FS<R> &c, const R g[4], R off, bool ax, const EosR<R> &eos, R igm1,
                                           F &&rarely) {
    if constexpr (sizeof(R) == 8) {
        // r e = (p + gamma P0) / (gamma - 1) + r e0: no reciprocal density
        double r = rfma(g[0], off, c.r), u = rfma(g[1], off, c.u), v = rfma(g[2], off, c.v), p = rfma(g[3], off, c.p);
        double re = rfma(rfma(eos.gamma, eos.P0, p), igm1, rmul(r, eos.e0));
        rarely(bad_rp(r, p, eos.pmin), [&] {
            r = c.r, u = c.u, v = c.v, p = c.p;
            re = rmul(r, c.e);
        });
        const double n = ax ? u : v, rn = rmul(r, n), E = rfma(rmul(0.5, r), sq2(u, v), re);
        return C4<R>{rn, ax ? rfma(rn, u, p) : rmul(rn, u), ax ? rmul(rn, v) : rfma(rn, v, p), rmul(radd(E, p), n)};
    } else {
        FS<R> zm{radd(c.r, rmul(g[0], off)), rfma(g[1], off, c.u), rfma(g[2], off, c.v), radd(c.p, rmul(g[3], off)),
                 R(0), R(0)};
        zm.ri = rcp_r(zm.r);
        zm.e = energy_ri(eos, zm.p, zm.ri, igm1, true);
        rarely(bad_fs(zm, eos.pmin), [&] { zm = c; });
        if (ax) return flux_x(zm);
        // flux along y: swap the velocity components
        const C4<R> t = flux_x(FS<R>{zm.r, zm.v, zm.u, zm.p, zm.e, zm.ri});
        return C4<R>{t.r, t.mv, t.mu, t.E};
    }
}
// F += f w, and q -= k F
template <typename R>
__device__ __forceinline__ void add_half(double F[4], const C4<R> &f, double w) {
    F[0] = rfma((double)f.r, w, F[0]);
    F[1] = rfma((double)f.mu, w, F[1]);
    F[2] = rfma((double)f.mv, w, F[2]);
    F[3] = rfma((double)f.E, w, F[3]);
}
__device__ __forceinline__ void subtract(C4<double> &q, double k, const double F[4]) {
    q.r = rfma(-k, F[0], q.r);
    q.mu = rfma(-k, F[1], q.mu);
    q.mv = rfma(-k, F[2], q.mv);
    q.E = rfma(-k, F[3], q.E);
}

// A cell's outward flux sum from its faces' fluxes (low x, high x, low y, high
// y): MIXED in the slots' order; FP64 with the high x face last, which the march
// has last.
__device__ __forceinline__ double flux_sum(double xl, double xh, double yl, double yh, double hx, double hy) {
    return rfma(yh, hx, rfma(-yl, hx, rfma(xh, hy, -rmul(xl, hy))));
}
__device__ __forceinline__ double three_fluxes(double xl, double yl, double yh, double hx, double hy) {
    return rfma(yh, hx, rfma(-yl, hx, -rmul(xl, hy)));
}

// Conserved variables of an FP64 primitive state (models.cpp:20-25).
__device__ __forceinline__ C4<double> cons_of(double r, double u, double v, double e) {
    return C4<double>{r, r * u, r * v, r * rfma(0.5, sq2(u, v), e)};
}

// The same less k F.
__device__ __forceinline__ C4<double> cons_less(double r, double u, double v, double e, double k, const double F[4]) {
    return C4<double>{rfma(-k, F[0], r), rfma(r, u, -rmul(k, F[1])), rfma(r, v, -rmul(k, F[2])),
                      rfma(r, rfma(0.5, sq2(u, v), e), -rmul(k, F[3]))};
}

// Conserved state of cell ic at t^n.
template <typename R, bool MIXED>
__device__ __forceinline__ C4<double> q_n(const Fields<R> &f, int ic) {
    if (MIXED) return C4<double>{f.q[0][ic], f.q[1][ic], f.q[2][ic], f.q[3][ic]};
    return cons_of(f.w[0][ic], f.w[1][ic], f.w[2][ic], f.w[4][ic]);
}

// FP64 primitive state from conserved variables (models.cpp:27-32) with the
// reciprocal density kept for the sound speed.
__device__ __forceinline__ P5<double> prim_ri(const C4<double> &q, const EosD &eos, double &ri) {
    P5<double> z;
    z.r = q.r;
    ri = rcp_nr(q.r);
    z.u = q.mu * ri;
    z.v = q.mv * ri;
    z.e = rfma(q.E, ri, -0.5 * sq2(z.u, z.v));
    z.p = eos.kind == EOS_IDEAL ? eos.gm1 * z.r * z.e
                                : rfma(eos.gm1 * z.r, z.e - eos.e0, -rmul(eos.gamma, eos.P0));
    return z;
}

template <bool VL, bool VR, typename R>
__device__ __forceinline__ C4<R> hllc_any(const FS<R> &L, const FS<R> &Rs, const EosR<R> &eos) {
    if constexpr (sizeof(R) == 8) return hllc_d<false>(L, Rs, eos);
    else return hllc_fs<VL, VR>(L, Rs, eos);
}

// Flux across a boundary face (WALL / ZOE, sm_fluid.cpp:69-79) from the
// reconstructed state zm of its only cell, whose slot s_own it is: the ghost
// state reflects the normal velocity at a wall; the flux is returned in the
// +x / +y direction.  FP64: in that direction's frame, as the march has it.
// MIXED: in the frame of the cell's outward normal.  Out of line: boundary
// faces are few, and one copy of the Riemann solver serves all of them.
template <bool FIRST, typename R>
__device__ __noinline__ C4<R> boundary_flux(FS<R> zm, int s_own, int bc, bool use_hll, EosR<R> eos, bool own_a) {
    FS<R> zp = zm;
    if (bc == BC_WALL) {
        if (s_own < 2) zp.u = -zp.u;
        else zp.v = -zp.v;
    }
    if constexpr (sizeof(R) == 8) {
        if (!own_a) {
            const FS<R> t = zm;
            zm = zp;
            zp = t;
        }
        const int s = s_own | 1;  // the high slot of the axis: the + direction
        to_local(s, zm.u, zm.v);
        to_local(s, zp.u, zp.v);
        C4<R> lf;
        if (!use_hll) lf = hllc_any<true, true>(zm, zp, eos);
        else if (s == 1) lf = hll_fs<FIRST, false, false>(zm, zp, eos);
        else lf = hll_fs<true, true, true>(zm, zp, eos);
        to_global(s, lf.mu, lf.mv);
        return lf;
    }
    to_local(s_own, zm.u, zm.v);
    to_local(s_own, zp.u, zp.v);
    C4<R> lf = use_hll ? hll_fs<true, true, false>(zm, zp, eos) : hllc_any<true, true>(zm, zp, eos);
    to_global(s_own, lf.mu, lf.mv);
    if (!own_a) {
        lf.r = -lf.r;
        lf.mu = -lf.mu;
        lf.mv = -lf.mv;
        lf.E = -lf.E;
    }
    return lf;
}

template <typename R, int TH, int MODE>
struct FusedLayout {
    static constexpr int ZR = TH + 4, ZC = 34;  // Z region
    static constexpr int GR = TH + 2, GC = 32;  // G region (= the block)
    static constexpr int NT = 32 * GR;
    static constexpr bool PC = MODE == FUSED_PC;
    static constexpr size_t al(size_t x) { return (x + 15) / 16 * 16; }
    static constexpr size_t z_bytes = al(sizeof(R) * 5 * ZR * ZC);
    // face fluxes (widened to FP64 once, where they are computed): +x faces
    // of G rows 0..TH, +y faces of G rows 1..TH
    static constexpr size_t fx_bytes = al(sizeof(double) * 4 * (TH + 1) * GC);
    static constexpr size_t fy_bytes = al(sizeof(double) * 4 * TH * GC);
    // The predictor-corrector reads only the G region after phase 1, so the
    // fluxes may overwrite Z; the Heun stages reconstruct from Z itself.
    static constexpr size_t off_z = 0;
    static constexpr size_t off_fx = PC ? 0 : z_bytes;
    static constexpr size_t off_fy = off_fx + fx_bytes;
    static constexpr size_t zf_end = PC ? (z_bytes > fx_bytes + fy_bytes ? z_bytes : fx_bytes + fy_bytes)
                                        : z_bytes + fx_bytes + fy_bytes;
    static constexpr size_t off_g = zf_end;
    static constexpr size_t g_bytes = al(sizeof(R) * 8 * GR * GC);
    static constexpr size_t off_h = off_g + g_bytes;
    static constexpr size_t h_bytes = PC ? al(sizeof(R) * 5 * GR * GC) : 0;
    // conserved state at t^n of the G cells (predictor-corrector)
    static constexpr size_t off_q = off_h + h_bytes;
    static constexpr size_t q_bytes = PC ? al(sizeof(double) * 4 * GR * GC) : 0;
    static constexpr size_t off_zin = off_q + q_bytes;
    static constexpr size_t zin_bytes = al(ZR * ZC);
    static constexpr size_t off_wt = off_zin + zin_bytes;
    static constexpr size_t wt_bytes = al(GR * GC);
    static constexpr size_t off_red = off_wt + wt_bytes;
    static constexpr size_t bytes = off_red + al(16 + 4 * GR);  // dt / V, a CFL minimum, a bound per warp
};

// x wrapped into [0, n) for any x (the Z region reaches two cells beyond the
// mesh, more than one period when n == 1).
__device__ __forceinline__ int wrap_any(int x, int n) {
    x = wrap_idx(x, n);
    return x < 0 ? (x % n + n) % n : x;
}

// Global cell of Z entry (zr, zc) (entry (2, 2) is cell (i0, j0)); false
// outside a non-periodic side.
__device__ __forceinline__ bool z_cell(const StructMesh &m, int i0, int j0, int zr, int zc, int &gi, int &gj) {
    gi = i0 + zr - 2;
    gj = j0 + zc - 2;
    if (gi < 0 || gi >= m.nx) {
        if (!m.xper) return false;
        gi = wrap_any(gi, m.nx);
    }
    if (gj < 0 || gj >= m.ny) {
        if (!m.yper) return false;
        gj = wrap_any(gj, m.ny);
    }
    return true;
}

// Quotients that are the same for every cell, formed once on the host (an
// FP64 division is some 25 instructions: the seven of them that each thread
// used to form were a tenth of the kernel's instructions).
template <typename R>
struct StepConst {
    R halfx, halfy;    // h / 2
    R inv2hx, inv2hy;  // 1 / 2h
    R invhx, invhy;    // 1 / h
    R igm1;            // 1 / (gamma - 1)
};
template <typename R>
inline StepConst<R> step_const(const SmfArgs &a) {
    const StructMesh &m = a.mesh;
    return StepConst<R>{R(0.5 * m.hx), R(0.5 * m.hy), R(0.5 / m.hx),      R(0.5 / m.hy),
                        R(1.0 / m.hx), R(1.0 / m.hy), R(1.0 / a.eos.gm1)};
}

// A lower bound of the CFL term dinc / (|v| + c) in FP32: dinc^2 and the
// squares of the two speeds rounded to FP32, each step within a few 2^-24,
// the quotient taken 2e-4 too small.  0 where FP32 cannot hold the squares
// (the caller then takes the FP64 term).
__device__ __forceinline__ float cfl_lower(double dinc2, double c2, double v2) {
    const float d = sqrtf((float)dinc2), s = sqrtf((float)c2) + sqrtf((float)v2);
    const bool in_range = d > 1e-15f && d < 1e15f && s > 1e-10f && s < 1e15f;
    return in_range ? __fdividef(d, s) * 0.9998f : 0.0f;
}

// One block's tile.  INTERIOR: the whole Z region lies inside the mesh (no
// boundary face, no wrapped index), so the boundary selects, the wrapping and
// the domain marks drop out.
template <typename R, bool MIXED, int MODE, int LIM, int TH, bool INTERIOR>
__device__ __forceinline__ void step_tile(const SmfArgs &a, const Fields<R> &f, const StepConst<R> &k) {
    using L = FusedLayout<R, TH, MODE>;
    constexpr int ZR = L::ZR, ZC = L::ZC, GR = L::GR, GC = L::GC, NT = L::NT;
    constexpr bool PC = MODE == FUSED_PC;
    extern __shared__ __align__(16) unsigned char smem[];
    R(*Z)[ZR][ZC] = reinterpret_cast<R(*)[ZR][ZC]>(smem + L::off_z);
    double(*FX)[TH + 1][GC] = reinterpret_cast<double(*)[TH + 1][GC]>(smem + L::off_fx);
    double(*FY)[TH][GC] = reinterpret_cast<double(*)[TH][GC]>(smem + L::off_fy);
    R(*G)[GR][GC] = reinterpret_cast<R(*)[GR][GC]>(smem + L::off_g);
    R(*H)[GR][GC] = reinterpret_cast<R(*)[GR][GC]>(smem + L::off_h);
    double(*Q)[GR][GC] = reinterpret_cast<double(*)[GR][GC]>(smem + L::off_q);
    unsigned char(*zin)[ZC] = reinterpret_cast<unsigned char(*)[ZC]>(smem + L::off_zin);
    unsigned char(*wt)[GC] = reinterpret_cast<unsigned char(*)[GC]>(smem + L::off_wt);
    unsigned long long *red = reinterpret_cast<unsigned long long *>(smem + L::off_red);

    const StructMesh &m = a.mesh;
    const int l = threadIdx.x, r = threadIdx.y, tid = r * 32 + l;
    const int i0 = blockIdx.y * TH, j0 = blockIdx.x * 30;
    const EosR<R> eos = eos_as<R>(a.eos);
    const R igm1 = k.igm1, halfx = k.halfx, halfy = k.halfy;
    // source of the stage: the state at t^n, or the Heun stage value z*
    const R *const *src = MODE == FUSED_HEUN_B ? const_cast<const R *const *>(f.h) : f.w;

    if (MODE != FUSED_HEUN_B && blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) {
        *f.dt_out = step_dt(a, f.slot_cur);
        *f.slot_clr = 0x7FEFFFFFFFFFFFFFull;
    }
    const double dt = step_dt(a, f.slot_cur);

    // ---- phase 0: stage Z ----------------------------------------------------
    if (INTERIOR) {
        // row by row: 32 columns by every warp, the last two by its low lanes
        const R *p0 = src[0], *p1 = src[1], *p2 = src[2], *p3 = src[3], *p4 = src[4];
        for (int zr = r; zr < ZR; zr += GR) {
            int g = (i0 + zr - 2) * m.ny + j0 - 2 + l;
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
            int gi, gj;
            const bool in = z_cell(m, i0, j0, zr, zc, gi, gj);
            zin[zr][zc] = in;
            if (in) {
                const int g = gi * m.ny + gj;
#pragma unroll
                for (int q = 0; q < 5; ++q) Z[q][zr][zc] = src[q][g];
            }
        }
    }
    // dt / V once per block, and the next step's CFL minimum so far
    if (tid == 0) {
        red[0] = dbits(dt / m.vol);
        if (MODE != FUSED_HEUN_A) red[1] = __ldcg(f.slot_nxt);
    }
    __syncthreads();
    const double coef = __longlong_as_double((long long)red[0]);

    // ---- phase 1: gradients (and the half step) of the G cell (r, l) ---------
    if (INTERIOR || zin[r + 1][l + 1]) {
        int gi = i0 - 1 + r, gj = j0 - 1 + l;  // wrapped global coordinates
        if (!INTERIOR && m.xper) gi = wrap_idx(gi, m.nx);
        if (!INTERIOR && m.yper) gj = wrap_idx(gj, m.ny);
        const int zr = r + 1, zc = l + 1;
        // conserved state of the cell at t^n (predictor-corrector): FAST from
        // the staged primitive state, MIXED from the FP64 fields (loaded here,
        // ahead of the gradient arithmetic)
        C4<double> q0{0.0, 0.0, 0.0, 0.0};
        if (PC) {
            if (MIXED) {
                const int g = gi * m.ny + gj;
                q0 = C4<double>{f.q[0][g], f.q[1][g], f.q[2][g], f.q[3][g]};
            } else {
                q0 = cons_of(Z[0][zr][zc], Z[1][zr][zc], Z[2][zr][zc], Z[4][zr][zc]);
            }
        }
        // boundary flags of the four slots (the normals are the axes)
        const int fL = INTERIOR || gi > 0 ? BC_INNER : m.bc[0];
        const int fR = INTERIOR || gi < m.nx - 1 ? BC_INNER : m.bc[1];
        const int fB = INTERIOR || gj > 0 ? BC_INNER : m.bc[2];
        const int fT = INTERIOR || gj < m.ny - 1 ? BC_INNER : m.bc[3];
        const bool bL = is_boundary(fL), bR = is_boundary(fR), bB = is_boundary(fB), bT = is_boundary(fT);
        R gx[4], gy[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            // a boundary slot takes the reflected own value (only the normal
            // velocity changes sign at a wall)
            const R c = Z[q][zr][zc];
            const R nL = bL ? ((q == 1 && fL == BC_WALL) ? -c : c) : Z[q][zr - 1][zc];
            const R nR = bR ? ((q == 1 && fR == BC_WALL) ? -c : c) : Z[q][zr + 1][zc];
            const R nB = bB ? ((q == 2 && fB == BC_WALL) ? -c : c) : Z[q][zr][zc - 1];
            const R nT = bT ? ((q == 2 && fT == BC_WALL) ? -c : c) : Z[q][zr][zc + 1];
            gx[q] = slope<LIM, R>(a.limiter, nL - c, nR - c, k.inv2hx, k.invhx);
            gy[q] = slope<LIM, R>(a.limiter, nB - c, nT - c, k.inv2hy, k.invhy);
            G[q][r][l] = gx[q];
            G[4 + q][r][l] = gy[q];
        }
        if (PC) {
            const int g = gi * m.ny + gj;
            const bool waiting = f.wait_in[g] > 0;
            wt[r][l] = waiting;
            const FS<R> zc5{Z[0][zr][zc], Z[1][zr][zc], Z[2][zr][zc], Z[3][zr][zc], Z[4][zr][zc], R(0)};
            P5<R> hz{zc5.r, zc5.u, zc5.v, zc5.p, zc5.e};
            if (!waiting) {
                // predictor (sm_fluid.cpp:176-253): half step with the physical
                // flux of the cell's own face values; the flux of the low face
                // (normal -x or -y) is minus the flux along the axis
                double F[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const bool ax = s < 2;
                    const R off = s == 0 ? -halfx : (s == 1 ? halfx : (s == 2 ? -halfy : halfy));
                    const C4<R> lf = half_flux(zc5, ax ? gx : gy, off, ax, eos, igm1, [](bool on, auto &&fix) {
                        if (on) fix();
                    });
                    add_half(F, lf, (s == 0 || s == 2) ? -(ax ? m.hy : m.hx) : (ax ? m.hy : m.hx));
                }
                const double half = 0.5 * coef;
                C4<double> q = q0;
                subtract(q, half, F);
                double ri;
                const P5<double> hd = prim_ri(q, a.eos, ri);
                if (!bad64(hd, a.eos)) hz = down<R>(hd);
            }
            H[0][r][l] = hz.r;
            H[1][r][l] = hz.u;
            H[2][r][l] = hz.v;
            H[3][r][l] = hz.p;
            H[4][r][l] = hz.e;
            Q[0][r][l] = q0.r;
            Q[1][r][l] = q0.mu;
            Q[2][r][l] = q0.mv;
            Q[3][r][l] = q0.E;
        }
    }
    __syncthreads();

    // ---- phase 2: the faces bounding interior cells, each once ---------------
    // face-state source of G cell (gr, gc): the half step, or the Z state
    // (its reciprocal density is formed only where the state itself is used)
    auto sc = [&](int gr, int gc) {
        if (PC) return FS<R>{H[0][gr][gc], H[1][gr][gc], H[2][gr][gc], H[3][gr][gc], H[4][gr][gc], R(0)};
        return FS<R>{Z[0][gr + 1][gc + 1], Z[1][gr + 1][gc + 1], Z[2][gr + 1][gc + 1], Z[3][gr + 1][gc + 1],
                     Z[4][gr + 1][gc + 1], R(0)};
    };
    auto sc_ri = [&](int gr, int gc) {
        FS<R> z = sc(gr, gc);
        z.ri = rcp_r(z.r);
        return z;
    };
    // reconstruction of G cell (gr, gc) at its face on axis `ax` (0: x, 1: y),
    // side `hi` (the +x / +y face, else the low one), FaceExtra::Direct
    // (face_extra.h:121-184); a bad value falls back to the cell state
    auto recon = [&](int gr, int gc, int ax, bool hi, bool boundary) {
        const FS<R> z = sc(gr, gc);
        const R off = ax == 0 ? (hi ? halfx : -halfx) : (hi ? halfy : -halfy);
        const int b = 4 * ax;
        FS<R> o = reconstruct(z, G[b][gr][gc], G[b + 1][gr][gc], G[b + 2][gr][gc], G[b + 3][gr][gc], off,
                              !hi && !boundary);
        o.ri = rcp_r(o.r);
        o.e = energy_ri(eos, o.p, o.ri, igm1);
        if (bad_value(o, eos.pmin)) {
            o = z;
            o.ri = rcp_r(z.r);
        }
        return o;
    };
    // interior face: the frame of the +x (DIR 0) or +y (DIR 1) normal, where
    // the rotation of rotate.cpp is the identity or (u, v) -> (v, -u)
    auto face_interior = [&](auto dirc) {
        constexpr int DIR = decltype(dirc)::value;
        const int rB = r + (DIR == 0), lB = l + (DIR == 1);
        const bool robust = PC && (wt[r][l] || wt[rB][lB]);
        FS<R> zm, zp;
        if (robust) {
            zm = sc_ri(r, l);
            zp = sc_ri(rB, lB);
        } else {
            zm = recon(r, l, DIR, true, false);
            zp = recon(rB, lB, DIR, false, false);
        }
        if (DIR == 1) {
            R t = zm.u;
            zm.u = zm.v;
            zm.v = -t;
            t = zp.u;
            zp.u = zp.v;
            zp.v = -t;
        }
        constexpr bool VR = DIR == 1, VL = VR || MODE == FUSED_HEUN_A;
        C4<R> lf = (robust || a.flux == FLUX_HLL) ? hll_fs<VL, VR, DIR == 1>(zm, zp, eos)
                                                  : hllc_any<VL, VR>(zm, zp, eos);
        if (DIR == 1) {
            const R t = lf.mu;
            lf.mu = -lf.mv;
            lf.mv = t;
        }
        return lf;
    };
    // boundary face (WALL / ZOE) seen from its only cell (out of line)
    auto face_boundary = [&](int dir, bool own_a) {
        const int gr = own_a ? r : r + (dir == 0), gc = own_a ? l : l + (dir == 1);
        const int s_own = own_a ? (dir == 0 ? 1 : 3) : (dir == 0 ? 0 : 2);
        const bool robust = PC && wt[gr][gc];
        const FS<R> zm = robust ? sc_ri(gr, gc) : recon(gr, gc, dir, own_a, true);
        return boundary_flux<MODE == FUSED_HEUN_A>(zm, s_own, m.bc[s_own], robust || a.flux == FLUX_HLL, eos, own_a);
    };
    // (predictor-corrector: the fluxes overwrite Z, which no thread reads
    // after phase 1)
    if (r <= TH && l >= 1 && l <= 30) {  // +x face between G cells (r, l) and (r + 1, l)
        const bool inA = INTERIOR || zin[r + 1][l + 1], inB = INTERIOR || zin[r + 2][l + 1];
        C4<R> lf{R(0), R(0), R(0), R(0)};
        if (inA && inB) lf = face_interior(std::integral_constant<int, 0>{});
        else if (!INTERIOR && (inA || inB)) lf = face_boundary(0, inA);
        FX[0][r][l] = lf.r;
        FX[1][r][l] = lf.mu;
        FX[2][r][l] = lf.mv;
        FX[3][r][l] = lf.E;
    }
    if (r >= 1 && r <= TH && l <= 30) {  // +y face between G cells (r, l) and (r, l + 1)
        const bool inA = INTERIOR || zin[r + 1][l + 1], inB = INTERIOR || zin[r + 1][l + 2];
        C4<R> lf{R(0), R(0), R(0), R(0)};
        if (inA && inB) lf = face_interior(std::integral_constant<int, 1>{});
        else if (!INTERIOR && (inA || inB)) lf = face_boundary(1, inA);
        FY[0][r - 1][l] = lf.r;
        FY[1][r - 1][l] = lf.mu;
        FY[2][r - 1][l] = lf.mv;
        FY[3][r - 1][l] = lf.E;
    }
    __syncthreads();

    // ---- phase 3: update of the interior cells --------------------------------
    float low = INFINITY;  // lower bound of the cell's CFL term (0: none; infinite: no cell)
    P5<double> zn{};
    const int i = i0 - 1 + r, j = j0 - 1 + l;
    if (r >= 1 && r <= TH && l >= 1 && l <= 30 && (INTERIOR || (i < m.nx && j < m.ny))) {
        const int ic = i * m.ny + j;
        const double hy = m.hy, hx = m.hx;
        double F[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            F[k] = MIXED ? flux_sum(FX[k][r - 1][l], FX[k][r][l], FY[k][r - 1][l - 1], FY[k][r - 1][l], hx, hy)
                         : rfma(FX[k][r][l], hy,
                                three_fluxes(FX[k][r - 1][l], FY[k][r - 1][l - 1], FY[k][r - 1][l], hx, hy));
        C4<double> q;
        if (MODE == FUSED_HEUN_B) {
            // Q(z*) of the stage value, its step, and the mean with Q(z^n)
            q = cons_less(Z[0][r + 1][l + 1], Z[1][r + 1][l + 1], Z[2][r + 1][l + 1], Z[4][r + 1][l + 1], coef, F);
            const C4<double> q0 = q_n<R, MIXED>(f, ic);
            q.r = 0.5 * (q0.r + q.r);
            q.mu = 0.5 * (q0.mu + q.mu);
            q.mv = 0.5 * (q0.mv + q.mv);
            q.E = 0.5 * (q0.E + q.E);
        } else {
            q = PC ? C4<double>{Q[0][r][l], Q[1][r][l], Q[2][r][l], Q[3][r][l]} : q_n<R, MIXED>(f, ic);
            subtract(q, coef, F);
        }
        double ri;
        zn = prim_ri(q, a.eos, ri);
        if (MODE == FUSED_HEUN_A) {
            st5(f.h, ic, down<R>(zn));  // Heun stage value
        } else {
            if (PC) {
                int wn = f.wait_in[ic];
                if (bad64(zn, a.eos)) {
                    // isolation (sm_fluid.cpp:354-358): keep the old state
                    zn = P5<double>{(double)f.w[0][ic], (double)f.w[1][ic], (double)f.w[2][ic],
                                    (double)f.w[3][ic], (double)f.w[4][ic]};
                    q = q_n<R, MIXED>(f, ic);
                    ri = rcp_nr(zn.r);
                    wn = 3;
                } else if (wn > 0) {
                    --wn;
                }
                f.wait_out[ic] = wn;
            }
            if (MIXED) {
                f.qn[0][ic] = q.r;
                f.qn[1][ic] = q.mu;
                f.qn[2][ic] = q.mv;
                f.qn[3][ic] = q.E;
            }
            st5(f.wn, ic, down<R>(zn));
            low = cfl_lower(smin(m.inc2x[i], m.inc2y[j]), a.eos.gamma * (zn.p + a.eos.P0) * ri, sq2(zn.u, zn.v));
        }
    }
    // The minimum of the CFL terms of the new state for the next step
    // (sm_fluid.cpp:104-111), with the arithmetic of k_cfl, which takes the
    // minimum after an upload or a halo exchange: the same state gives the
    // same dt.  That term (two divisions and three square roots in FP64) is
    // formed only where its FP32 lower bound does not exceed the block's
    // smallest and the minimum that other blocks have reached: a larger
    // bound cannot hold the minimum.
    if (MODE != FUSED_HEUN_A) {
        float wmin = low > 0.0f ? low : INFINITY;
        for (int o = 16; o > 0; o >>= 1) wmin = fminf(wmin, __shfl_xor_sync(0xffffffffu, wmin, o));
        float *redf = reinterpret_cast<float *>(red + 2);
        if (l == 0) redf[r] = wmin;
        __syncthreads();
        float lim = redf[l < GR ? l : 0];
        for (int o = 16; o > 0; o >>= 1) lim = fminf(lim, __shfl_xor_sync(0xffffffffu, lim, o));
        // 1.0005: the bound is at most 3e-4 below its term
        lim = fminf(lim * 1.0005f, __double2float_ru(__longlong_as_double((long long)red[1])));
        const bool take = low <= lim && low < INFINITY;
        if (__any_sync(0xffffffffu, take)) {
            unsigned long long best = 0x7FEFFFFFFFFFFFFFull;
            if (take) {
                const double lam = cfl_term(a, i, j, zn.r, zn.u, zn.v, zn.p, MIXED && PC);
                if (lam >= 0.0) best = dbits(lam);
            }
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long t2 = __shfl_xor_sync(0xffffffffu, best, o);
                best = t2 < best ? t2 : best;
            }
            if (l == 0) atomicMin(f.slot_nxt, best);
        }
    }
}

template <typename R, bool MIXED, int MODE, int LIM, int TH, int MINB>
__global__ void __launch_bounds__(32 * (TH + 2), MINB) k_step(SmfArgs a, Fields<R> f, StepConst<R> k) {
    after_previous();
    const int i0 = blockIdx.y * TH, j0 = blockIdx.x * 30;
    // (a limiter chosen at run time: one copy of its code)
    if constexpr (LIM >= 0) {
        if (i0 >= 2 && i0 + TH + 2 <= a.mesh.nx && j0 >= 2 && j0 + 32 <= a.mesh.ny) {
            step_tile<R, MIXED, MODE, LIM, TH, true>(a, f, k);
            return;
        }
    }
    step_tile<R, MIXED, MODE, LIM, TH, false>(a, f, k);
}

// Meshes that leave the 14-row tiles few blocks run tiles of 4 rows, as long as
// their blocks are resident at once (192 threads each; FP64's predictor-corrector
// has registers for three on an SM, the others for four): one block's phases,
// one after the other, are what a step of such a mesh takes.  us a step, 4 rows /
// 14 rows (van Albada HLLC): FP64 predictor-corrector 64^2 7.3 / 9.0, 129x67 8.8 /
// 9.1, 200^2 8.8 / 10.3, 220x210 8.7 / 10.3; Heun 200^2 15.8 / 18.4; MIXED Heun
// 129x67 11.0 / 12.1, 240^2 14.8 / 15.5 (2 rows: 200^2 8.5 and 14.8, but 2 waves
// from 210^2 on; MIXED Heun with MC 129x67 16.7 against 12.5).
// One wave of 14-row tiles on more than half of the SMs is launched normally:
// blocks of the next kernel that wait beside it cost more than the launch saves
// (240^2 12.4 us with the dependent launch, 10.3 without; 256^2, more than one
// wave, 12.5 with, 14.4 without).
constexpr int SMALL_TH = 4, SMALL_MINB = 3, SMS = 148;
inline bool small_tiles(const StructMesh &m, int resident) {
    return (long long)((m.ny + 29) / 30) * ((m.nx + SMALL_TH - 1) / SMALL_TH) <= (long long)resident * SMS;
}

// Launch one stage of the fused step on `stream` (dynamic shared memory of
// FusedLayout::bytes, above the 48 KB default).
template <typename R, bool MIXED, int MODE, int LIM, int TH, int MINB>
inline void launch_fused_stage(const SmfArgs &a, const Fields<R> &f, cudaStream_t s) {
    using L = FusedLayout<R, TH, MODE>;
    static unsigned long long attr_set = 0;  // devices on which the attribute is set
    auto kern = k_step<R, MIXED, MODE, LIM, TH, MINB>;
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 64 || !(attr_set >> dev & 1ull)) {
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::bytes);
        if (dev < 64) attr_set |= 1ull << dev;
    }
    dim3 block(32, TH + 2);
    dim3 grid((a.mesh.ny + 29) / 30, (a.mesh.nx + TH - 1) / TH);
    const long long blocks = (long long)grid.x * grid.y;
    if (TH == SMALL_TH || 2 * blocks <= SMS || blocks > SMS)
        launch_after(kern, grid, block, L::bytes, s, a, f, step_const<R>(a));
    else
        kern<<<grid, block, L::bytes, s>>>(a, f, step_const<R>(a));
}

// One stage (FUSED_PC, FUSED_HEUN_A or FUSED_HEUN_B) with the limiter
// compiled in for the common ones.  HLLC and HLL only: the fused kernels
// carry neither Godunov's exact solver nor Rusanov.
template <typename R, bool MIXED, int TH, int MINB, int MODE>
inline void fused_stage(const SmfArgs &a, const Fields<R> &f, cudaStream_t s) {
    switch (a.limiter) {
        case LIM_VANALBADA1: launch_fused_stage<R, MIXED, MODE, LIM_VANALBADA1, TH, MINB>(a, f, s); break;
        case LIM_MC: launch_fused_stage<R, MIXED, MODE, LIM_MC, TH, MINB>(a, f, s); break;
        case LIM_MINMOD: launch_fused_stage<R, MIXED, MODE, LIM_MINMOD, TH, MINB>(a, f, s); break;
        case LIM_VANLEER: launch_fused_stage<R, MIXED, MODE, LIM_VANLEER, TH, MINB>(a, f, s); break;
        default: launch_fused_stage<R, MIXED, MODE, -1, TH, MINB>(a, f, s); break;
    }
}

template <typename R, bool MIXED, int TH, int MINB>
inline void fused_dispatch(const SmfArgs &a, const Fields<R> &f, int mode, cudaStream_t s) {
    if (mode == FUSED_PC) fused_stage<R, MIXED, TH, MINB, FUSED_PC>(a, f, s);
    else if (mode == FUSED_HEUN_A) fused_stage<R, MIXED, TH, MINB, FUSED_HEUN_A>(a, f, s);
    else fused_stage<R, MIXED, TH, MINB, FUSED_HEUN_B>(a, f, s);
}

}  // namespace tiled
}  // namespace zg
