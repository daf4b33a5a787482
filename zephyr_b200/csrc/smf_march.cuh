// smf_march.cuh -- the second-order step of a structured rectangle with every
// warp marching down the rows of its own strip of columns: the arithmetic of
// the fused tile kernel (smf_fused.cuh: limited gradients, half step, face-once
// corrector, update, the next step's CFL minimum) without block barriers.
//
// A warp owns 28 columns: lane l holds column j0 - 2 + l, lanes 2..29 are
// updated, the outer two on each side are the stencil's halo.  It walks the
// rows g = i_lo - 1 .. i_hi of its segment; at row g it has the states of
// rows g - 1, g and g + 1 (its own ring in shared memory), forms the gradients
// and the half step of row g, the faces between lanes l and l + 1 of row g
// (the neighbour's face state by shuffles), the faces between rows g - 1 and g
// (the row above's face state is carried over), and then finishes row g - 1.
//
// Why this form: the tile kernel (30 x 14 cells per 512-thread block) waits a
// third of its time at its four barriers and for the staging loads (ncu, issue
// slots 57 % used), and its tile halo costs 1.22 evaluations per cell.  Here a
// warp waits for nobody; its rows come through a ring in shared memory, copied
// asynchronously a row ahead; the halo costs 32/28 in the row and two rows per
// segment.  Bound: FP64 pipe 49 % and issue 58 %, fixed-latency dependencies
// with 4 warps per scheduler (128 registers).  Two things that cost more than
// they look: an atomic minimum per cell on the one CFL slot (190 us at 1024^2
// against 88 with one per warp), and bad-value fallbacks as selects instead of
// branches under a warp vote (5 % of a step at 2048^2).
// Measured (B200, one step of van Albada HLLC, march / tile with the same
// formulas): FP64 predictor-corrector 2048^2 310 / 317 us, 3072^2 648 / 704, Heun
// 2048^2 430 / 463; MIXED 246 / 248, 514 / 544, 304 / 375 (before the march: FP64
// 353 and 542, MIXED 293 and 457 at 2048^2).
// Both forms give the same bits: shared formulas with written-out roundings.  In
// MIXED that holds on periodic axes (a boundary face is another instance in the
// tile, seen from its own cell), so MIXED marches only on rectangles that are
// periodic both ways.
#pragma once

#include "smf_fused.cuh"

namespace zg {
namespace tiled {

constexpr int MARCH_COLS = 28;   // columns a warp updates
constexpr int MARCH_WARPS = 4;   // warps per block (they do not cooperate)

template <typename R>
__device__ __forceinline__ FS<R> shfl_down_fs(const FS<R> &z) {
    return FS<R>{__shfl_down_sync(0xffffffffu, z.r, 1), __shfl_down_sync(0xffffffffu, z.u, 1),
                 __shfl_down_sync(0xffffffffu, z.v, 1), __shfl_down_sync(0xffffffffu, z.p, 1),
                 __shfl_down_sync(0xffffffffu, z.e, 1), __shfl_down_sync(0xffffffffu, z.ri, 1)};
}

// Rare corrections (a bad reconstructed value) run under a warp vote, so that
// the common path carries a branch instead of a select per value.
template <typename F>
__device__ __forceinline__ void rare(bool on, F &&fix) {
    if (__any_sync(0xffffffffu, on)) {
        if (on) fix();
    }
}

// A cell's value at the face centre `off` along an axis (FaceExtra::Direct,
// face_extra.h:121-184) with slopes gr; the cell's own state where that is
// bad.  All lanes of the warp call it.
template <typename R>
__device__ __forceinline__ FS<R> face_value(const FS<R> &h, const R gr[4], R off, bool low, const EosR<R> &eos,
                                            R igm1) {
    FS<R> o = reconstruct(h, gr[0], gr[1], gr[2], gr[3], off, low);
    o.ri = rcp_r(o.r);
    o.e = energy_ri(eos, o.p, o.ri, igm1);
    rare(bad_value(o, eos.pmin), [&] {
        o = h;
        o.ri = rcp_r(h.r);
    });
    return o;
}

// Half step (sm_fluid.cpp:176-253) of a cell: the state after dt / 2 of the
// physical fluxes of its own face values; the cell's own state where it comes
// out bad.  All lanes of the warp call it.
template <typename R>
__device__ __forceinline__ FS<R> half_step(const FS<R> &c, const C4<double> &q0, const R gx[4], const R gy[4],
                                           const StepConst<R> &k, const EosR<R> &eos, const EosD &eosd, double hx,
                                           double hy, double coef) {
    double F[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const bool ax = s < 2;
        const R off = s == 0 ? -k.halfx : (s == 1 ? k.halfx : (s == 2 ? -k.halfy : k.halfy));
        const C4<R> lf = half_flux(c, ax ? gx : gy, off, ax, eos, k.igm1, [](bool on, auto &&fix) { rare(on, fix); });
        add_half(F, lf, (s == 0 || s == 2) ? -(ax ? hy : hx) : (ax ? hy : hx));
    }
    const double half = 0.5 * coef;
    C4<double> q = q0;
    subtract(q, half, F);
    double ri;
    const P5<double> hd = prim_ri(q, eosd, ri);
    const P5<R> hr = down<R>(hd);
    FS<R> h{hr.r, hr.u, hr.v, hr.p, hr.e, R(0)};
    rare(bad64(hd, eosd), [&] { h = c; });
    return h;
}

// VL, VR, Y: as hll_fs
template <bool HLL, bool VL, bool VR, bool Y, typename R>
__device__ __forceinline__ C4<R> march_flux(const FS<R> &L, const FS<R> &Rs, const EosR<R> &eos) {
    if constexpr (HLL) return hll_fs<VL, VR, Y>(L, Rs, eos);
    else if constexpr (sizeof(R) == 4) return hllc_fs<VL, VR>(L, Rs, eos);
    else return hllc_d<true>(L, Rs, eos);
}

// The next step's CFL minimum (sm_fluid.cpp:104-111) over a warp's cells, with
// k_cfl's arithmetic.  Two divisions and three square roots a cell, so the
// term is formed only where its FP32 lower bound exceeds neither the smallest
// of the warp's cells so far nor what other warps have reported.
struct WarpCfl {
    unsigned long long best = 0x7FEFFFFFFFFFFFFFull;  // smallest term of the lane's cells
    float low = INFINITY;                             // smallest bound of the warp's cells
    float reported = INFINITY;                        // other warps' minimum

    // other warps' minimum so far: read now and then (every read of every
    // warp goes to one address)
    __device__ __forceinline__ void refresh(const unsigned long long *slot) {
        reported = __double2float_ru(__longlong_as_double((long long)__ldcg(slot)));
    }
    // all lanes of the warp call it; `live`: with a cell; VU: as cfl_term's vu
    template <bool VU>
    __device__ __forceinline__ void add(const SmfArgs &a, int i, int j, const P5<double> &z, double ri, bool live) {
        const StructMesh &m = a.mesh;
        const float lo = cfl_lower(m.inc2min, a.eos.gamma * (z.p + a.eos.P0) * ri, sq2(z.u, z.v));
        // (bounds are >= 0, so they order like their bits)
        const float w = live && lo > 0.0f ? lo : INFINITY;
        low = fminf(low, __uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(w))));
        // 1.0005: a bound is at most 3e-4 below its term
        if (live && lo <= fminf(low * 1.0005f, reported)) {
            const double lam = cfl_term(a, i, j, z.r, z.u, z.v, z.p, VU);
            if (lam >= 0.0 && dbits(lam) < best) best = dbits(lam);
        }
    }
    __device__ __forceinline__ void commit(unsigned long long *slot) {
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long t = __shfl_xor_sync(0xffffffffu, best, o);
            best = t < best ? t : best;
        }
        if ((threadIdx.x & 31) == 0 && best < __ldcg(slot)) atomicMin(slot, best);
    }
};

// New state of an updated cell (`live` lanes; all lanes call): isolation,
// stores, CFL term.
template <typename R, bool MIXED, int MODE>
__device__ __forceinline__ void store_cell(const SmfArgs &a, const Fields<R> &f, int i, int j, bool live,
                                           C4<double> q, int wait, WarpCfl &cfl) {
    const int ic = i * a.mesh.ny + j;
    double ri;
    P5<double> zn = prim_ri(q, a.eos, ri);
    if (MODE == FUSED_HEUN_A) {
        if (live) st5(f.h, ic, down<R>(zn));
        return;
    }
    if (live) {
        if (MODE == FUSED_PC) {
            int wn = wait;
            if (bad64(zn, a.eos)) {
                // isolation (sm_fluid.cpp:354-358): keep the old state
                zn = P5<double>{(double)f.w[0][ic], (double)f.w[1][ic], (double)f.w[2][ic], (double)f.w[3][ic],
                                (double)f.w[4][ic]};
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
    }
    cfl.add<MIXED && MODE == FUSED_PC>(a, i, j, zn, ri, live);
}

// One asynchronous copy of a lane's value (4 or 8 bytes) into shared memory.
template <typename T>
__device__ __forceinline__ void async_copy(T *dst, const T *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(T) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void async_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// A warp's rows in shared memory: the stage's source state of four rows (g - 1,
// g, g + 1 and the one on its way), and, where the conserved state at t^n is
// not that source, what it is formed from, of three rows (g - 1, g, g + 1).
template <typename R, bool MIXED, int MODE>
struct MarchRing {
    static constexpr bool BASE = (MIXED && MODE != FUSED_HEUN_B) || MODE == FUSED_HEUN_B;
    R z[4][5][32];
    double b[BASE ? 3 : 1][BASE ? 4 : 1][BASE ? 32 : 1];
};

template <typename R, bool MIXED, int MODE, bool HLL, int MINB>
__global__ void __launch_bounds__(32 * MARCH_WARPS, MINB) k_march(const __grid_constant__ SmfArgs a,
                                                                  const __grid_constant__ Fields<R> f,
                                                                  const __grid_constant__ StepConst<R> k, int strips,
                                                                  int rows) {
    constexpr bool PC = MODE == FUSED_PC, FIRST = MODE == FUSED_HEUN_A;
    constexpr unsigned ALL = 0xffffffffu;
    using Ring = MarchRing<R, MIXED, MODE>;
    __shared__ Ring rings[MARCH_WARPS];
    Ring &ring = rings[threadIdx.x >> 5];
    const StructMesh &m = a.mesh;
    const int l = threadIdx.x & 31;
    const int w = blockIdx.x * MARCH_WARPS + (threadIdx.x >> 5);
    const double dt = step_dt(a, f.slot_cur);
    if (MODE != FUSED_HEUN_B && blockIdx.x == 0 && threadIdx.x == 0) {
        *f.dt_out = dt;
        *f.slot_clr = 0x7FEFFFFFFFFFFFFFull;
    }
    const int seg = w / strips, strip = w - seg * strips;
    const int i_lo = seg * rows;
    if (i_lo >= m.nx) return;  // whole warps (no barrier follows)
    const int i_hi = min(i_lo + rows, m.nx);
    const int j = strip * MARCH_COLS - 2 + l;
    const bool live = l >= 2 && l < 2 + MARCH_COLS && j < m.ny;  // updated columns
    // the column in memory: wrapped, or the nearest one where a side has no
    // neighbour (those lanes' results reach no updated cell)
    const int jc = m.yper ? wrap_any(j, m.ny) : min(max(j, 0), m.ny - 1);
    const bool jlow = !m.yper && j == 0, jhigh = !m.yper && j == m.ny - 1;
    const bool sides = __any_sync(ALL, jlow || jhigh);  // a side of the mesh runs through the strip
    auto row = [&](int i) { return (m.xper ? wrap_any(i, m.nx) : min(max(i, 0), m.nx - 1)) * m.ny + jc; };
    const double coef = dt / m.vol, hx = m.hx, hy = m.hy;
    WarpCfl cfl;
    bool iso = false;  // an isolated cell in the segment or beside it
    if (PC) {
        int any = 0;
        for (int g = i_lo - 1; g <= i_hi; ++g) any |= f.wait_in[row(g)];  // counters are never negative
        iso = __any_sync(ALL, any != 0);
    }
    const EosR<R> eos = eos_as<R>(a.eos);
    // source of the stage: the state at t^n, or the Heun stage value z*
    const R *const *src = MODE == FUSED_HEUN_B ? const_cast<const R *const *>(f.h) : f.w;
    // row g into its ring slots
    auto fetch_z = [&](int g, int slot) {
        const int ic = row(g);
#pragma unroll
        for (int q = 0; q < 5; ++q) async_copy(&ring.z[slot][q][l], src[q] + ic);
    };
    auto fetch_b = [&](int g, int slot) {
        if constexpr (Ring::BASE) {
            const int ic = row(g);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if constexpr (MIXED) async_copy(&ring.b[slot][q][l], f.q[q] + ic);
                else async_copy(&ring.b[slot][q][l], f.w[q == 3 ? 4 : q] + ic);
            }
        }
    };
    // conserved state at t^n of the row in slot sb of the base ring (slot sz of the state ring)
    auto base = [&](int sz, int sb) {
        if constexpr (Ring::BASE) {
            const double b0 = ring.b[sb][0][l], b1 = ring.b[sb][1][l], b2 = ring.b[sb][2][l], b3 = ring.b[sb][3][l];
            if constexpr (MIXED) return C4<double>{b0, b1, b2, b3};
            else return cons_of(b0, b1, b2, b3);
        } else {
            return cons_of(ring.z[sz][0][l], ring.z[sz][1][l], ring.z[sz][2][l], ring.z[sz][4][l]);
        }
    };

    FS<R> up{};     // row g - 1's state at its high face
    // row g - 1: the fluxes through its other three faces.  FP64: their sum.
    // MIXED: the FP32 fluxes themselves (low x, low y, high y), whose sum takes
    // them in another order (flux_sum)
    double acc[4];
    C4<R> fxl{}, fyl{}, fyh{};
    int sm = 0, sc = 1, sp = 2, sn = 3;  // state slots of rows g - 1, g, g + 1, g + 2
    int bm = 2, bc = 0, bp = 1;          // base slots of rows g - 1, g, g + 1
    fetch_z(i_lo - 2, sm);
    fetch_z(i_lo - 1, sc);
    fetch_z(i_lo, sp);
    fetch_b(i_lo - 1, bc);
    async_commit();
    const int lu = max(l - 1, 0), ld = min(l + 1, 31);
    // Isolated cells (sm_fluid.cpp:285-351) take no half step, and HLL runs
    // between the cells' own states at their faces: branches of the one loop on
    // a flag of the segment.  A second copy of the loop for such segments saves
    // 0.6 % without them (312.5 against 314.4 us at 2048^2), but where both
    // kinds run beside each other they do not fit the instruction cache (1 cell
    // of 10^4 isolated: 380 us against 322; the tile kernel 355).
    int wm = 0, wc = 0;  // counters of rows g - 1 and g
    if (iso) wc = f.wait_in[row(i_lo - 1)];
#pragma unroll 1
    for (int g = i_lo - 1; g <= i_hi; ++g) {
        async_wait();
        __syncwarp();
        // the next iteration's row on its way while this one is computed
        if (g < i_hi) {
            fetch_z(g + 2, sn);
            fetch_b(g + 1, bp);
        }
        async_commit();

        // ---- limited gradients of row g ----------------------------------
        const bool low = !m.xper && g == 0, high = !m.xper && g == m.nx - 1;  // sides of the mesh
        FS<R> h{ring.z[sc][0][l], ring.z[sc][1][l], ring.z[sc][2][l], ring.z[sc][3][l], ring.z[sc][4][l], R(0)};
        const R c4[4] = {h.r, h.u, h.v, h.p};
        R gx[4], gy[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const R c = c4[q];
            R nL = ring.z[sm][q][l], nR = ring.z[sp][q][l];
            if (low) nL = q == 1 && m.bc[0] == BC_WALL ? -c : c;
            if (high) nR = q == 1 && m.bc[1] == BC_WALL ? -c : c;
            R nB = ring.z[sc][q][lu], nT = ring.z[sc][q][ld];
            if (sides) {
                if (jlow) nB = q == 2 && m.bc[2] == BC_WALL ? -c : c;
                if (jhigh) nT = q == 2 && m.bc[3] == BC_WALL ? -c : c;
            }
            gx[q] = slope<LIM_VANALBADA1, R>(LIM_VANALBADA1, nL - c, nR - c, k.inv2hx, k.invhx);
            gy[q] = slope<LIM_VANALBADA1, R>(LIM_VANALBADA1, nB - c, nT - c, k.inv2hy, k.invhy);
        }
        // ---- state the faces are reconstructed from: the half step, or z --
        if (PC) {
            const FS<R> hs = half_step<R>(h, base(sc, bc), gx, gy, k, eos, a.eos, hx, hy, coef);
            if (!iso || wc == 0) h = hs;
        }
        FS<R> own = h;  // for an isolated cell's faces
        int wp = 0;     // counter of row g + 1
        if (iso) {
            own.ri = rcp_r(h.r);
            if (g < i_hi) wp = f.wait_in[row(g + 1)];
        }
        // ---- faces between lanes l and l + 1 (frame of the +y normal) ------
        C4<R> fy;
        {
            FS<R> L = face_value<R>(h, gy, k.halfy, false, eos, k.igm1);
            FS<R> Rs = shfl_down_fs(face_value<R>(h, gy, -k.halfy, true, eos, k.igm1));
            bool robust = false;
            if (iso) {
                const FS<R> next = shfl_down_fs(own);
                robust = (wc | __shfl_down_sync(ALL, wc, 1)) != 0;
                if (robust) L = own, Rs = next;
            }
            if (sides) {  // past a side the mirror of the face's own state
                if (j == -1) {
                    L = Rs;
                    if (m.bc[2] == BC_WALL) L.v = -L.v;
                }
                if (jhigh) {
                    Rs = L;
                    if (m.bc[3] == BC_WALL) Rs.v = -Rs.v;
                }
            }
            const FS<R> Ln{L.r, L.v, L.u, L.p, L.e, L.ri}, Rn{Rs.r, Rs.v, Rs.u, Rs.p, Rs.e, Rs.ri};
            C4<R> t = march_flux<HLL, true, true, true, R>(Ln, Rn, eos);
            if (!HLL && robust) t = hll_fs<true, true, true>(Ln, Rn, eos);
            fy = C4<R>{t.r, t.mv, t.mu, t.E};
        }
        // ---- faces between rows g - 1 and g -------------------------------
        C4<R> fx{};
        if (g > i_lo - 1) {
            FS<R> L = up, Rs = face_value<R>(h, gx, -k.halfx, true, eos, k.igm1);
            const bool robust = iso && (wm | wc) != 0;
            if (robust) Rs = own;
            if (low) {
                L = Rs;
                if (m.bc[0] == BC_WALL) L.u = -L.u;
            }
            if (!m.xper && g == m.nx) {  // the row past the mesh: its low face belongs to row nx - 1
                Rs = L;
                if (m.bc[1] == BC_WALL) Rs.u = -Rs.u;
            }
            fx = march_flux<HLL, FIRST, false, false, R>(L, Rs, eos);
            if (!HLL && robust) fx = hll_fs<FIRST, false, false>(L, Rs, eos);
        }
        // ---- update of row g - 1 -------------------------------------------
        if (g > i_lo) {
            if (MODE != FUSED_HEUN_A && (g - i_lo) % 16 == 1) cfl.refresh(f.slot_nxt);
            double F[4];
            if constexpr (MIXED) {
                F[0] = flux_sum(fxl.r, fx.r, fyl.r, fyh.r, hx, hy);
                F[1] = flux_sum(fxl.mu, fx.mu, fyl.mu, fyh.mu, hx, hy);
                F[2] = flux_sum(fxl.mv, fx.mv, fyl.mv, fyh.mv, hx, hy);
                F[3] = flux_sum(fxl.E, fx.E, fyl.E, fyh.E, hx, hy);
            } else {
                F[0] = rfma(fx.r, hy, acc[0]);
                F[1] = rfma(fx.mu, hy, acc[1]);
                F[2] = rfma(fx.mv, hy, acc[2]);
                F[3] = rfma(fx.E, hy, acc[3]);
            }
            C4<double> q = base(sm, bm);
            if (MODE == FUSED_HEUN_B) {  // starts from the stage value's own Q
                const C4<double> t = cons_less(ring.z[sm][0][l], ring.z[sm][1][l], ring.z[sm][2][l], ring.z[sm][4][l],
                                               coef, F);
                q.r = 0.5 * (q.r + t.r);
                q.mu = 0.5 * (q.mu + t.mu);
                q.mv = 0.5 * (q.mv + t.mv);
                q.E = 0.5 * (q.E + t.E);
            } else {
                subtract(q, coef, F);
            }
            store_cell<R, MIXED, MODE>(a, f, g - 1, j, live, q, wm, cfl);
        }
        // ---- carry row g over -----------------------------------------------
        const C4<R> fb{__shfl_up_sync(ALL, fy.r, 1), __shfl_up_sync(ALL, fy.mu, 1), __shfl_up_sync(ALL, fy.mv, 1),
                       __shfl_up_sync(ALL, fy.E, 1)};
        if constexpr (MIXED) {
            fxl = fx, fyl = fb, fyh = fy;
        } else {
            acc[0] = three_fluxes(fx.r, fb.r, fy.r, hx, hy);
            acc[1] = three_fluxes(fx.mu, fb.mu, fy.mu, hx, hy);
            acc[2] = three_fluxes(fx.mv, fb.mv, fy.mv, hx, hy);
            acc[3] = three_fluxes(fx.E, fb.E, fy.E, hx, hy);
        }
        up = face_value<R>(h, gx, k.halfx, false, eos, k.igm1);
        if (iso && (wc | wp) != 0) up = own;
        wm = wc;
        wc = wp;
        const int t = sm;
        sm = sc;
        sc = sp;
        sp = sn;
        sn = t;
        const int tb = bm;
        bm = bc;
        bc = bp;
        bp = tb;
    }
    if (MODE != FUSED_HEUN_A) cfl.commit(f.slot_nxt);
}

// The split of the mesh into strips and segments: as many segments as fill
// the GPU's resident warps (148 SMs x MINB blocks x MARCH_WARPS) a whole
// number of times with at most 96 rows each, so that no last wave runs with a
// few warps (at 1700^2 a split 0.5 % over one wave took 243 us, this one
// fewer than the tile kernel's 236).
struct MarchSplit {
    int strips, rows;
};
inline MarchSplit march_split(const StructMesh &m, int minb) {
    const long long strips = (m.ny + MARCH_COLS - 1) / MARCH_COLS, cap = 148LL * minb * MARCH_WARPS;
    int rows = 0;
    for (long long waves = 1; waves <= 1 << 20; ++waves) {
        long long segs = waves * cap / strips;
        if (segs < 1) segs = 1;
        rows = (int)((m.nx + segs - 1) / segs);
        if (rows <= 96) break;
    }
    return MarchSplit{(int)strips, rows};
}
template <typename R, bool MIXED, int MODE, int MINB>
inline void launch_march(const SmfArgs &a, const Fields<R> &f, const MarchSplit &sp, cudaStream_t s) {
    const int segs = (a.mesh.nx + sp.rows - 1) / sp.rows;
    const unsigned blocks = (unsigned)(((long long)segs * sp.strips + MARCH_WARPS - 1) / MARCH_WARPS);
    const dim3 nt(32 * MARCH_WARPS);
    if (a.flux == FLUX_HLL)
        k_march<R, MIXED, MODE, true, MINB><<<blocks, nt, 0, s>>>(a, f, step_const<R>(a), sp.strips, sp.rows);
    else
        k_march<R, MIXED, MODE, false, MINB><<<blocks, nt, 0, s>>>(a, f, step_const<R>(a), sp.strips, sp.rows);
}
// The march runs van Albada 1, whose slope has a closed form.  The limiters that
// are formed from the general refit keep more values alive, and 128 registers a
// thread leave too few warps to cover their divisions: tile against march, FP64
// predictor-corrector at 2000^2 on smooth data, with the formulas both had at
// first: MC 402 / 461, minmod 365 / 395, van Leer 368 / 399 us (van Albada 1 338 /
// 314 at 2048^2); MIXED at 2048^2 MC 291 / 318.
inline bool march_limiter(int lim) { return lim == LIM_VANALBADA1; }
template <typename R, bool MIXED, int MINB>
inline void march_dispatch(const SmfArgs &a, const Fields<R> &f, int mode, const MarchSplit &sp, cudaStream_t s) {
    if (mode == FUSED_PC) launch_march<R, MIXED, FUSED_PC, MINB>(a, f, sp, s);
    else if (mode == FUSED_HEUN_A) launch_march<R, MIXED, FUSED_HEUN_A, MINB>(a, f, sp, s);
    else launch_march<R, MIXED, FUSED_HEUN_B, MINB>(a, f, sp, s);
}

}  // namespace tiled
}  // namespace zg
