// smf_parity.cu -- instantiates the gather-form FP64 kernels for both mesh
// accessors.  This file is compiled with -fmad=false: no multiply is fused
// into an add, matching the reference's x86-64 build, so results agree bit
// for bit with the oracle and the reference.
#include <cuda_runtime.h>

#include "smf_parity_tile.cuh"
#include "smf_slot_parity.cuh"
#include "smf_struct.cuh"

namespace zg {
namespace parity {

constexpr int BLOCK = 128;

static inline unsigned blocks(const SmfArgs &a, bool slots) {
    int n = slots ? a.smesh.n : a.mesh.n;
    return (unsigned)((n + BLOCK - 1) / BLOCK);
}

#define ZG_DISPATCH(KERNEL, ...)                                                                            \
    do {                                                                                                    \
        if (slots)                                                                                          \
            KERNEL<SlotAcc, BLOCK><<<blocks(a, true), BLOCK, 0, (cudaStream_t)stream>>>(__VA_ARGS__);      \
        else                                                                                                \
            KERNEL<StructAcc, BLOCK><<<blocks(a, false), BLOCK, 0, (cudaStream_t)stream>>>(__VA_ARGS__);   \
    } while (0)

void launch_dt(const SmfArgs &a, PrimPtr z, bool slots, void *stream) {
    SmfArgs b = a;
    b.z = z;
    ZG_DISPATCH(k_dt, b);
}
// The kernels that evaluate face fluxes, instantiated per flux family: HLLC
// and HLL without the other fluxes' code (the run-time switch over the
// eight fluxes of NumFlux::create costs registers and spills), the general
// switch for the rest.  The same operations either way.  On a rectangle the
// second order with HLLC or HLL runs in the tile kernels.
template <int FX>
static void flux1_fx(const SmfArgs &a, double *dt_next, bool slots, void *stream) {
    if (slots) k_flux1<SlotAcc, BLOCK, 1, FX><<<blocks(a, true), BLOCK, 0, (cudaStream_t)stream>>>(a, dt_next);
    else launch_after(k_flux1<StructAcc, BLOCK, 1, FX>, blocks(a, false), BLOCK, 0, (cudaStream_t)stream, a, dt_next);
}
template <int FX>
static void stage2_fx(const SmfArgs &a, double *dt_next, bool slots, void *stream) {
    if (slots) slotpar::k_stage2_4<FX><<<slotpar::blocks(a), slotpar::BLOCK, 0, (cudaStream_t)stream>>>(a, dt_next);
    else k_stage2<StructAcc, BLOCK, 1, -1><<<blocks(a, false), BLOCK, 0, (cudaStream_t)stream>>>(a, dt_next);
}
template <int FX>
static void heun_fx(const SmfArgs &a, PrimPtr zin, PrimPtr zout, bool final, double *dt_next, bool slots,
                    void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (slots) {
        if (final) k_heun<SlotAcc, BLOCK, true, 1, FX><<<blocks(a, true), BLOCK, 0, st>>>(a, zin, zout, dt_next);
        else k_heun<SlotAcc, BLOCK, false, 1, FX><<<blocks(a, true), BLOCK, 0, st>>>(a, zin, zout);
    } else {
        if (final) k_heun<StructAcc, BLOCK, true, 1, -1><<<blocks(a, false), BLOCK, 0, st>>>(a, zin, zout, dt_next);
        else k_heun<StructAcc, BLOCK, false, 1, -1><<<blocks(a, false), BLOCK, 0, st>>>(a, zin, zout);
    }
}
#define ZG_FLUX_FAMILY(FN, ...)                                        \
    do {                                                               \
        if (a.flux == FLUX_HLLC) FN<FLUX_HLLC>(__VA_ARGS__);           \
        else if (a.flux == FLUX_HLL) FN<FLUX_HLL>(__VA_ARGS__);        \
        else FN<-1>(__VA_ARGS__);                                      \
    } while (0)

void launch_flux1(const SmfArgs &a, double *dt_next, bool slots, void *stream) {
    ZG_FLUX_FAMILY(flux1_fx, a, dt_next, slots, stream);
}
void launch_grad(const SmfArgs &a, PrimPtr z, bool slots, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (slots) slotpar::k_grad4<false><<<slotpar::blocks(a), slotpar::BLOCK, 0, st>>>(a, z);
    else k_grad<StructAcc, BLOCK><<<blocks(a, false), BLOCK, 0, st>>>(a, z);
}
void launch_grad_stage1(const SmfArgs &a, bool slots, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (slots) {
        slotpar::k_grad4<true><<<slotpar::blocks(a), slotpar::BLOCK, 0, st>>>(a, a.z);
    } else {
        k_grad<StructAcc, BLOCK><<<blocks(a, false), BLOCK, 0, st>>>(a, a.z);
        k_stage1<StructAcc, BLOCK><<<blocks(a, false), BLOCK, 0, st>>>(a);
    }
}
void launch_stage2(const SmfArgs &a, double *dt_next, bool slots, void *stream) {
    ZG_FLUX_FAMILY(stage2_fx, a, dt_next, slots, stream);
}
void launch_heun(const SmfArgs &a, PrimPtr zin, PrimPtr zout, bool final, double *dt_next, bool slots, void *stream) {
    ZG_FLUX_FAMILY(heun_fx, a, zin, zout, final, dt_next, slots, stream);
}

// Rows of a tile and blocks per SM of the tile kernels (smf_parity_tile.cuh).
#ifndef ZG_PTILE_TH
#define ZG_PTILE_TH 12
#endif
#ifndef ZG_PTILE_MINB
#define ZG_PTILE_MINB 2
#endif
template <int MODE, int LIM>
static void tile_flux(const ptile::Args &A, cudaStream_t s) {
    if (A.a.flux == FLUX_HLL) ptile::launch<MODE, LIM, true, ZG_PTILE_TH, ZG_PTILE_MINB>(A, s);
    else ptile::launch<MODE, LIM, false, ZG_PTILE_TH, ZG_PTILE_MINB>(A, s);
}
template <int MODE>
static void tile_lim(const ptile::Args &A, cudaStream_t s) {
    switch (A.a.limiter) {  // the common limiters are compiled in
        case LIM_VANALBADA1: tile_flux<MODE, LIM_VANALBADA1>(A, s); break;
        case LIM_MC: tile_flux<MODE, LIM_MC>(A, s); break;
        case LIM_MINMOD: tile_flux<MODE, LIM_MINMOD>(A, s); break;
        case LIM_VANLEER: tile_flux<MODE, LIM_VANLEER>(A, s); break;
        default: tile_flux<MODE, -1>(A, s); break;
    }
}
void launch_tile(const SmfArgs &a, const ptile::Axis &x, const ptile::Axis &y, int stage, PrimPtr zin, PrimPtr zout,
                 const double *dt_in, double *dt_next, void *stream) {
    const ptile::Args A{a, x, y, zin, zout, dt_in, dt_next};
    const cudaStream_t s = (cudaStream_t)stream;
    if (stage == ptile::PC) tile_lim<ptile::PC>(A, s);
    else if (stage == ptile::HEUN_A) tile_lim<ptile::HEUN_A>(A, s);
    else tile_lim<ptile::HEUN_B>(A, s);
}
void launch_flags(const SmfArgs &a, int *flags, bool slots, void *stream) { ZG_DISPATCH(k_flags, a, flags); }

}  // namespace parity
}  // namespace zg
