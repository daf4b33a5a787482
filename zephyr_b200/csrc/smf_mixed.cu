// smf_mixed.cu -- the tiled MIXED kernels: FP32 reconstruction and Riemann
// fluxes (approximate single-precision division and square root allowed),
// FP64 conserved state, accumulation, update and dt.
#include "smf_fused.cuh"
#include "smf_march.cuh"
#include "smf_tiled.cuh"
#include "smf_tiled_launch.h"

namespace zg {
namespace mixed {

using tiled::Fields;
// Tile shapes and minimum resident blocks per SM.  The kernels are latency-
// bound, so residency decides their speed: the minimum-block counts cap the
// registers per thread (spilling a few bytes in the gradient pass) and were
// chosen by timing the 2048^2 step over a sweep of these values on a B200.
#ifndef ZG_MIXED_TY
#define ZG_MIXED_TY 8
#endif
#ifndef ZG_MIXED_GY
#define ZG_MIXED_GY 4
#endif
#ifndef ZG_MIXED_FACES_MINB
#define ZG_MIXED_FACES_MINB 6
#endif
#ifndef ZG_MIXED_GP_MINB
#define ZG_MIXED_GP_MINB 12
#endif
constexpr int BLOCK = 128, TX = 32, TY = ZG_MIXED_TY;  // faces: 32 x TY threads, 31 x (TY - 1) interior cells
constexpr int GX = 32, GY = ZG_MIXED_GY;               // gradients + predictor: 32 x GY cells
constexpr int FMINB = ZG_MIXED_FACES_MINB, GMINB = ZG_MIXED_GP_MINB;

static inline unsigned blocks(int n) { return (unsigned)((n + BLOCK - 1) / BLOCK); }

void launch_cfl(const SmfArgs &a, const Fields<float> &f, void *stream) {
    tiled::k_cfl<float, BLOCK><<<blocks(a.mesh.n), BLOCK, 0, (cudaStream_t)stream>>>(a, f);
}

template <int LIM>
static void grad_predict(const SmfArgs &a, const Fields<float> &f, bool predict, cudaStream_t s) {
    dim3 block(GX, GY);
    dim3 grid((a.mesh.ny + GX - 1) / GX, (a.mesh.nx + GY - 1) / GY);
    if (predict)
        tiled::k_grad_predict<float, true, true, LIM, GX, GY, GMINB><<<grid, block, 0, s>>>(a, f);
    else
        tiled::k_grad_predict<float, true, false, LIM, GX, GY, GMINB><<<grid, block, 0, s>>>(a, f);
}

void launch_grad_predict(const SmfArgs &a, const Fields<float> &f, bool predict, void *stream) {
    cudaStream_t s = (cudaStream_t)stream;
    switch (a.limiter) {  // the common limiters are compiled in; others are selected at run time
        case LIM_VANALBADA1: grad_predict<LIM_VANALBADA1>(a, f, predict, s); break;
        case LIM_MC: grad_predict<LIM_MC>(a, f, predict, s); break;
        case LIM_MINMOD: grad_predict<LIM_MINMOD>(a, f, predict, s); break;
        default: grad_predict<-1>(a, f, predict, s); break;
    }
}

void launch_faces(const SmfArgs &a, const Fields<float> &f, int mode, void *stream) {
    dim3 block(TX, TY);
    dim3 grid((a.mesh.ny + TX - 2) / (TX - 1), (a.mesh.nx + TY - 2) / (TY - 1));
    cudaStream_t s = (cudaStream_t)stream;
    // HLLC and HLL get kernels without the other fluxes' code (registers)
    if (a.flux == FLUX_HLLC || a.flux == FLUX_HLL) {
        switch (mode) {
            case 0:
                if (early_first_order(grid)) launch_after(tiled::k_faces<float, true, 0, TX, TY, FMINB, false>, grid, block, 0, s, a, f);
                else tiled::k_faces<float, true, 0, TX, TY, FMINB, false><<<grid, block, 0, s>>>(a, f);
                break;
            case 1: tiled::k_faces<float, true, 1, TX, TY, FMINB, false><<<grid, block, 0, s>>>(a, f); break;
            case 2: tiled::k_faces<float, true, 2, TX, TY, FMINB, false><<<grid, block, 0, s>>>(a, f); break;
            default: tiled::k_faces<float, true, 3, TX, TY, FMINB, false><<<grid, block, 0, s>>>(a, f); break;
        }
        return;
    }
    switch (mode) {
        case 0:
                if (early_first_order(grid)) launch_after(tiled::k_faces<float, true, 0, TX, TY, FMINB>, grid, block, 0, s, a, f);
                else tiled::k_faces<float, true, 0, TX, TY, FMINB><<<grid, block, 0, s>>>(a, f);
                break;
        case 1: tiled::k_faces<float, true, 1, TX, TY, FMINB><<<grid, block, 0, s>>>(a, f); break;
        case 2: tiled::k_faces<float, true, 2, TX, TY, FMINB><<<grid, block, 0, s>>>(a, f); break;
        default: tiled::k_faces<float, true, 3, TX, TY, FMINB><<<grid, block, 0, s>>>(a, f); break;
    }
}

void launch_to_mixed(int n, PrimPtr z, const Fields<float> &f, void *stream) {
    tiled::k_to_mixed<BLOCK><<<blocks(n), BLOCK, 0, (cudaStream_t)stream>>>(n, z, f);
}

void launch_to_prim(int n, const Fields<float> &f, EosD eos, PrimPtr z, void *stream) {
    tiled::k_to_prim<BLOCK><<<blocks(n), BLOCK, 0, (cudaStream_t)stream>>>(n, f, eos, z);
}

// Fused single-pass stages (smf_fused.cuh).
#ifndef ZG_MIXED_FUSED_TH
#define ZG_MIXED_FUSED_TH 14
#endif
#ifndef ZG_MIXED_FUSED_MINB
#define ZG_MIXED_FUSED_MINB 2
#endif
#ifndef ZG_MIXED_MARCH_MINB
#define ZG_MIXED_MARCH_MINB 5
#endif
// The form by size, measured on B200 (us per step of van Albada HLLC, march / tile):
//   predictor-corrector  1700^2 177 / 173, 2048^2 246 / 248, 3072^2 514 / 544, 4096^2 889 / 960, 6000x1200 426 / 417
//   Heun                 896^2 74 / 73, 1024^2 92 / 98, 2048^2 304 / 375, 3072^2 631 / 824
// (the predictor's FP64 half makes the march's registers the limit).  Small
// meshes take tiles of 4 rows instead of 14, as in the FP64 form.
constexpr int MARCH_MIN_ROWS_PC = 48, MARCH_MIN_ROWS_HEUN = 11;
void launch_step(const SmfArgs &a, const Fields<float> &f, int mode, void *stream) {
    const cudaStream_t s = (cudaStream_t)stream;
    const tiled::MarchSplit sp = tiled::march_split(a.mesh, ZG_MIXED_MARCH_MINB);
    constexpr int TH = ZG_MIXED_FUSED_TH;
    if (tiled::march_limiter(a.limiter) && a.mesh.xper && a.mesh.yper &&
        sp.rows >= (mode == tiled::FUSED_PC ? MARCH_MIN_ROWS_PC : MARCH_MIN_ROWS_HEUN))
        tiled::march_dispatch<float, true, ZG_MIXED_MARCH_MINB>(a, f, mode, sp, s);
    else if (tiled::small_tiles(a.mesh, 4))
        tiled::fused_dispatch<float, true, tiled::SMALL_TH, tiled::SMALL_MINB>(a, f, mode, s);
    else
        tiled::fused_dispatch<float, true, TH, ZG_MIXED_FUSED_MINB>(a, f, mode, s);
}

}  // namespace mixed
}  // namespace zg
