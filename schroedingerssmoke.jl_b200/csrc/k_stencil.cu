// z-marching stencil kernels of the velocity one-form (the body is in
// isf_stencil.cuh): k_stencil for the one-form, k_stencil_div for the
// divergence.
#include "isf_stencil.cuh"

namespace isf {

// Both stencils are compiled for 4 resident CTAs per SM (at most 64
// registers).  The one-form stencil: 60 registers and 185 instructions per
// cell left to ptxas (35.9 us at 256x128x128), 64 and 181 capped (34.6 us).
template <int OP, bool JET, bool SHARP = false>
__global__ void __launch_bounds__(st::BX* st::TY, 4) k_stencil(StencilArgs a) {
    pdl_enter();
    __shared__ StencilSmem<OP> sm;
    stencil_body<OP, JET, SHARP>(a, launch_blk(), sm);
}

// The div stencil: 48 registers and 235 instructions per cell left to
// ptxas (40.9 us at 256x128x128), 64 and 200 capped (37.9 us).
template <bool JET>
__global__ void __launch_bounds__(st::BX* st::TY, 4) k_stencil_div(StencilArgs a) {
    pdl_enter();
    __shared__ StencilSmem<ST_DIV> sm;
    stencil_body<ST_DIV, JET>(a, launch_blk(), sm);
}

// z planes per CTA: as many as leave about 1024 CTAs (of 592 resident ones),
// 1 to kPlanes.  A CTA walks its planes one after another, so on a small grid
// the walk is the whole launch: with 8 planes 64x32x32 made 16 CTAs.  Measured
// (one-form stencil / projection / nozzle projection, us per call, 8 planes
// -> the rule's): 64x32x32 7.7 / 23.6 / 35.7 -> 6.0 / 15.6 / 24.2 (1 plane),
// 128x64x64 16.3 / 42.8 / 46.1 -> 6.6 / 25.7 / 34.6 (1), 160x96x80 17.9 / 56.4 /
// 73.2 -> 11.7 / 48.9 / 64.3 (2), 200x100x112 23.0 / 79.1 / 105.5 -> 20.5 / 75.5 /
// 103 (5), 256x128x128 unchanged (8; 1 plane there: 44.7 / 114 / 158).
static int planes_of(const Grid& g, long long columns) {
    const long long sz = columns * g.n[2] / 1024;
    return (int)(sz < 1 ? 1 : (sz > st::kPlanes ? st::kPlanes : sz));
}

cudaError_t launch_stencil(int op, const StencilArgs& args, cudaStream_t s) {
    StencilArgs a = args;
    const int nsim = a.nsim > 1 ? a.nsim : 1;
    const unsigned bx = (unsigned)((a.g.n[0] + st::BX - 1) / st::BX), by = (unsigned)((a.g.n[1] + st::BY - 1) / st::BY);
    a.sz = planes_of(a.g, (long long)bx * by * nsim);
    const dim3 grid(bx, by, (unsigned)(((a.g.n[2] + a.sz - 1) / a.sz) * nsim));
    const dim3 blk(st::BX * st::TY);
    const bool jet = a.use_jet != 0;
    if (op == ST_DIV)
        return jet ? launch_pdl(k_stencil_div<true>, grid, blk, 0, s, a)
                   : launch_pdl(k_stencil_div<false>, grid, blk, 0, s, a);
    if (op == ST_VEL) {
        if (a.sharp)
            return jet ? launch_pdl(k_stencil<ST_VEL, true, true>, grid, blk, 0, s, a)
                       : launch_pdl(k_stencil<ST_VEL, false, true>, grid, blk, 0, s, a);
        return jet ? launch_pdl(k_stencil<ST_VEL, true>, grid, blk, 0, s, a)
                   : launch_pdl(k_stencil<ST_VEL, false>, grid, blk, 0, s, a);
    }
    return cudaErrorInvalidValue;
}

}  // namespace isf
