// z-marching stencil kernels of the velocity one-form (the body is in
// isf_stencil.cuh): k_stencil for the one-form, k_stencil_div for the
// divergence.
#include "isf_stencil.cuh"

namespace isf {

// Both stencils are compiled for 4 resident CTAs per SM (at most 64
// registers).  The one-form stencil: 60 registers and 185 instructions per
// cell left to ptxas (35.9 us at 256x128x128), 64 and 181 capped (34.6 us).
template <int OP, bool SHARP = false>
__global__ void __launch_bounds__(st::BX* st::TY, 4) k_stencil(StencilArgs a) {
    pdl_enter();
    __shared__ StencilSmem<OP> sm;
    stencil_body<OP, SHARP>(a, launch_blk(), sm);
}

// The div stencil: 48 registers and 235 instructions per cell left to
// ptxas (40.9 us at 256x128x128), 64 and 200 capped (37.9 us).
__global__ void __launch_bounds__(st::BX* st::TY, 4) k_stencil_div(StencilArgs a) {
    pdl_enter();
    __shared__ StencilSmem<ST_DIV> sm;
    stencil_body<ST_DIV>(a, launch_blk(), sm);
}

// z planes per CTA: as many as leave about one wave of the 592 resident CTAs,
// 1 to kPlanes.  A CTA walks its planes one after another, so on a small grid
// the walk is the whole launch (with 8 planes 64x32x32 made 16 CTAs); every
// CTA also loads a plane more than it writes and evaluates an extra z edge, so
// fewer planes cost more in all, which shows when other streams keep the GPU
// busy.  Jet step, us alone / three simulations side by side: 128x64x64 95.6 /
// 59.5 at 1 plane, 100 / 53.7 at 2 (the rule's), 124 / 62.4 at 8; 96x96x96 171 /
// 106, 162 / 93 at 3 (the rule's), 191 / 106; 256x128x128 419 / 430 at 1, 347 /
// 346 at 8 (the rule's).  One-form stencil on 64x32x32 7.7 at 8, 6.0 at 1.
static int planes_of(const Grid& g, long long columns) {
    const long long sz = (columns * g.n[2] + 296) / 592;
    return (int)(sz < 1 ? 1 : (sz > st::kPlanes ? st::kPlanes : sz));
}

cudaError_t launch_stencil(int op, const StencilArgs& args, cudaStream_t s) {
    StencilArgs a = args;
    const int nsim = a.nsim > 1 ? a.nsim : 1;
    const unsigned bx = (unsigned)((a.g.n[0] + st::BX - 1) / st::BX), by = (unsigned)((a.g.n[1] + st::BY - 1) / st::BY);
    a.sz = planes_of(a.g, (long long)bx * by * nsim);
    const dim3 grid(bx, by, (unsigned)(((a.g.n[2] + a.sz - 1) / a.sz) * nsim));
    const dim3 blk(st::BX * st::TY);
    if (op == ST_DIV) return launch_pdl(k_stencil_div, grid, blk, 0, s, a);
    if (op == ST_VEL)
        return a.sharp ? launch_pdl(k_stencil<ST_VEL, true>, grid, blk, 0, s, a)
                       : launch_pdl(k_stencil<ST_VEL>, grid, blk, 0, s, a);
    return cudaErrorInvalidValue;
}

}  // namespace isf
