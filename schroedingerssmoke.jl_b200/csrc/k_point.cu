// Pointwise and nearest-neighbour kernels of the ISF API that are not fused
// into an FFT pass or a stencil: the standalone forms of normalize_psi,
// restrict_velocity!, isjet, the staggered sharp and div! (from the velocity
// grid), and layout conversions of the handle's padded velocity grid.
#include "isf_launch.h"

namespace isf {

static inline unsigned grid_for(long long n, int block) {
    long long b = (n + block - 1) / block;
    const long long cap = 148LL * 32;  // grid-stride beyond 32 CTAs per SM
    return (unsigned)(b < cap ? b : cap);
}

// normalize_psi broadcast (parallel.jl:162-165, examples/benchmark.jl:50)
__global__ void k_normalize(float4* __restrict__ psi, long long N) {
    pdl_enter();
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < N; c += (long long)gridDim.x * blockDim.x)
        psi[c] = normalize4(psi[c]);
}

// restrict_velocity! (particles.jl:25-27) in place; a batch launch (jets !=
// null) restricts simulation blockIdx.z mod nsim with its jets entry.  Only
// the nozzle's cells of psi are read and written.  A nozzle given by its geometry
// takes 3.0 us on 64x32x32, 4.6 on 128x64x64 and 7.8 on 256x128x128 (a quarter of
// the box wide); with a mask, whose bytes every column reads plane by plane, 3.3,
// 5.1 and 12.  It stands before the projection's passes: fused into the
// divergence stencil and the gauge pass, both evaluated the restriction for
// every load, and a nozzle projection took 112 us at 256x128x128 instead of 98, 33
// on 128x64x64 instead of 29 and 22.6 on 64x32x32 instead of 18.5.
__global__ void __launch_bounds__(256) k_restrict(Grid g, float4* __restrict__ psi, JetArgs j,
                                                  const JetArgs* __restrict__ jets, int nsim, long long bs_psi) {
    pdl_enter();
    const int sim = blockIdx.z % nsim, z0 = blockIdx.z / nsim, dz = gridDim.z / nsim;
    if (jets) j = jets[sim];
    restrict_columns(g, psi + sim * bs_psi, j, cell_x(g), cell_y(g), z0, dz);
}

// isjet.(isf.positions, ...) (particles.jl:6-10, examples/benchmark.jl:26)
__global__ void __launch_bounds__(256) k_isjet(Grid g, uint8_t* __restrict__ out, float c0, float c1, float c2, float len,
                                               float rad) {
    pdl_enter();
    const float cen[3] = {c0, c1, c2};
    const int x = cell_x(g), y = cell_y(g);
    if (x >= g.n[0] || y >= g.n[1]) return;
    for (int z = blockIdx.z; z < g.n[2]; z += gridDim.z) {
        const float px = __fmul_rn((float)x, g.d[0]), py = __fmul_rn((float)y, g.d[1]), pz = __fmul_rn((float)z, g.d[2]);
        out[cell(g, x, y, z)] = isjet_f32(px, py, pz, cen, len, rad) ? 1 : 0;
    }
}

// staggered sharp on the handle's padded velocity grid (examples/benchmark.jl:61-63)
__global__ void k_sharp(Grid g, float4* __restrict__ vel) {
    pdl_enter();
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < g.NP; c += (long long)gridDim.x * blockDim.x) {
        float4 v = vel[c];
        v.x = __fmul_rn(v.x, g.dinv[0]);
        v.y = __fmul_rn(v.y, g.dinv[1]);
        v.z = __fmul_rn(v.z, g.dinv[2]);
        vel[c] = v;
    }
}

// div! (parallel.jl:131-152) from the padded velocity grid
__global__ void __launch_bounds__(256) k_div(Grid g, const float4* __restrict__ vel, float* __restrict__ f) {
    pdl_enter();
    const int x = cell_x(g), y = cell_y(g);
    if (x >= g.n[0] || y >= g.n[1]) return;
    const int xm = (x == 0) ? g.n[0] - 1 : x - 1, ym = (y == 0) ? g.n[1] - 1 : y - 1;
    for (int z = blockIdx.z; z < g.n[2]; z += gridDim.z) {
        const int zm = (z == 0) ? g.n[2] - 1 : z - 1;
        const float4 v = vel[pcell(g, x, y, z)];
        const float t0 = (v.x - vel[pcell(g, xm, y, z)].x) * g.inv_d2[0];
        const float t1 = (v.y - vel[pcell(g, x, ym, z)].y) * g.inv_d2[1];
        const float t2 = (v.z - vel[pcell(g, x, y, zm)].z) * g.inv_d2[2];
        f[cell(g, x, y, z)] = (t0 + t1) + t2;
    }
}

// The velocity as AoS float3: the 384 bytes of a warp's 32 cells (of one row,
// or of the rows of a narrower tile) leave as three stores of whole 128-byte
// lines, each lane fetching the components of its words from the lanes that
// loaded them (12-byte strided stores touch every sector three times).
__global__ void __launch_bounds__(256) k_vel_to_aos(Grid g, const float4* __restrict__ vel, float* __restrict__ aos) {
    pdl_enter();
    const int lane = threadIdx.x & 31, first = threadIdx.x & ~31;
    const int x = cell_x(g), y = cell_y(g);
    if (cell_y(g, (int)blockIdx.y, first) >= g.n[1]) return;  // whole warps
    for (int z = blockIdx.z; z < g.n[2]; z += gridDim.z) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (x < g.n[0] && y < g.n[1]) v = vel[pcell(g, x, y, z)];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int w = lane + 32 * k, from = w / 3, comp = w - 3 * from;
            const float vx = __shfl_sync(0xffffffffu, v.x, from), vy = __shfl_sync(0xffffffffu, v.y, from),
                        vz = __shfl_sync(0xffffffffu, v.z, from);
            const int xf = cell_x(g, (int)blockIdx.x, first + from), yf = cell_y(g, (int)blockIdx.y, first + from);
            if (xf < g.n[0] && yf < g.n[1])
                aos[3 * cell(g, xf, yf, z) + comp] = comp == 0 ? vx : (comp == 1 ? vy : vz);
        }
    }
}

__global__ void __launch_bounds__(256) k_vel_from_aos(Grid g, const float* __restrict__ aos, float4* __restrict__ vel) {
    pdl_enter();
    const int x = cell_x(g), y = cell_y(g);
    if (x >= g.n[0] || y >= g.n[1]) return;
    for (int z = blockIdx.z; z < g.n[2]; z += gridDim.z) {
        const long long c = cell(g, x, y, z);
        pstore(g, vel, x, y, z, make_float3(aos[3 * c + 0], aos[3 * c + 1], aos[3 * c + 2]));
    }
}

__global__ void k_scale_c(float2* __restrict__ a, long long N, float s) {
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < N; c += (long long)gridDim.x * blockDim.x)
        a[c] = cscale(a[c], s);
}

// cells of psi with a non-finite component, added into *count
__global__ void k_count_nonfinite(const float4* __restrict__ psi, long long N, unsigned long long* __restrict__ count) {
    unsigned n = 0;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < N; c += (long long)gridDim.x * blockDim.x) {
        const float4 v = psi[c];
        n += (isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w)) ? 0u : 1u;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_down_sync(0xffffffffu, n, o);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(count, (unsigned long long)n);
}

cudaError_t launch_count_nonfinite(const Grid& g, const float4* psi, unsigned long long* count, cudaStream_t s) {
    k_count_nonfinite<<<grid_for(g.N, 256), 256, 0, s>>>(psi, g.N, count);
    return cudaGetLastError();
}

cudaError_t launch_scale_c(const Grid& g, float2* a, float s, cudaStream_t st) {
    k_scale_c<<<grid_for(g.N, 256), 256, 0, st>>>(a, g.N, s);
    return cudaGetLastError();
}
cudaError_t launch_normalize(const Grid& g, float4* psi, cudaStream_t s) {
    return launch_pdl(k_normalize, dim3(grid_for(g.N, 256)), dim3(256), 0, s, psi, g.N);
}
cudaError_t launch_restrict(const Grid& g, float4* psi, const JetArgs& j, cudaStream_t s) {
    return launch_pdl(k_restrict, cell_grid(g), dim3(256), 0, s, g, psi, j, (const JetArgs*)nullptr, 1, 0LL);
}
cudaError_t launch_restrict_batch(const Grid& g, float4* psi, const JetArgs* jets, int nsim, long long bs_psi,
                                  cudaStream_t s) {
    dim3 grid = cell_grid(g);
    grid.z = (grid.z / (unsigned)nsim > 0 ? grid.z / (unsigned)nsim : 1u) * (unsigned)nsim;
    return launch_pdl(k_restrict, grid, dim3(256), 0, s, g, psi, JetArgs{}, jets, nsim, bs_psi);
}
cudaError_t launch_isjet(const Grid& g, uint8_t* out, const float* cen, float len, float rad, cudaStream_t s) {
    return launch_pdl(k_isjet, cell_grid(g), dim3(256), 0, s, g, out, cen[0], cen[1], cen[2], len, rad);
}
cudaError_t launch_sharp(const Grid& g, float* vel, cudaStream_t s) {
    return launch_pdl(k_sharp, dim3(grid_for(g.NP, 256)), dim3(256), 0, s, g, reinterpret_cast<float4*>(vel));
}
cudaError_t launch_div(const Grid& g, const float* vel, float* f, cudaStream_t s) {
    return launch_pdl(k_div, cell_grid(g), dim3(256), 0, s, g, reinterpret_cast<const float4*>(vel), f);
}
cudaError_t launch_vel_to_aos(const Grid& g, const float* vel, float* aos, cudaStream_t s) {
    return launch_pdl(k_vel_to_aos, cell_grid(g), dim3(256), 0, s, g, reinterpret_cast<const float4*>(vel), aos);
}
cudaError_t launch_vel_from_aos(const Grid& g, const float* aos, float* vel, cudaStream_t s) {
    return launch_pdl(k_vel_from_aos, cell_grid(g), dim3(256), 0, s, g, aos, reinterpret_cast<float4*>(vel));
}

}  // namespace isf
