// Adjoint (reverse-mode) kernels of the ISF time step.
//
// Convention: psi is treated as 4 reals per cell; for a complex component z
// the adjoint zbar holds (dL/dRe z, dL/dIm z), so dL = Re(conj(zbar) dz)
// summed over components.  Each kernel maps the adjoint of a stage's output
// to the adjoint of its input (and of its parameters) at the forward input
// the caller passes; none of them is the reference's, which has no
// derivatives -- they differentiate its operators:
//   normalize_psi          parallel.jl:162-165
//   gauge_transform        parallel.jl:125-129 (real q)
//   velocity_one_form/div  parallel.jl:100-152 (angle derivative
//                          d angle(z) = Im(conj(z) dz) / |z|^2)
//   restrict_kernel        particles.jl:12-20
//   staggered_advect       parallel.jl:197-246 (RK4 and the unnormalised
//                          staggered interpolation, differentiated inside a
//                          cell; the jumps at cell faces carry no derivative)
#include "isf_launch.h"
#include "isf_particles.cuh"

namespace isf {

namespace {

inline unsigned grid_n(long long n, int block) {
    long long b = (n + block - 1) / block;
    const long long cap = 148LL * 32;
    return (unsigned)(b < cap ? b : cap);
}

// block-wide sum of n doubles into acc[] (one atomicAdd per value per block)
template <int NV>
__device__ __forceinline__ void block_sum_add(double (&v)[NV], double* acc) {
    __shared__ double red[NV][32];
#pragma unroll
    for (int k = 0; k < NV; ++k)
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) red[k][warp] = v[k];
    __syncthreads();
    if (warp == 0) {
        const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            double s = lane < nw ? red[k][lane] : 0.0;
            for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
            if (lane == 0 && s != 0.0) atomicAdd(&acc[k], s);
        }
    }
}

}  // namespace

// out = in exp(-i q) with a real q per cell (the forward gauge on its own)
__global__ void k_gauge(const float4* __restrict__ in, const float* __restrict__ q, float4* __restrict__ out,
                        long long N) {
    pdl_enter();
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < N; c += (long long)gridDim.x * blockDim.x)
        out[c] = gauge4(in[c], q[c]);
}

// out = normalize_psi(in)
__global__ void k_normalize_to(const float4* __restrict__ in, float4* __restrict__ out, long long N) {
    pdl_enter();
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < N; c += (long long)gridDim.x * blockDim.x)
        out[c] = normalize4(in[c]);
}

// out = restrict_velocity(in) (every cell written).  With q, in is gauged
// first and mid gets what is restricted: mid = in exp(-i q), out = restrict(mid)
template <bool GAUGE>
__global__ void __launch_bounds__(256) k_restrict_to(Grid g, const float4* __restrict__ in, const float* __restrict__ q,
                                                     float4* __restrict__ mid, float4* __restrict__ out, JetArgs j) {
    pdl_enter();
    const int x = cell_x(g), y = cell_y(g);
    if (x >= g.n[0] || y >= g.n[1]) return;
    for (int z = blockIdx.z; z < g.n[2]; z += gridDim.z) {
        const long long c = cell(g, x, y, z);
        float4 v = in[c];
        if constexpr (GAUGE) {
            v = gauge4(v, q[c]);
            mid[c] = v;
        }
        out[c] = jet_cell(g, j, x, y, z, c) ? restrict_value(g, j, x, y, z, v) : v;
    }
}

// normalize: out = v / |v| (4 reals); bar_in = (bar_out - b (b . bar_out)) / |v|
__global__ void k_adj_normalize(const float4* __restrict__ psi_in, float4* __restrict__ bar, long long N) {
    pdl_enter();
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < N; c += (long long)gridDim.x * blockDim.x) {
        const float4 v = psi_in[c];
        const float r = sqrtf(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
        if (!(r > 0.f)) {
            bar[c] = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        const float ir = 1.0f / r;
        const float4 b = make_float4(v.x * ir, v.y * ir, v.z * ir, v.w * ir);
        const float4 g = bar[c];
        const float d = b.x * g.x + b.y * g.y + b.z * g.z + b.w * g.w;
        bar[c] = make_float4((g.x - b.x * d) * ir, (g.y - b.y * d) * ir, (g.z - b.z * d) * ir, (g.w - b.w * d) * ir);
    }
}

// gauge: out = in exp(-i q).  qbar = sum_k Im(conj(bar_k) out_k);
// bar_in = bar_out exp(+i q)
__global__ void __launch_bounds__(256) k_adj_gauge(const float4* __restrict__ psi_in, const float* __restrict__ q,
                                                   float4* __restrict__ bar, float* __restrict__ qbar, long long N) {
    pdl_enter();
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < N; c += (long long)gridDim.x * blockDim.x) {
        const float qc = q[c];
        const float4 v = psi_in[c];
        const float4 g = bar[c];
        float s, co;
        sincosf(qc, &s, &co);
        const float4 o = make_float4(v.x * co + v.y * s, v.y * co - v.x * s, v.z * co + v.w * s, v.w * co - v.z * s);
        qbar[c] = (g.x * o.y - g.y * o.x) + (g.z * o.w - g.w * o.z);
        bar[c] = make_float4(g.x * co - g.y * s, g.x * s + g.y * co, g.z * co - g.w * s, g.z * s + g.w * co);
    }
}

// Transpose of the one-form at psi, added into bar.  The one-form's cotangent
// per edge (cell i, axis a) is
//   DIV:  wbar_a[i] = s_a (fbar[i] - fbar[i + e_a])   (through div, s_a = 1/d_a^2)
//   else: wbar_a[i] = s_a ubar_a[i]                    (velocity, s_a = hbar [/ d_a])
// and w_a[i] = angle(z), z = sum_k conj(psi_k[i]) psi_k[i+e_a], contributes
//   bar_k[i]     += wbar (-i conj(z) psi_k[i+e_a]) / |z|^2
//   bar_k[i+e_a] += wbar ( i z psi_k[i]) / |z|^2
// gathered here per cell from the edges i and i - e_a.  The velocity cotangent
// lives on the padded grid; a cell on a low face collects the periodic copies
// of its value on the +faces as it reads.  Bound by the seven psi cells and
// the neighbours' cotangents, most of them L1 hits of the tile.
struct AdjOneFormArgs {
    Grid g;
    const float4* psi;
    float4* bar;
    const float* fbar;   // DIV
    const float4* ubar;  // padded velocity cotangent
    float s[3];
};

// the cotangent of cell (x, y, z)'s velocity: its own entry and those of its
// periodic copies on the +faces
__device__ __forceinline__ float4 ubar_at(const Grid& g, const float4* __restrict__ u, int x, int y, int z) {
    const int p = pcell(g, x, y, z);
    float4 v = u[p];
    const bool cx = x == 0, cy = y == 0, cz = z == 0;
    if (cx | cy | cz) {
        const int ox = g.n[0], oy = g.n[1] * g.pnx, oz = g.n[2] * g.pnxy;
#pragma unroll
        for (int k = 1; k < 8; ++k) {
            const bool on = (!(k & 1) || cx) && (!(k & 2) || cy) && (!(k & 4) || cz);
            if (on) v = cadd(v, u[p + ((k & 1) ? ox : 0) + ((k & 2) ? oy : 0) + ((k & 4) ? oz : 0)]);
        }
    }
    return v;
}

template <bool DIV>
__global__ void __launch_bounds__(256) k_adj_oneform(AdjOneFormArgs A) {
    pdl_enter();
    const Grid& g = A.g;
    const int nx = g.n[0], ny = g.n[1], nz = g.n[2];
    const int x = cell_x(g), y = cell_y(g);
    if (x >= nx || y >= ny) return;
    const int xp = (x + 1 == nx) ? 0 : x + 1, xm = (x == 0) ? nx - 1 : x - 1;
    const int yp = (y + 1 == ny) ? 0 : y + 1, ym = (y == 0) ? ny - 1 : y - 1;
    for (int z = blockIdx.z; z < nz; z += gridDim.z) {
        const int zp = (z + 1 == nz) ? 0 : z + 1, zm = (z == 0) ? nz - 1 : z - 1;
        const int cp[3] = {(int)cell(g, xp, y, z), (int)cell(g, x, yp, z), (int)cell(g, x, y, zp)};
        const int cm[3] = {(int)cell(g, xm, y, z), (int)cell(g, x, ym, z), (int)cell(g, x, y, zm)};
        const int c = (int)cell(g, x, y, z);
        const float4 p0 = A.psi[c];
        float4 acc = A.bar[c];
        float wh[3], wp[3];
        if constexpr (DIV) {
            const float f0 = A.fbar[c];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                wh[a] = A.s[a] * (f0 - A.fbar[cp[a]]);
                wp[a] = A.s[a] * (A.fbar[cm[a]] - f0);
            }
        } else {
            const float4 u = ubar_at(g, A.ubar, x, y, z);
            wh[0] = A.s[0] * u.x;
            wh[1] = A.s[1] * u.y;
            wh[2] = A.s[2] * u.z;
            wp[0] = A.s[0] * ubar_at(g, A.ubar, xm, y, z).x;
            wp[1] = A.s[1] * ubar_at(g, A.ubar, x, ym, z).y;
            wp[2] = A.s[2] * ubar_at(g, A.ubar, x, y, zm).z;
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float4 pp = A.psi[cp[a]], pm = A.psi[cm[a]];
            const float2 z1 = pair_z(p0, pp);
            const float n1 = z1.x * z1.x + z1.y * z1.y;
            if (n1 > 0.f && wh[a] != 0.f) {
                const float t = wh[a] / n1;
                // -i conj(z1) pp_k
                float mx = z1.x * pp.x + z1.y * pp.y, my = z1.x * pp.y - z1.y * pp.x;
                acc.x += t * my;
                acc.y -= t * mx;
                mx = z1.x * pp.z + z1.y * pp.w;
                my = z1.x * pp.w - z1.y * pp.z;
                acc.z += t * my;
                acc.w -= t * mx;
            }
            const float2 z2 = pair_z(pm, p0);
            const float n2 = z2.x * z2.x + z2.y * z2.y;
            if (n2 > 0.f && wp[a] != 0.f) {
                const float t = wp[a] / n2;
                // i z2 pm_k
                float mx = z2.x * pm.x - z2.y * pm.y, my = z2.x * pm.y + z2.y * pm.x;
                acc.x -= t * my;
                acc.y += t * mx;
                mx = z2.x * pm.z - z2.y * pm.w;
                my = z2.x * pm.w + z2.y * pm.z;
                acc.z -= t * my;
                acc.w += t * mx;
            }
        }
        A.bar[c] = acc;
    }
}

// restrict_kernel: in the nozzle out_k = |in_k| exp(i phi), phi = phase(k, x)
// - omega t.  bar_in,k = Re(conj(bar_k) e^{i phi}) in_k / |in_k|; phibar =
// -sum_k Im(conj(bar_k) out_k); acc[0..2] += phibar dphi/dk_a, acc[3] +=
// -phibar wscale (the adjoint of omega t times wscale: t for the adjoint of
// omega itself).
//
// After a projection phibar could be had from the sum of its qbar alone: the
// projection turns a phase per cell into the mean phase, wherever every edge
// at the nozzle carries the phase difference.  An edge with z = 0 (psi exactly
// zero on a side) carries none, so the sum over the cells is taken, which
// holds in every case.  It is what remains of a cancellation between the
// gauge's and the one-form's parts: 2e-7 to 7e-4 relative to 64 bits (70 states
// on 56x40x40 to 128x80x80).
__global__ void __launch_bounds__(256) k_adj_restrict(Grid g, const float4* __restrict__ psi_in,
                                                      float4* __restrict__ bar, JetArgs j, double* __restrict__ acc,
                                                      float wscale) {
    pdl_enter();
    double v4[4] = {0.0, 0.0, 0.0, 0.0};
    bool any = false;
    const int x = cell_x(g), y = cell_y(g);
    for (int z = blockIdx.z; z < g.n[2]; z += gridDim.z) {
        if (x >= g.n[0] || y >= g.n[1]) break;
        const long long c = cell(g, x, y, z);
        const float px = __fmul_rn((float)x, g.d[0]);
        const float py = __fmul_rn((float)y, g.d[1]);
        const float pz = __fmul_rn((float)z, g.d[2]);
        const bool jet = j.mask ? (j.mask[c] != 0) : isjet_f32(px, py, pz, j.cen, j.len, j.rad);
        if (!jet) continue;
        any = true;
        float ph;
        if (j.phase_mode == 0)
            ph = __fadd_rn(__fadd_rn(__fadd_rn(j.kvec[0], px), __fadd_rn(j.kvec[1], py)), __fadd_rn(j.kvec[2], pz));
        else
            ph = j.kvec[0] * px + j.kvec[1] * py + j.kvec[2] * pz;
        ph = ph - j.omgterm;
        float s, co;
        sincosf(ph, &s, &co);
        const float4 v = psi_in[c];
        const float a1 = hypotf(v.x, v.y), a2 = hypotf(v.z, v.w);
        const float4 gb = bar[c];
        const float r1 = gb.x * co + gb.y * s, r2 = gb.z * co + gb.w * s;
        const float i1 = a1 > 0.f ? r1 / a1 : 0.f, i2 = a2 > 0.f ? r2 / a2 : 0.f;
        bar[c] = make_float4(i1 * v.x, i1 * v.y, i2 * v.z, i2 * v.w);
        const float4 o = make_float4(a1 * co, a1 * s, a2 * co, a2 * s);
        const double phb = -((gb.x * o.y - gb.y * o.x) + (gb.z * o.w - gb.w * o.z));
        if (j.phase_mode == 0) {
            v4[0] += phb;
            v4[1] += phb;
            v4[2] += phb;
        } else {
            v4[0] += phb * px;
            v4[1] += phb * py;
            v4[2] += phb * pz;
        }
        v4[3] -= phb * wscale;
    }
    if (__syncthreads_or(any)) block_sum_add<4>(v4, acc);  // most blocks lie outside the nozzle
}

namespace {

// one staggered sample: its base cell and weights
struct Sample {
    int c;
    float wx, wy, wz;
};

template <bool POW2, bool NORMW>
__device__ __forceinline__ Sample stag_sample(const AdvConst& k, float3 pt) {
    float P[3] = {pt.x, pt.y, pt.z};
    const bool inbox = (pt.x >= 0.f && pt.x < k.L[0]) && (pt.y >= 0.f && pt.y < k.L[1]) &&
                       (pt.z >= 0.f && pt.z < k.L[2]);
    if (!inbox) {
#pragma unroll
        for (int a = 0; a < 3; ++a) P[a] = jl_mod_box(P[a], k.L[a]);
    }
    int i[3];
    float w[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int ii = cell_floor<POW2>(P[a], k.dinv[a], k.d[a], k.feps[a]);
        ii = max(min(ii, k.nm[a]), 0);
        i[a] = ii;
        w[a] = __fsub_rn(P[a], __fmul_rn((float)ii, k.d[a]));
        if (NORMW) w[a] = __fdiv_rn(w[a], k.d[a]);
    }
    return Sample{i[0] + k.pnx * i[1] + k.pnxy * i[2], w[0], w[1], w[2]};
}

// v <- the twelve velocity samples of cell c, unless it holds them already
__device__ __forceinline__ void hold_cell(const AdvConst& k, int c, CellVel& v) {
    if (c == v.c) return;
    v.c = c;
    const float4* b0 = k.v + c;
    const float4* by = b0 + k.pnx;
    const float4* bz = b0 + k.pnxy;
    const float4 a000 = __ldg(b0), a100 = __ldg(b0 + 1), a010 = __ldg(by), a001 = __ldg(bz);
    const float4 a011 = __ldg(by + k.pnxy), a101 = __ldg(bz + 1), a110 = __ldg(by + 1);
    v.x00 = a000.x, v.x10 = a010.x, v.x01 = a001.x, v.x11 = a011.x;
    v.y00 = a000.y, v.y10 = a100.y, v.y01 = a001.y, v.y11 = a101.y;
    v.z00 = a000.z, v.z10 = a100.z, v.z01 = a010.z, v.z11 = a110.z;
}

__device__ __forceinline__ float3 sample_u(const CellVel& v, const Sample& s) {
    const float wx = s.wx, wy = s.wy, wz = s.wz;
    float3 u;
    u.x = (1.f - wz) * ((1.f - wy) * v.x00 + wy * v.x10) + wz * ((1.f - wy) * v.x01 + wy * v.x11);
    u.y = (1.f - wz) * ((1.f - wx) * v.y00 + wx * v.y10) + wz * ((1.f - wx) * v.y01 + wx * v.y11);
    u.z = (1.f - wy) * ((1.f - wx) * v.z00 + wx * v.z10) + wy * ((1.f - wx) * v.z01 + wx * v.z11);
    return u;
}

// add the cotangents of cell b.c's twelve samples into the padded velocity
// cotangent: the cells with two or three of them as one vector reduction each.
// Zeros are not added: particles with no part in the loss, and slots an emission
// overwrote, cost no reductions (2^20 particles on 128x64x64 that move up to 7
// cells a step, none with a cotangent: 96 us, 264 with the zeros added).
__device__ __forceinline__ void flush_cell(const AdvConst& k, const CellVel& b, float4* __restrict__ ubar) {
    float4* u0 = ubar + b.c;
    float4* uy = u0 + k.pnx;
    float4* uz = u0 + k.pnxy;
    if (b.x00 != 0.f || b.y00 != 0.f || b.z00 != 0.f) atomicAdd(u0, make_float4(b.x00, b.y00, b.z00, 0.f));
    if (b.y10 != 0.f || b.z10 != 0.f) atomicAdd(u0 + 1, make_float4(0.f, b.y10, b.z10, 0.f));
    if (b.x10 != 0.f || b.z01 != 0.f) atomicAdd(uy, make_float4(b.x10, 0.f, b.z01, 0.f));
    if (b.x01 != 0.f || b.y01 != 0.f) atomicAdd(uz, make_float4(b.x01, b.y01, 0.f, 0.f));
    if (b.x11 != 0.f) atomicAdd(&uy[k.pnxy].x, b.x11);
    if (b.y11 != 0.f) atomicAdd(&uz[1].y, b.y11);
    if (b.z11 != 0.f) atomicAdd(&uy[1].z, b.z11);
}

// adjoint of one sample: ub = cotangent of u; returns the cotangent of the
// sample point and adds ub times the weights to b, the cotangents of the
// sample's cell (b of another cell goes to memory first).  known: u is the
// sampled velocity.  A finite one has finite samples and weights, so a zero
// cotangent gives zeros, and the cell's samples are not fetched again.
template <bool NORMW>
__device__ __forceinline__ float3 stag_sample_adj(const AdvConst& k, const Sample& s, float3 ub, bool known, float3 u,
                                                  CellVel& v, CellVel& b, float4* __restrict__ ubar) {
    if (known && ub.x == 0.f && ub.y == 0.f && ub.z == 0.f && isfinite(u.x) && isfinite(u.y) && isfinite(u.z))
        return make_float3(0.f, 0.f, 0.f);
    hold_cell(k, s.c, v);
    const float wx = s.wx, wy = s.wy, wz = s.wz;
    // d u / d w (the weights are unnormalised: dw/dp = 1)
    const float dux_dwy = (1.f - wz) * (v.x10 - v.x00) + wz * (v.x11 - v.x01);
    const float dux_dwz = ((1.f - wy) * v.x01 + wy * v.x11) - ((1.f - wy) * v.x00 + wy * v.x10);
    const float duy_dwx = (1.f - wz) * (v.y10 - v.y00) + wz * (v.y11 - v.y01);
    const float duy_dwz = ((1.f - wx) * v.y01 + wx * v.y11) - ((1.f - wx) * v.y00 + wx * v.y10);
    const float duz_dwx = (1.f - wy) * (v.z10 - v.z00) + wy * (v.z11 - v.z01);
    const float duz_dwy = ((1.f - wx) * v.z01 + wx * v.z11) - ((1.f - wx) * v.z00 + wx * v.z10);
    float3 pb;
    pb.x = ub.y * duy_dwx + ub.z * duz_dwx;
    pb.y = ub.x * dux_dwy + ub.z * duz_dwy;
    pb.z = ub.x * dux_dwz + ub.y * duy_dwz;
    if (NORMW) {  // w = (p - i d) / d
        pb.x *= k.dinv[0];
        pb.y *= k.dinv[1];
        pb.z *= k.dinv[2];
    }
    if (s.c != b.c) {
        if (b.c >= 0) flush_cell(k, b, ubar);
        b.c = s.c;
        b.x00 = b.x10 = b.x01 = b.x11 = 0.f;
        b.y00 = b.y10 = b.y01 = b.y11 = 0.f;
        b.z00 = b.z10 = b.z01 = b.z11 = 0.f;
    }
    // a component without a cotangent adds nothing, whatever its weights are (a
    // sample point that is not finite has none)
    if (ub.x != 0.f) {
        b.x00 += ub.x * (1.f - wz) * (1.f - wy);
        b.x10 += ub.x * (1.f - wz) * wy;
        b.x01 += ub.x * wz * (1.f - wy);
        b.x11 += ub.x * wz * wy;
    }
    if (ub.y != 0.f) {
        b.y00 += ub.y * (1.f - wz) * (1.f - wx);
        b.y10 += ub.y * (1.f - wz) * wx;
        b.y01 += ub.y * wz * (1.f - wx);
        b.y11 += ub.y * wz * wx;
    }
    if (ub.z != 0.f) {
        b.z00 += ub.z * (1.f - wy) * (1.f - wx);
        b.z10 += ub.z * (1.f - wy) * wx;
        b.z01 += ub.z * wy * (1.f - wx);
        b.z11 += ub.z * wy * wx;
    }
    return pb;
}

__device__ __forceinline__ float3 f3add(float3 a, float3 b) { return make_float3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 f3scale(float3 a, float s) { return make_float3(a.x * s, a.y * s, a.z * s); }

}  // namespace

// Reverse of one RK4 advection (staggered_advect!, parallel.jl:197-216):
// lam holds the cotangent of the positions after the step and becomes that
// of the positions before it (parts, the positions the forward step started
// from); the cotangent of the padded velocity (float4 per cell) is added into
// ubar.  A slot outside the open box was set to (-1,-1,-1): its cotangent is 0.
// Bound by the reductions into ubar: the four stages of a particle lie in one
// or two cells, so their cotangents are summed per cell in registers and leave
// as 7 reductions instead of 12 scalar ones per stage.
template <bool POW2, bool NORMW>
__global__ void __launch_bounds__(256) k_adj_advect(Grid g, const float* __restrict__ parts, float* __restrict__ lam,
                                                    int np, const float* __restrict__ vel, float4* __restrict__ ubar) {
    pdl_enter();
    const AdvConst kc = adv_const(g, vel);
    const float dt = g.dt, s6 = g.dt / 6.0f;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < np; k += gridDim.x * blockDim.x) {
        const float3 p = make_float3(parts[3 * k], parts[3 * k + 1], parts[3 * k + 2]);
        const bool inside = (p.x > 0.f && p.x < kc.L[0]) && (p.y > 0.f && p.y < kc.L[1]) &&
                            (p.z > 0.f && p.z < kc.L[2]);
        if (!inside) {
            lam[3 * k] = lam[3 * k + 1] = lam[3 * k + 2] = 0.f;
            continue;
        }
        CellVel v, b;
        v.c = b.c = -1;
        auto at = [&](const Sample& s) {
            hold_cell(kc, s.c, v);
            return sample_u(v, s);
        };
        const Sample S1 = stag_sample<POW2, NORMW>(kc, p);
        const float3 k1 = at(S1);
        float3 q = make_float3(p.x + k1.x * dt * 0.5f, p.y + k1.y * dt * 0.5f, p.z + k1.z * dt * 0.5f);
        const Sample S2 = stag_sample<POW2, NORMW>(kc, q);
        const float3 k2 = at(S2);
        q = make_float3(p.x + k2.x * dt * 0.5f, p.y + k2.y * dt * 0.5f, p.z + k2.z * dt * 0.5f);
        const Sample S3 = stag_sample<POW2, NORMW>(kc, q);
        const float3 k3 = at(S3);
        q = make_float3(p.x + k3.x * dt, p.y + k3.y * dt, p.z + k3.z * dt);
        const Sample S4 = stag_sample<POW2, NORMW>(kc, q);
        // reverse of p' = p + dt/6 (k1 + 2 k2 + 2 k3 + k4)
        const float3 L = make_float3(lam[3 * k], lam[3 * k + 1], lam[3 * k + 2]);
        float3 pb = L;
        float3 kb1 = f3scale(L, s6), kb2 = f3scale(L, 2.f * s6), kb3 = f3scale(L, 2.f * s6);
        const float3 kb4 = f3scale(L, s6);
        float3 qb = stag_sample_adj<NORMW>(kc, S4, kb4, false, k3, v, b, ubar);  // q4 = p + dt k3
        pb = f3add(pb, qb);
        kb3 = f3add(kb3, f3scale(qb, dt));
        qb = stag_sample_adj<NORMW>(kc, S3, kb3, true, k3, v, b, ubar);  // q3 = p + dt/2 k2
        pb = f3add(pb, qb);
        kb2 = f3add(kb2, f3scale(qb, 0.5f * dt));
        qb = stag_sample_adj<NORMW>(kc, S2, kb2, true, k2, v, b, ubar);  // q2 = p + dt/2 k1
        pb = f3add(pb, qb);
        kb1 = f3add(kb1, f3scale(qb, 0.5f * dt));
        qb = stag_sample_adj<NORMW>(kc, S1, kb1, true, k1, v, b, ubar);  // k1 at p
        pb = f3add(pb, qb);
        flush_cell(kc, b, ubar);
        lam[3 * k] = pb.x;
        lam[3 * k + 1] = pb.y;
        lam[3 * k + 2] = pb.z;
    }
}

// L = sum over slots alive in x (x >= 0) of |x - y|^2 (into loss[0], double);
// lam = dL/dx = 2 (x - y), 0 for dead slots
__global__ void k_loss(const float* __restrict__ x, const float* __restrict__ y, float* __restrict__ lam, int np,
                       double* __restrict__ loss) {
    pdl_enter();
    double v[1] = {0.0};
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < np; k += gridDim.x * blockDim.x) {
        const bool alive = x[3 * k] >= 0.f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float d = alive ? x[3 * k + a] - y[3 * k + a] : 0.f;
            v[0] += (double)d * d;
            lam[3 * k + a] = 2.f * d;
        }
    }
    block_sum_add<1>(v, loss);
}

// velocity cotangent from AoS float3 per cell: the cells themselves only (the
// periodic copies stay 0)
__global__ void __launch_bounds__(256) k_adj_from_aos(Grid g, const float* __restrict__ aos, float4* __restrict__ ubar) {
    pdl_enter();
    const int x = cell_x(g), y = cell_y(g);
    if (x >= g.n[0] || y >= g.n[1]) return;
    for (int z = blockIdx.z; z < g.n[2]; z += gridDim.z) {
        const long long c = cell(g, x, y, z);
        ubar[pcell(g, x, y, z)] = make_float4(aos[3 * c], aos[3 * c + 1], aos[3 * c + 2], 0.f);
    }
}

// the velocity cotangent (padded, its copies collected) as AoS float3 per cell
__global__ void __launch_bounds__(256) k_adj_to_aos(Grid g, const float4* __restrict__ ubar, float* __restrict__ aos) {
    pdl_enter();
    const int x = cell_x(g), y = cell_y(g);
    if (x >= g.n[0] || y >= g.n[1]) return;
    for (int z = blockIdx.z; z < g.n[2]; z += gridDim.z) {
        const long long c = cell(g, x, y, z);
        const float4 v = ubar_at(g, ubar, x, y, z);
        aos[3 * c] = v.x;
        aos[3 * c + 1] = v.y;
        aos[3 * c + 2] = v.z;
    }
}

// cotangent 0 for the ring slots an emission overwrote
__global__ void k_zero_slots(float* __restrict__ lam, long long nslots, long long start, long long count) {
    pdl_enter();
    const long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (j >= count) return;
    const long long s = (start + j) % nslots;
    lam[3 * s] = lam[3 * s + 1] = lam[3 * s + 2] = 0.f;
}

// ---------------------------------------------------------------- launchers

cudaError_t launch_gauge(const Grid& g, const float4* in, const float* q, float4* out, cudaStream_t s) {
    return launch_pdl(k_gauge, dim3(grid_n(g.N, 256)), dim3(256), 0, s, in, q, out, g.N);
}
cudaError_t launch_normalize_to(const Grid& g, const float4* in, float4* out, cudaStream_t s) {
    return launch_pdl(k_normalize_to, dim3(grid_n(g.N, 256)), dim3(256), 0, s, in, out, g.N);
}
cudaError_t launch_restrict_to(const Grid& g, const float4* in, float4* out, const JetArgs& j, cudaStream_t s) {
    return launch_pdl(k_restrict_to<false>, cell_grid(g), dim3(256), 0, s, g, in, (const float*)nullptr,
                      (float4*)nullptr, out, j);
}
cudaError_t launch_gauge_restrict(const Grid& g, const float4* in, const float* q, float4* mid, float4* out,
                                  const JetArgs& j, cudaStream_t s) {
    return launch_pdl(k_restrict_to<true>, cell_grid(g), dim3(256), 0, s, g, in, q, mid, out, j);
}
cudaError_t launch_adj_normalize(const Grid& g, const float4* psi_in, float4* bar, cudaStream_t s) {
    return launch_pdl(k_adj_normalize, dim3(grid_n(g.N, 256)), dim3(256), 0, s, psi_in, bar, g.N);
}
cudaError_t launch_adj_gauge(const Grid& g, const float4* psi_in, const float* q, float4* bar, float* qbar,
                             cudaStream_t s) {
    return launch_pdl(k_adj_gauge, dim3(grid_n(g.N, 256)), dim3(256), 0, s, psi_in, q, bar, qbar, g.N);
}
cudaError_t launch_adj_oneform_div(const Grid& g, const float4* psi, float4* bar, const float* fbar, cudaStream_t s) {
    AdjOneFormArgs a;
    a.g = g;
    a.psi = psi;
    a.bar = bar;
    a.fbar = fbar;
    a.ubar = nullptr;
    for (int k = 0; k < 3; ++k) a.s[k] = g.inv_d2[k];
    return launch_pdl(k_adj_oneform<true>, cell_grid(g), dim3(256), 0, s, a);
}
cudaError_t launch_adj_oneform_vel(const Grid& g, const float4* psi, float4* bar, const float4* ubar, float hbar,
                                   int sharp, cudaStream_t s) {
    AdjOneFormArgs a;
    a.g = g;
    a.psi = psi;
    a.bar = bar;
    a.fbar = nullptr;
    a.ubar = ubar;
    for (int k = 0; k < 3; ++k) a.s[k] = sharp ? hbar * g.dinv[k] : hbar;
    return launch_pdl(k_adj_oneform<false>, cell_grid(g), dim3(256), 0, s, a);
}
cudaError_t launch_adj_restrict(const Grid& g, const float4* psi_in, float4* bar, const JetArgs& j, double* acc,
                                float wscale, cudaStream_t s) {
    return launch_pdl(k_adj_restrict, cell_grid(g), dim3(256), 0, s, g, psi_in, bar, j, acc, wscale);
}
cudaError_t launch_adj_advect(const Grid& g, const float* parts, float* lam, long long np, const float* vel,
                              float4* ubar, cudaStream_t s) {
    if (np <= 0) return cudaSuccess;
    if (np > kMaxParticles) return cudaErrorInvalidValue;
    const bool pow2 = g.d_pow2[0] && g.d_pow2[1] && g.d_pow2[2];
    auto go = [&](auto kernel) {
        return launch_pdl(kernel, dim3(grid_n(np, 256)), dim3(256), 0, s, g, parts, lam, (int)np, vel, ubar);
    };
    if (g.norm_w) return pow2 ? go(k_adj_advect<true, true>) : go(k_adj_advect<false, true>);
    return pow2 ? go(k_adj_advect<true, false>) : go(k_adj_advect<false, false>);
}
cudaError_t launch_loss(const float* x, const float* y, float* lam, long long np, double* loss, cudaStream_t s) {
    if (np <= 0) return cudaSuccess;
    return launch_pdl(k_loss, dim3(grid_n(np, 256)), dim3(256), 0, s, x, y, lam, (int)np, loss);
}
cudaError_t launch_adj_from_aos(const Grid& g, const float* aos, float4* ubar, cudaStream_t s) {
    return launch_pdl(k_adj_from_aos, cell_grid(g), dim3(256), 0, s, g, aos, ubar);
}
cudaError_t launch_adj_to_aos(const Grid& g, const float4* ubar, float* aos, cudaStream_t s) {
    return launch_pdl(k_adj_to_aos, cell_grid(g), dim3(256), 0, s, g, ubar, aos);
}
cudaError_t launch_zero_slots(float* lam, long long nslots, long long start, long long count, cudaStream_t s) {
    if (count <= 0) return cudaSuccess;
    return launch_pdl(k_zero_slots, dim3((unsigned)((count + 255) / 256)), dim3(256), 0, s, lam, nslots, start % nslots,
                      count);
}

}  // namespace isf
