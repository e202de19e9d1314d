"""Launch shapes chosen from the grid: sizes at the edges of the rules that
pick tiles, planes per CTA and kernels, against the FP64 oracle."""
import numpy as np
import pytest
import torch

from helpers import rel, smooth_field, smooth_psi

pytestmark = pytest.mark.gpu

HBAR = float(np.float32(0.1))
DT = float(np.float32(1 / 48))


def cuda(a, dtype=torch.float32):
    return torch.tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


def host(t):
    return t.detach().double().cpu().numpy()


# planes per stencil CTA: 1 (few columns), 3 and 6 with a remainder of 2, 5, and 8, on
# whole and partial tiles
@pytest.mark.parametrize("L,dims", [((2, 1, 1), (40, 12, 50)), ((5, 3, 2), (160, 96, 56)), ((8, 1, 1), (512, 64, 56)),
                                    ((8, 1, 1), (512, 64, 50)), ((6, 2, 1), (384, 100, 56)),
                                    ((6, 3, 3), (200, 100, 112)), ((8, 4, 1), (512, 128, 64))])
def test_stencil_planes_per_cta(isfpkg, oracle_mod, L, dims):
    isf = isfpkg.ISF(L, dims, HBAR, DT)
    orc = oracle_mod.Oracle(L, dims, HBAR, DT)
    psi64 = smooth_psi(dims, seed=31)
    psi = cuda(psi64)
    isfpkg.velocity_one_form(isf, psi, HBAR)
    assert np.abs(host(isf.velocity) - orc.velocity_one_form(psi64, HBAR)).max() < 2e-6
    # the divergence stencil, through the projection
    isfpkg.pressure_project(isf, psi)
    orc.pressure_project(psi64)
    isf.sync()
    assert rel(host(psi), psi64) < 1e-5


# RK stages that stay in the particle's cell, change it now and then, and
# change it at every stage, on power-of-two and general cell sizes
@pytest.mark.parametrize("L,dims", [((4, 2, 2), (64, 32, 32)), ((3, 2, 2), (50, 40, 24))])
@pytest.mark.parametrize("cells_per_step", [0.01, 0.7, 5.0])
def test_advect_across_cells(isfpkg, oracle_mod, L, dims, cells_per_step):
    isf = isfpkg.ISF(L, dims, HBAR, DT)
    orc = oracle_mod.Oracle(L, dims, HBAR, DT)
    rng = np.random.default_rng(41)
    speed = cells_per_step * min(length / n for length, n in zip(L, dims)) / DT
    vel = (speed * rng.uniform(-1, 1, dims[::-1] + (3,))).astype(np.float32)
    parts64 = (rng.uniform(0, 1, (20011, 3)) * np.asarray(L)).astype(np.float32).astype(np.float64)
    isf.velocity = cuda(vel)
    orc.set_velocity(vel.astype(np.float64))
    parts = cuda(parts64)
    isfpkg.staggered_advect(parts, isf)
    isf.sync()
    po, margin = orc.staggered_advect(parts64.copy(), margin=True)
    clear = margin >= 1e-4
    assert clear.mean() > 0.9
    assert (np.abs(host(parts) - po).max(axis=1)[clear] / min(L) < 1e-5).all()


# real x passes with 4 row pairs per CTA (short grids, partial last tile) and
# with 16, k-major (ny = nz in the plane sizes) and row-major, 1 to 64 lanes a row
@pytest.mark.parametrize("L,dims", [((1, 1, 1), (8, 12, 20)), ((1, 1, 1), (12, 32, 32)), ((2, 1, 1), (50, 12, 50)),
                                    ((4, 2, 2), (100, 48, 48)), ((2, 2, 2), (56, 64, 64)), ((4, 2, 2), (160, 50, 100)),
                                    ((8, 1, 1), (512, 20, 50)), ((4, 4, 4), (112, 96, 96))])
def test_real_x_passes(isfpkg, oracle_mod, L, dims):
    isf = isfpkg.ISF(L, dims, HBAR, DT)
    orc = oracle_mod.Oracle(L, dims, HBAR, DT)
    cen, length, rad = [0.3 * v for v in L], 0.3 * L[0], 0.3 * L[1]
    psi64 = smooth_psi(dims, seed=32)
    psi = cuda(psi64)
    isfpkg.init_jet(isf, psi, 1, (10.0, 0.0, 0.0), nozzle=(cen, length, rad), phase_mode=1)
    orc.restrict_velocity(psi64, (10.0, 0.0, 0.0), 0.0, cen, length, rad, phase_mode=1)
    orc.pressure_project(psi64)
    isf.sync()
    assert rel(host(psi), psi64) < 1e-5
    rng = np.random.default_rng(5)
    f = smooth_field(dims, rng, modes=6) + 0.1 * rng.normal(size=dims[::-1])
    q = isf.poisson_solve(cuda(f))
    isf.sync()
    orc.set_f(f)
    assert rel(host(q), orc.poisson_solve().real) < 1e-5


# adjoint kernels over 32 x 8 cell tiles and z walks: partial tiles, a grid
# thinner than a tile, and one with more planes than blocks along z; the
# advection's cotangent with particles that stay in their cell and that leave it
@pytest.mark.parametrize("L,dims", [((1, 1, 1), (8, 12, 20)), ((2, 2, 2), (50, 20, 56)), ((8, 2, 4), (256, 48, 100))])
@pytest.mark.parametrize("cells_per_step", [0.05, 3.0])
def test_adj_advect_uniform_velocity(isfpkg, L, dims, cells_per_step):
    """A uniform velocity u is sampled as itself, so p' = p + dt u: the
    cotangents of all samples sum to dt times that of the particles, and the
    positions' cotangent passes through."""
    isf = isfpkg.ISF(L, dims, HBAR, DT)
    rng = np.random.default_rng(51)
    P = 5003
    d = [length / n for length, n in zip(L, dims)]
    u = np.array([cells_per_step, -0.6 * cells_per_step, 0.3 * cells_per_step]) * min(d) / DT
    # away from the box walls: no particle dies
    p = (0.35 + 0.3 * rng.uniform(0, 1, (P, 3))) * np.asarray(L)
    w = rng.normal(size=(P, 3)).astype(np.float32)
    isf.velocity = cuda(np.broadcast_to(u.astype(np.float32), dims[::-1] + (3,)))
    bar = cuda(w)
    isfpkg.adj_staggered_advect(isf, cuda(p), bar)
    ub = host(isfpkg.get_velocity_bar(isf))
    want = DT * w.astype(np.float64).sum(axis=0)
    scale = DT * np.abs(w).sum(axis=0)
    assert (np.abs(ub.sum(axis=(0, 1, 2)) - want) <= 1e-5 * scale).all()
    assert (np.abs(host(bar) - w) <= 1e-5 * np.abs(w).max()).all()


@pytest.mark.parametrize("L,dims", [((1, 1, 1), (12, 8, 20)), ((2, 1, 2), (50, 20, 40))])
def test_adj_project_and_one_form_on_partial_tiles(isfpkg, oracle_mod, L, dims):
    """The projection's and the velocity one-form's transposes against central
    differences of the FP64 oracle along a random direction."""
    isf = isfpkg.ISF(L, dims, HBAR, DT)
    orc = oracle_mod.Oracle(L, dims, HBAR, DT)
    rng = np.random.default_rng(52)
    x = smooth_psi(dims, seed=52, phase_scale=0.5).astype(np.float32).astype(np.float64)
    u, w = rng.normal(size=x.shape), rng.normal(size=x.shape).astype(np.float32)
    h = 1e-6
    t = cuda(w)
    isfpkg.adj_pressure_project(isf, cuda(x), t)
    g = (w * (orc.pressure_project(x + h * u) - orc.pressure_project(x - h * u))).sum() / (2 * h)
    assert abs((host(t) * u).sum() - g) <= 1e-3 * abs(g) + 1e-6 * np.linalg.norm(w) * np.linalg.norm(u)
    wv = rng.normal(size=dims[::-1] + (3,)).astype(np.float32)
    isfpkg.set_velocity_bar(isf, cuda(wv))
    assert np.array_equal(host(isfpkg.get_velocity_bar(isf)), wv)
    t = torch.zeros(x.shape, device="cuda")
    isfpkg.adj_velocity_one_form(isf, cuda(x), t, HBAR)
    g = (wv * (orc.velocity_one_form(x + h * u, HBAR) - orc.velocity_one_form(x - h * u, HBAR))).sum() / (2 * h)
    assert abs((host(t) * u).sum() - g) <= 1e-3 * abs(g) + 1e-6 * np.linalg.norm(wv) * np.linalg.norm(u)


# every pencil length whose psi passes join two stages in registers, in each
# direction, on whole and partial tiles
@pytest.mark.parametrize("dims", [(112, 8, 8), (100, 8, 112), (50, 112, 8), (8, 128, 100), (20, 384, 96), (12, 20, 384),
                                  (16, 96, 128)])
def test_schroedinger_flow_lengths(isfpkg, oracle_mod, dims):
    L = (1, 1, 1)
    isf = isfpkg.ISF(L, dims, HBAR, DT)
    orc = oracle_mod.Oracle(L, dims, HBAR, DT)
    psi64 = np.random.default_rng(61).normal(size=dims[::-1] + (4,)).astype(np.float32).astype(np.float64)
    psi = cuda(psi64)
    isfpkg.schroedinger_flow(isf, psi)
    isf.sync()
    orc.schroedinger_flow(psi64)
    assert rel(host(psi), psi64) < 1e-5


@pytest.mark.parametrize("L,dims", [((2, 1, 1), (32, 16, 16)), ((2, 2, 2), (40, 20, 24))])
@pytest.mark.parametrize("caller_stream", [False, True])
def test_sequences_as_graphs(isfpkg, cfgs, L, dims, caller_stream):
    """A sequence of kernels that comes back is launched as a graph, with every
    argument set per call: steps that change psi buffer, particle count, jet and
    emission from call to call give the bits of a handle that launches kernel by
    kernel (profiling), and so do steps under stream capture."""
    st = torch.cuda.Stream() if caller_stream else None
    a = isfpkg.ISF(L, dims, HBAR, DT, stream=st)
    b = isfpkg.ISF(L, dims, HBAR, DT)
    b.profile_start()
    kvec, omega = cfgs.jet_omega()
    psis = [[cuda(smooth_psi(dims, seed=70 + k)) for k in range(2)] for _ in range(2)]
    rng = np.random.default_rng(71)
    parts = [[cuda(p) for p in (rng.uniform(0, 1, (n, 3)) * np.asarray(L))] for n in (300, 5000)]
    parts = [[torch.stack(p).contiguous() for p in parts] for _ in range(2)]
    torch.cuda.synchronize()

    def run(h, s, k):
        jet = None
        if k % 3:
            jet = dict(kvec=kvec, omega_t=0.1 * k, cen=(0.3 * L[0], 0.5 * L[1], 0.5 * L[2]), len=0.1 + 0.01 * k, rad=0.3,
                       emit_start=10 * k, emit_count=10 + k, seed=5, counter=k, emit_mode=1, phase_mode=1)
        isfpkg.step(h, psis[s][k % 2], parts[s][(k // 2) % 2], jet)
        isfpkg.schroedinger_flow(h, psis[s][(k + 1) % 2])
        isfpkg.pressure_project(h, psis[s][(k + 1) % 2])

    for k in range(24):
        run(a, 0, k)
        run(b, 1, k)
    a.sync()
    b.sync()
    if caller_stream:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            run(a, 0, 24)
        g.replay()
        run(b, 1, 24)
        torch.cuda.synchronize()
    for k in range(2):
        assert torch.equal(psis[0][k], psis[1][k])
        assert torch.equal(parts[0][k], parts[1][k])
    assert a.counters()["live"] == b.counters()["live"]
    b.profile_stop()
