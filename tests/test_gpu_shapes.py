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


# planes per stencil CTA: 1 (few columns), 3 with a remainder of 2, 4, 5 with a
# remainder of 2, and 8, on whole and partial tiles
@pytest.mark.parametrize("L,dims", [((2, 1, 1), (40, 12, 50)), ((8, 1, 1), (512, 64, 50)), ((6, 2, 1), (384, 100, 56)),
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
