"""Launch shapes chosen from the grid: sizes at the edges of the rules that
pick tiles, planes per CTA and kernels, against the FP64 oracle."""
import numpy as np
import pytest
import torch

from helpers import rel, smooth_psi

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
