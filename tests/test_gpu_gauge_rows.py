"""The real x passes of long rows at the row counts where their tile changes,
against the FP64 oracle."""
import numpy as np
import pytest
import torch

from helpers import rel, smooth_psi

pytestmark = pytest.mark.gpu

HBAR, DT = float(np.float32(0.1)), float(np.float32(1 / 48))


# rows of 512 cells change at 2369 (a k-major spectrum below; the last two with a
# partial last tile of 16 pairs), shorter ones at 4096
@pytest.mark.parametrize("dims", [(512, 48, 48), (512, 50, 48), (512, 50, 50), (512, 100, 24), (384, 64, 56),
                                  (384, 64, 64), (256, 40, 100)])
def test_projection_on_both_sides(isfpkg, oracle_mod, dims):
    L = tuple(max(1, n // 32) for n in dims)
    isf = isfpkg.ISF(L, dims, HBAR, DT)
    orc = oracle_mod.Oracle(L, dims, HBAR, DT)
    psi64 = smooth_psi(dims, seed=37)
    psi = torch.tensor(psi64, dtype=torch.float32, device="cuda")
    isfpkg.pressure_project(isf, psi)
    isf.sync()
    orc.pressure_project(psi64)
    assert rel(psi.double().cpu().numpy(), psi64) < 1e-5
