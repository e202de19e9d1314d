"""Passes whose plan depends on the number of CTAs: the flow on both sides of
the line, in every direction, against the FP64 oracle."""
import numpy as np
import pytest
import torch

from helpers import rel

pytestmark = pytest.mark.gpu

HBAR, DT = float(np.float32(0.1)), float(np.float32(1 / 48))


# CTAs of the pass at the long axis: just below and from 320 (z at 100 and 112, y
# at 128) and 512 (x and y at 112) on; the last two partial tiles
@pytest.mark.parametrize("dims", [(24, 100, 100), (32, 100, 100), (24, 96, 112), (32, 96, 112), (16, 128, 128),
                                  (24, 128, 128), (64, 112, 56), (64, 112, 64), (112, 50, 80), (112, 64, 64),
                                  (20, 100, 100), (112, 50, 100)])
def test_flow_on_both_sides_of_the_joined_plans(isfpkg, oracle_mod, dims):
    L = (1, 1, 1)
    isf = isfpkg.ISF(L, dims, HBAR, DT)
    orc = oracle_mod.Oracle(L, dims, HBAR, DT)
    psi64 = np.random.default_rng(91).normal(size=dims[::-1] + (4,)).astype(np.float32).astype(np.float64)
    psi = torch.tensor(psi64, dtype=torch.float32, device="cuda")
    isfpkg.schroedinger_flow(isf, psi)
    isf.sync()
    orc.schroedinger_flow(psi64)
    assert rel(psi.double().cpu().numpy(), psi64) < 1e-5
