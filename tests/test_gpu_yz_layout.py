"""psi y / z passes whose tile layout or plan is an exception of their length,
against the FP64 oracle."""
import numpy as np
import pytest
import torch

from helpers import rel

pytestmark = pytest.mark.gpu

HBAR, DT = float(np.float32(0.1)), float(np.float32(1 / 48))


def check(isfpkg, oracle_mod, dims):
    isf = isfpkg.ISF((1, 1, 1), dims, HBAR, DT)
    orc = oracle_mod.Oracle((1, 1, 1), dims, HBAR, DT)
    psi64 = np.random.default_rng(93).normal(size=dims[::-1] + (4,)).astype(np.float32).astype(np.float64)
    psi = torch.tensor(psi64, dtype=torch.float32, device="cuda")
    isfpkg.schroedinger_flow(isf, psi)
    isf.sync()
    orc.schroedinger_flow(psi64)
    assert rel(psi.double().cpu().numpy(), psi64) < 1e-5


# swizzled in y (whole and partial tiles), rows in z
@pytest.mark.parametrize("dims", [(16, 192, 8), (20, 192, 12), (50, 192, 24), (8, 12, 192)])
def test_flow_at_192(isfpkg, oracle_mod, dims):
    check(isfpkg, oracle_mod, dims)


# z at 96 with the mask: 560 CTAs (joined), 600, 640, 672 (plain; the last with
# a partial tile) and 768 (joined)
@pytest.mark.parametrize("dims", [(40, 112, 96), (96, 50, 96), (80, 64, 96), (50, 96, 96), (24, 256, 96)])
def test_flow_around_the_plain_plans_of_96(isfpkg, oracle_mod, dims):
    check(isfpkg, oracle_mod, dims)


# just below and from 384 CTAs (z at 100) and 640 (y at 112); the last partial
@pytest.mark.parametrize("dims", [(32, 80, 100), (32, 96, 100), (56, 112, 80), (64, 112, 80), (50, 112, 100)])
def test_flow_around_the_lines_of_100_and_112(isfpkg, oracle_mod, dims):
    check(isfpkg, oracle_mod, dims)
