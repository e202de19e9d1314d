"""Reverse advection: cotangents that are zero add nothing to the velocity's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

L, DIMS = (1, 1, 1), (16, 16, 16)
D = 1 / 16
DT = 1 / 64


def test_a_sample_point_that_is_not_finite_adds_nothing_without_a_cotangent(isfpkg):
    """A particle without a cotangent whose last RK sample point is infinite
    in x.  Along y it goes from row 4 to 5 (stage 2) and 6 (stage 3); row 7,
    which stage 3 is the first to interpolate from, has an infinite x velocity.
    The stage 4 point is x = inf on row 4, so its clamped base cell has x = 0,
    and x = 0 and 1 are the only cells of its samples.  Its cotangent is zero,
    so those cells get none (the particle itself is at x = 8)."""
    isf = isfpkg.ISF(L, DIMS, 0.1, DT)
    v = np.zeros((16, 16, 16, 3), dtype=np.float32)          # z, y, x
    v[:, 4, :, 1] = 1.0 * D / (0.5 * DT)
    v[:, 5, :, 1] = 2.0 * D / (0.5 * DT)
    v[:, 7, :, 0] = np.inf
    # u_y does not change along x and z, and the weights of its four samples add
    # up to 1, so it is the row's value; the point lies off the faces in y and z,
    # so the weight of row 7 is not 0
    p = np.array([[8 * D, 4.5 * D, 8.25 * D]], dtype=np.float32)
    isf.velocity = torch.tensor(v, device="cuda")
    parts = torch.tensor(p, device="cuda")
    lam = torch.zeros_like(parts)
    isfpkg.set_velocity_bar(isf, torch.zeros(16, 16, 16, 3, device="cuda"))
    isfpkg.adj_staggered_advect(isf, parts, lam)
    bar = isfpkg.get_velocity_bar(isf)
    isf.sync()
    assert torch.isnan(lam).any()   # the stages did run into it
    assert (bar[:, :, :2] == 0).all()


def test_zero_cotangents_leave_the_others_sums(isfpkg):
    """Particles with a zero cotangent, or zero components of it, among others
    change no sum: the same velocity cotangent as without them, bit for bit
    (one particle per four cells, so no two of those that count share one)."""
    n = 16
    isf = isfpkg.ISF(L, DIMS, 0.1, DT)
    rng = np.random.default_rng(5)
    isf.velocity = torch.tensor(rng.uniform(-0.5, 0.5, (n, n, n, 3)), dtype=torch.float32, device="cuda")
    g = np.stack(np.meshgrid(*[np.arange(0, n, 4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    some = torch.tensor((g + 0.4) * D, dtype=torch.float32, device="cuda")
    lam = torch.tensor(rng.normal(size=some.shape), dtype=torch.float32, device="cuda")
    lam[::3, 0] = 0
    lam[1::3, 1:] = 0
    others = torch.tensor(rng.uniform(0.01, 0.99, (1000, 3)), dtype=torch.float32, device="cuda")
    bars = []
    for p, y in ((some, lam), (torch.cat([some, others]), torch.cat([lam, torch.zeros_like(others)]))):
        y = y.clone()
        isfpkg.set_velocity_bar(isf, torch.zeros(n, n, n, 3, device="cuda"))
        isfpkg.adj_staggered_advect(isf, p.contiguous(), y)
        bars.append(isfpkg.get_velocity_bar(isf))
    isf.sync()
    assert (y[len(some):] == 0).all()
    assert bars[0].abs().max() > 0
    assert torch.equal(bars[0], bars[1])
