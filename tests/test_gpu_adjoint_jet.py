"""The jet's cotangent of a step and of the whole run is the one of the
operators they are made of: isf_adj_step and isf_adj_gradient against the
reversed operators called one by one.

Both sides run the same kernels on the same bits (the particles are far enough
apart that no two add into the same velocity cell, so no sum depends on an
order) but for the last one: the nozzle cells' FP64 terms are added in any
order.  With under 1e4 terms, each at most |cotangent| |psi| |x| of its cell,
that costs under 1e4 x 1.1e-16 x 4 of the cells' summed cotangent sizes."""
import numpy as np
import pytest
import torch

from helpers import smooth_psi

pytestmark = pytest.mark.gpu

L, DIMS = (4, 2, 2), (32, 16, 16)
HBAR, DT = float(np.float32(0.1)), float(np.float32(1 / 48))
NOZZLE = ((1.0, 1.0, 1.0), 0.8, 0.6)
KVEC = tuple(float(np.float32(k)) for k in (6.0, 0.5, -0.3))
TOL = 1e-11


def cuda(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float32, device="cuda")


def lattice():
    """One particle in every fourth cell along each axis, off the faces."""
    n = [d // 4 for d in DIMS]
    g = np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3)
    return (4.0 * g + 1.4) * (np.asarray(L) / np.asarray(DIMS))


def jet_of(omega_t):
    return dict(kvec=KVEC, omega_t=omega_t, cen=NOZZLE[0], len=NOZZLE[1], rad=NOZZLE[2], phase_mode=1)


def close(got, want, size):
    return np.abs(np.asarray(got) - np.asarray(want)).max() <= TOL * size


def size_of(bar):
    return float(bar.double().norm(dim=-1).sum())


@pytest.mark.parametrize("seed", [11, 12, 13])
def test_adj_step_jet_cotangent_is_the_restriction_s(isfpkg, seed):
    isf = isfpkg.ISF(L, DIMS, HBAR, DT)
    psi = cuda(smooth_psi(DIMS, seed))
    yb = cuda(np.random.default_rng(seed).normal(size=isf.shape + (4,)))
    wt = float(np.float32(0.35))
    bar = yb.clone()
    jb = isfpkg.adj_step(isf, psi, None, jet_of(wt), bar)
    # forward to the restriction's input and output, then their transposes
    c = psi.clone()
    isfpkg.schroedinger_flow(isf, c)
    isfpkg.normalize_psi(isf, c)
    isfpkg.pressure_project(isf, c)
    isf.sync()
    d = c.clone()
    torch.cuda.synchronize()
    isfpkg.restrict_velocity(isf, d, KVEC, None, wt, nozzle=NOZZLE, phase_mode=1)
    isfpkg.adj_pressure_project(isf, d, yb)
    isf.sync()
    size = size_of(yb)
    torch.cuda.synchronize()
    want = isfpkg.adj_restrict_velocity(isf, c, yb, KVEC, wt, nozzle=NOZZLE, phase_mode=1)
    assert close(jb, want, size), (jb, want, size)


@pytest.mark.parametrize("hole", [0, 2])
def test_adj_gradient_jet_cotangent_with_a_hole(isfpkg, hole):
    """A psi0 that is exactly zero in `hole`^3 cells inside the nozzle stays
    so through the initialisation (the restriction keeps amplitudes, the
    projection turns phases); the edges there carry no phase."""
    isf = isfpkg.ISF(L, DIMS, HBAR, DT)
    psi0 = smooth_psi(DIMS, 14)
    psi0[8:8 + hole, 8:8 + hole, 8:8 + hole] = 0.0
    psi0, p0 = cuda(psi0), cuda(lattice())
    target = p0 + 0.5
    omega, iters = float(np.float32(1.8)), 2
    prob = isfpkg.adj_problem(1, 1, KVEC, omega, NOZZLE, init_iters=iters)
    loss, gpsi, _, jb = isfpkg.adj_gradient(isf, prob, psi0, p0, target)
    # forward, with the states the transposes need
    psi, states = psi0.clone(), []
    for _ in range(iters):
        torch.cuda.synchronize()
        before = psi.clone()
        torch.cuda.synchronize()
        isfpkg.restrict_velocity(isf, psi, KVEC, None, 0.0, nozzle=NOZZLE, phase_mode=1)
        isf.sync()
        states.append((before, psi.clone()))
        torch.cuda.synchronize()
        isfpkg.pressure_project(isf, psi)
        isf.sync()
    t = np.float32(DT)
    wt = float(np.float32(np.float32(omega) * t))
    end, parts = psi.clone(), p0.clone()
    torch.cuda.synchronize()
    isfpkg.step(isf, end, parts, jet_of(wt))
    isf.sync()
    assert float(((parts - target).double() ** 2).sum()) == pytest.approx(loss, rel=1e-6)
    # backward
    bar, lam = torch.zeros_like(psi0), 2.0 * (parts - target)
    torch.cuda.synchronize()
    want = np.array(isfpkg.adj_step(isf, psi, p0, jet_of(wt), bar, lam))
    want[3] *= float(t)
    isf.sync()
    size = size_of(bar)
    for before, after in reversed(states):
        isfpkg.adj_pressure_project(isf, after, bar)
        isf.sync()
        size += size_of(bar)
        torch.cuda.synchronize()
        want[:3] += isfpkg.adj_restrict_velocity(isf, before, bar, KVEC, 0.0, nozzle=NOZZLE, phase_mode=1)[:3]
    isf.sync()
    assert torch.equal(bar, gpsi)
    assert close(jb, want, size), (jb, want, size)
