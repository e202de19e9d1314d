"""Kernel sequences (csrc/isf_seq.cu) on the GPU, through the C ABI."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import smooth_psi

pytestmark = pytest.mark.gpu

L, DIMS = (2, 1, 1), (32, 16, 16)
HBAR, DT = float(np.float32(0.1)), float(np.float32(1 / 48))


def cuda(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float32, device="cuda")


def ptr(t):
    return C.c_void_p(t.data_ptr())


def test_velocity_after_a_call_that_fails_midway(isfpkg):
    """isf_f64_velocity_one_form without an output array fails at its last
    part, as isf_velocity_to_f64 does on its own: the one-form before it is done."""
    isf, ref = isfpkg.ISF(L, DIMS, HBAR, DT), isfpkg.ISF(L, DIMS, HBAR, DT)
    psi, work = cuda(smooth_psi(DIMS, seed=81)), cuda(smooth_psi(DIMS, seed=82))
    isfpkg.velocity_one_form(ref, psi, HBAR)
    want = ref.velocity
    isfpkg.velocity_one_form(isf, work, HBAR)
    p = psi.double()
    p1, p2 = (torch.complex(p[..., 2 * k], p[..., 2 * k + 1]).contiguous() for k in (0, 1))
    torch.cuda.synchronize()
    rc = isf.L.isf_f64_velocity_one_form(isf.h, ptr(p1), ptr(p2), ptr(work), HBAR, None, None, None)
    assert rc == isfpkg._lib.ISF_ERR_INVALID
    assert torch.equal(isf.velocity, want)


BUILD_AT = 16   # the call of a sequence that goes out as a graph first


def jet(k):
    return dict(kvec=(6.0, 0.5, 0.0), omega_t=0.1 * k, cen=(0.6, 0.5, 0.5), len=0.4 + 0.01 * k, rad=0.3, phase_mode=1,
                emit_start=10 * k, emit_count=10 + k, seed=5, counter=k, emit_mode=1)


CALLS = {
    "flow": lambda p, h, a, k: p.schroedinger_flow(h, a["psi"]),
    "project": lambda p, h, a, k: p.pressure_project(h, a["psi"]),
    "init": lambda p, h, a, k: p.init_jet(h, a["psi"], 1, (6.0, 0.5, 0.0), nozzle=((0.6, 0.5, 0.5), 0.4, 0.3),
                                          phase_mode=1),
    "poisson": lambda p, h, a, k: a.__setitem__("f", h.poisson_solve(a["f"])),
    "step": lambda p, h, a, k: p.step(h, a["psi"], a["parts"], jet(k)),
}
# graph launches of a call: the step's particles are a sequence of their own
GRAPHS = {"step": 2}


def state(dims):
    rng = np.random.default_rng(83)
    a = {"psi": cuda(smooth_psi(dims, seed=84)), "f": cuda(rng.normal(size=dims[::-1])),
         "parts": cuda(rng.uniform(0.1, 0.9, (500, 3)))}
    torch.cuda.synchronize()
    return a


@pytest.mark.parametrize("dims", [(32, 16, 16), (20, 12, 24), (16, 32, 32)])
@pytest.mark.parametrize("what", sorted(CALLS))
def test_calls_go_out_as_graphs(isfpkg, dims, what):
    """From its 16th call on a sequence is one graph launch, none fails, and
    the results are those of a handle that launches kernel by kernel."""
    a, b = (isfpkg.ISF((2, 1, 1), dims, HBAR, DT) for _ in range(2))
    b.profile_start()
    sa, sb = state(dims), state(dims)
    for k in range(1, BUILD_AT + 6):
        CALLS[what](isfpkg, a, sa, k)
        CALLS[what](isfpkg, b, sb, k)
        assert a.graph_count() == (GRAPHS.get(what, 1) * max(0, k - BUILD_AT + 1), 0)
    a.sync()
    b.sync()
    assert b.graph_count() == (0, 0)
    b.profile_stop()
    for key in sa:
        assert torch.equal(sa[key], sb[key]), key


def test_no_graphs_under_capture_nor_on_large_grids(isfpkg):
    st = torch.cuda.Stream()
    isf = isfpkg.ISF((2, 1, 1), (32, 16, 16), HBAR, DT, stream=st)
    a = state((32, 16, 16))
    for k in range(BUILD_AT + 1):
        isfpkg.schroedinger_flow(isf, a["psi"])
    isf.sync()
    before = isf.graph_count()
    assert before == (2, 0)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        isfpkg.schroedinger_flow(isf, a["psi"])
    assert isf.graph_count() == before
    isfpkg.schroedinger_flow(isf, a["psi"])
    assert isf.graph_count() == (3, 0)
    isf.sync()
    large = isfpkg.ISF((2, 2, 2), (128, 64, 64), HBAR, DT)
    psi = isfpkg.new_psi(large)
    for k in range(BUILD_AT + 4):
        isfpkg.schroedinger_flow(large, psi)
    large.sync()
    assert large.graph_count() == (0, 0)


def test_tma_z_pass_in_a_graph(isfpkg):
    """The tensor map of the TMA-staged z pass as a graph node's argument: two
    psi arrays in turn, so the map changes from call to call."""
    dims = (32, 16, 64)
    tma = isfpkg.ISF((1, 1, 1), dims, HBAR, DT, flags=isfpkg.FLAG_TMA_Z_PASS)
    ref = isfpkg.ISF((1, 1, 1), dims, HBAR, DT)
    ref.profile_start()
    psis = [[cuda(smooth_psi(dims, seed=85 + k)) for k in range(2)] for _ in range(2)]
    torch.cuda.synchronize()
    for k in range(BUILD_AT + 9):
        isfpkg.schroedinger_flow(tma, psis[0][k % 2])
        isfpkg.schroedinger_flow(ref, psis[1][k % 2])
    tma.sync()
    ref.sync()
    assert tma.graph_count() == (10, 0)
    assert tma.counters()["wait_timeouts"] == 0
    ref.profile_stop()
    for k in range(2):
        assert torch.equal(psis[0][k], psis[1][k])


def test_matlabport_operators_in_graphs(isfpkg):
    m = isfpkg.matlabport
    dims = (32, 16, 16)
    isf = m.ISF((2, 1, 1), dims, HBAR, DT)
    h = isf._g.h
    psi = cuda(smooth_psi(dims, seed=88)).double()
    p = [torch.complex(psi[..., 2 * k], psi[..., 2 * k + 1]).contiguous().permute(2, 1, 0) for k in (0, 1)]

    def run():
        a = m.Normalize(*m.SchroedingerFlow(isf, *p))
        a = m.PressureProject(isf, *a)
        return (*a, *m.StaggeredSharp(isf, *m.VelocityOneForm(isf, *a, HBAR)))

    first = run()
    for k in range(BUILD_AT + 2):
        last = run()
    n, bad = C.c_uint64(), C.c_uint64()
    assert isf._g.L.isf_graph_count(h, C.byref(n), C.byref(bad)) == 0
    assert n.value > 0 and bad.value == 0
    for x, y in zip(first, last):
        assert torch.equal(x, y)
