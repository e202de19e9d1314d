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
