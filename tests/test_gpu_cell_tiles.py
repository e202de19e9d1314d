"""Kernels over cells on grids of each tile width (32 x 8, 16 x 16, 8 x 32),
whole and partial tiles."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HBAR, DT = float(np.float32(0.1)), float(np.float32(1 / 48))


def cuda(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float32, device="cuda")


# widths 16, 8, 8, 16, 8, 32, 32
@pytest.mark.parametrize("L,dims", [((1, 2, 1), (16, 64, 20)), ((1, 2, 1), (8, 50, 12)), ((1, 2, 1), (24, 64, 8)),
                                    ((1, 1, 1), (40, 12, 20)), ((1, 3, 1), (20, 96, 8)), ((2, 1, 1), (50, 8, 24)),
                                    ((1, 1, 1), (16, 8, 100))])
def test_cells(isfpkg, L, dims):
    """Copies are exact, div and isjet those of numpy, a restriction by mask the
    one by nozzle, and the one-form's transpose moves with the cells."""
    isf = isfpkg.ISF(L, dims, HBAR, DT, stream=isfpkg.STREAM_LEGACY)
    rng = np.random.default_rng(71)
    v = rng.normal(size=dims[::-1] + (3,)).astype(np.float32)
    isf.velocity = cuda(v)
    assert np.array_equal(isf.velocity.cpu().numpy(), v)
    f = isf.div().cpu().numpy().astype(np.float64)
    w = v.astype(np.float64)
    d = [np.float64(np.float32(length / n)) for length, n in zip(L, dims)]
    want, size = 0.0, 0.0
    for a in range(3):
        lo = np.roll(w[..., a], 1, axis=2 - a)
        want = want + (w[..., a] - lo) / d[a] ** 2
        size = size + (np.abs(w[..., a]) + np.abs(lo)) / d[a] ** 2
    # three rounded differences, products with a rounded 1/d^2 and two sums
    assert (np.abs(f - want) <= 8 * 2.0 ** -24 * size).all()
    isfpkg.set_velocity_bar(isf, cuda(v))
    assert np.array_equal(isfpkg.get_velocity_bar(isf).cpu().numpy(), v)
    cen, length, rad = tuple(0.5 * x for x in L), 0.43 * L[0], 0.4 * min(L)
    mask = isfpkg.isjet(isf, cen, length, rad)
    pos = isf.positions
    isf.sync()
    x, y, z = (pos[..., k].double().cpu().numpy() - cen[k] for k in range(3))
    r2 = y * y + z * z - rad * rad
    clear = (np.abs(np.abs(x) - length / 2) > 1e-5) & (np.abs(r2) > 1e-5)
    assert clear.mean() > 0.8
    assert np.array_equal(mask.cpu().numpy()[clear] != 0, ((np.abs(x) <= length / 2) & (r2 <= 0))[clear])
    assert 0 < int(mask.sum()) < mask.numel()
    psi = rng.normal(size=dims[::-1] + (4,))
    a, b = cuda(psi), cuda(psi)
    isfpkg.restrict_velocity(isf, a, (6.0, 0.5, 0.1), mask, 0.2)
    isfpkg.restrict_velocity(isf, b, (6.0, 0.5, 0.1), None, 0.2, nozzle=(cen, length, rad))
    isf.sync()
    assert torch.equal(a, b)
    changed = (a != cuda(psi)).any(dim=-1)
    assert torch.equal(changed, mask != 0)
    # the transposes: a cell's part does not depend on the tile
    wb = cuda(rng.normal(size=dims[::-1] + (4,)))
    isfpkg.set_velocity_bar(isf, cuda(v))
    one = wb.clone()
    isfpkg.adj_velocity_one_form(isf, b, one, HBAR)
    for axis in range(3):
        isfpkg.set_velocity_bar(isf, torch.roll(cuda(v), 1, dims=axis))
        two, pb = torch.roll(wb, 1, dims=axis), torch.roll(b, 1, dims=axis)
        isfpkg.adj_velocity_one_form(isf, pb, two, HBAR)
        assert torch.equal(two, torch.roll(one, 1, dims=axis))
