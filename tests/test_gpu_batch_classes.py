"""How many classes of simulations the persistent batch kernel takes."""
import pytest
import torch

from helpers import smooth_psi

pytestmark = pytest.mark.gpu

SHAPES = [(nx, n, n) for n in (32, 48, 64) for nx in (16, 32, 48, 64, 96, 128)]


def ensemble(cfgs, count, nslots):
    kvec, omega = cfgs.jet_omega()
    jet = dict(kvec=kvec, omega=omega, cen=(0.3, 0.5, 0.5), len=0.4, rad=0.3, phase_mode=1, emit_mode=1,
               emit_per_step=8 if nslots else 0, seed=3)
    return [dict(dims=d, physical_size=(1, 1, 1), hbar=cfgs.HBAR, dt=cfgs.CONFIGS["C1"]["dt"], nslots=nslots, jet=jet)
            for d in SHAPES[:count]]


# the largest ensembles of jets of one class each: 17 without particles, 15
# that emit and advect
@pytest.mark.parametrize("count,nslots", [(17, 0), (15, 64)])
def test_persistent_kernel_takes_as_many_jet_classes(isfpkg, cfgs, count, nslots):
    sims = ensemble(cfgs, count, nslots)
    batches = [isfpkg.ISFBatch(sims, tune=False) for _ in range(2)]
    assert batches[0].classes()[0] == count
    batches[0].set_persistent(True)
    for b in batches:
        for i, s in enumerate(sims):
            b.set_psi(i, torch.tensor(smooth_psi(s["dims"], seed=i), dtype=torch.float32, device="cuda"))
            if nslots:
                b.set_particles(i, torch.full((nslots, 3), -1.0, device="cuda"))
        b.step(2)
        b.sync()
    for i in range(count):
        assert torch.equal(batches[0].psi(i), batches[1].psi(i)), i
        if nslots:
            assert torch.equal(batches[0].particles(i), batches[1].particles(i)), i
    for b in batches:
        b.close()
