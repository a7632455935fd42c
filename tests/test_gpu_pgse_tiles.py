"""PGSE signals of warps that walk several tiles: a warp's window sums are read
by all its lanes at a tile's end and cleared for the next tile, and COMPAT rows
are stored by the first tile and added to by the later ones.

The shards of a job walk the whole job's walkers in fewer tiles a warp, so their
signals add up to the whole's: FP64 sums of the same terms (each at most one) in
another order, at most 1e-12 per walker apart; compartment counts are equal."""
import numpy as np
import pytest

from rms_b200 import engine, geometry

pytestmark = pytest.mark.gpu

WALKERS = 400_003   # 12501 tiles of 32: COMPAT holds at most 3552 warps (6 blocks of 4 on 148 SMs), SPLIT 4736


def gradients(n, seed=3):
    """n gradients in three timing pairs, phases of a few radians."""
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.array([[(0.004, 0.005, 0.006)[j % 3], 0.002, 1500.0 + 100.0 * (j % 7), *d[j]] for j in range(n)])


@pytest.mark.parametrize("precision", ["compat", "split"])
@pytest.mark.parametrize("ng", [1, 16, 17, 32, 33])
def test_shards_of_many_tiles_add_up(ng, precision):
    lab = geometry.axon_lattice(24, 24, 32, 0.1, seed=4, exterior=2, r0=0.6)
    kw = dict(dt=2e-4, tn=48, npar=WALKERS, res=0.1, diffusivity=[0.0, 2.0, 1.0], t2=[80.0, 80.0, 40.0],
              grad=gradients(ng), timepoints=6)
    whole = engine.Sim(lab, **kw).run(seed=11, precision=precision).outputs()
    parts = [engine.Sim(lab, **kw).run(seed=11, precision=precision, shard=(i, 16)).outputs() for i in range(16)]
    assert np.array_equal(sum(p["npar_count"] for p in parts), whole["npar_count"])
    assert np.abs(sum(p["sig"] for p in parts) - whole["sig"]).max() <= 1e-12 * WALKERS


def test_no_allocation_form_of_many_tiles():
    """The no-allocation walk (fixed scratch, so many tiles a warp) against the queue's."""
    import torch
    lab = geometry.axon_lattice(24, 24, 32, 0.1, seed=4, exterior=2, r0=0.6)
    ng = 33
    sim = engine.Sim(lab, dt=2e-4, tn=48, npar=WALKERS, res=0.1, diffusivity=[0.0, 2.0, 1.0], t2=[80.0, 80.0, 40.0],
                     grad=gradients(ng), timepoints=6)
    want = sim.run(seed=11, precision="split").outputs()["sig"]
    d_lab = torch.tensor(np.ascontiguousarray(lab), device="cuda")
    rows = torch.zeros((6, 32), dtype=torch.float64, device="cuda")
    sig = torch.zeros(64, dtype=torch.float64, device="cuda")
    sim.run_noalloc(d_lab.data_ptr(), rows.data_ptr(), sig.data_ptr(), seed=11)
    assert np.abs(sig.cpu().numpy()[:ng] - want).max() <= 1e-12 * WALKERS
