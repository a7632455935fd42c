"""The padded lattice's cells (labels, walls, free-flight flags) on odd lattices.

Between impermeable compartments nothing crosses, so each compartment keeps its
walkers exactly: a flag set on a voxel next to another label, or a wall code in
the wrong place, sends walkers across (or out of the lattice)."""
import numpy as np
import pytest

from rms_b200 import engine

pytestmark = pytest.mark.gpu


def blobs(shape, nc, seed, grain):
    """Random lattice with features of about `grain` voxels, labels 1..nc-1."""
    rng = np.random.default_rng(seed)
    coarse = rng.integers(1, nc, size=[s // grain + 2 for s in shape]).astype(np.uint8)
    big = np.kron(coarse, np.ones((grain,) * 3, dtype=np.uint8))
    off = rng.integers(0, grain, size=3)
    return np.ascontiguousarray(big[off[0]:, off[1]:, off[2]:][:shape[0], :shape[1], :shape[2]])


@pytest.mark.parametrize("boundary", ["mirror", "periodic"])
@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 1), (5, 4, 2), (4, 7, 3), (6, 5, 5), (9, 8, 6), (8, 9, 7),
                                   (11, 10, 8), (10, 11, 13), (20, 17, 31), (16, 16, 62), (33, 9, 130)])
@pytest.mark.parametrize("nc", [3, 8])
def test_impermeable_compartments_keep_their_walkers(shape, nc, boundary):
    lab = blobs(shape, nc, sum(shape) + nc, 4)
    kw = dict(dt=2e-4, tn=120, npar=6000, res=0.1, diffusivity=[0.0] + [2.5] * (nc - 1), t2=[80.0] * nc,
              timepoints=12, boundary=boundary, permeation="kappa", kappa=0.0, bval=[], bvec=np.zeros((0, 3)))
    cnt = engine.Sim(lab, **kw).run(seed=4, precision="split").outputs()["npar_count"]
    assert np.array_equal(cnt.sum(axis=1), np.full(12, 6000.0))
    assert (cnt == cnt[0]).all()
    assert set(np.flatnonzero(cnt[0])) <= set(np.unique(lab).tolist())


def test_one_label_is_free_diffusion_to_the_walls():
    """Every voxel flagged, walls on all sides: <x^2> of a step is step^2 / 3."""
    lab = np.ones((7, 6, 9), dtype=np.uint8)
    o = engine.Sim(lab, dt=2e-4, tn=1, npar=400000, res=0.1, diffusivity=[0, 2.0], t2=[80, 80], timepoints=1,
                   boundary="periodic", bval=[], bvec=np.zeros((0, 3))).run(seed=3, precision="split").outputs()
    want = 6 * 2.0 * 2e-4 / 3
    x2 = o["dx2"][0, [0, 3, 5]] / o["sig0"][0]
    # var(cos^2) = 4/45: standard error of the mean 0.9 / sqrt(4e5) relative, 6 of them
    assert np.abs(x2 / want - 1).max() < 6 * 0.9 / 400000 ** 0.5


def test_both_cell_widths_walk_the_same_walkers():
    """A lattice between the limits for one axon and for several: byte cells in
    its own launch, half bytes beside a second axon."""
    from rms_b200 import geometry
    kw = dict(dt=2e-4, tn=200, npar=20000, res=0.1, diffusivity=[0, 2.0, 1.5], t2=[80, 80, 60], timepoints=10,
              bval=[], bvec=np.zeros((0, 3)), permeation="kappa", kappa=0.05)
    big = engine.Sim(shape=(372, 372, 370), **kw)
    big.set_tube_lattice(*geometry.axon_slices(372, 372, 370, 0.1, 1), inside=1, outside=2)
    small = engine.Sim(shape=(32, 32, 40), **kw)
    small.set_tube_lattice(*geometry.axon_slices(32, 32, 40, 0.1, 2), inside=1, outside=2)
    alone = big.run(seed=5, precision="split").outputs()
    engine.batch_run([big, small], seed=5, precision="split")
    both = big.outputs()
    assert np.array_equal(alone["npar_count"], both["npar_count"])
    for k in ("sig0", "dx2", "dx4"):
        np.testing.assert_allclose(both[k], alone[k], rtol=1e-10, atol=1e-12 * np.abs(alone[k]).max())
