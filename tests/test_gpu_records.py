"""Record batches of the split walk: several records are staged per warp and
summed together, so the edges are record counts around the batch size, b-tables
around the warp width, walker counts around a tile, and every launch variant
(two batch sizes).

The oracle is the FP64 replay of the same walkers on a lattice with no membrane
in reach (one label, periodic walls), where the FP32 and FP64 walks cannot part:
a record's displacement carries the FP32 rounding of at most `tn` steps and of
its products.  |x| stays below 0.058 um per step, each step rounds at 2^-24 of a
voxel offset (0.1 um), so after tn <= 40 steps a displacement is within
40 x 6e-9 um of 0.05 um x sqrt(40), 1e-6 relative, and a fourth moment within
5e-6; a cosine of q x <= 15 rad within 2e-5.  Tolerances: 1e-5 of the record's
largest moment of the same order, 5e-5 of the walker count for a signal.
Two recordings of one walk differ by the order of FP64 sums alone: 1e-12.
"""
import numpy as np
import pytest

import pyoracle
from rms_b200 import engine

pytestmark = pytest.mark.gpu

LAB = np.ones((12, 12, 12), dtype=np.uint8)


def table(nb):
    rng = np.random.default_rng(nb)
    v = rng.normal(size=(nb, 3))
    return rng.uniform(0.5, 2.0, nb), v / np.linalg.norm(v, axis=1, keepdims=True)


def make(T, tn, npar, nb, lab=LAB, D=(0.0, 2.0), T2=(80.0, 60.0)):
    b, v = table(nb) if nb else (np.zeros(0), np.zeros((0, 3)))
    sim = engine.Sim(lab, dt=2e-4, tn=tn, npar=npar, res=0.1, diffusivity=list(D), t2=list(T2), bval=b, bvec=v,
                     timepoints=T, boundary="periodic")
    return sim, b, v


@pytest.mark.parametrize("T,tn,npar,nb", [(1, 1, 1, 1), (3, 10, 31, 0), (7, 7, 33, 31), (8, 16, 32, 32),
                                          (9, 9, 95, 33), (16, 33, 1000, 90), (17, 40, 257, 64)])
def test_records_equal_the_fp64_replay(T, tn, npar, nb):
    sim, b, v = make(T, tn, npar, nb)
    step, t2s, pij, td = pyoracle.reference_tables(2e-4, 0.1, [0.0, 2.0], [80.0, 60.0], T, tn)
    job = pyoracle.Job(LAB, dt=2e-4, tn=tn, npar=npar, res=0.1, step=step, t2_steps=t2s, pij=pij, seed=9,
                       timepoints=T, td=td, bval=b, bvec=v, boundary=pyoracle.BOUNDARY_PERIODIC)
    want = pyoracle.run_oracle(job, split=True)
    for variant in range(1, len(engine.split_variants()) + 1):
        got = sim.run(seed=9, precision="split", variant=variant).outputs()
        assert np.array_equal(got["npar_count"], want["npar_count"]), variant
        np.testing.assert_allclose(got["sig0"], want["sig0"], rtol=1e-6)
        for k in ("dx2", "dx4"):
            scale = np.abs(want[k]).max(axis=1, keepdims=True)
            assert (np.abs(got[k] - want[k]) <= 1e-5 * scale).all(), (variant, k)
        if nb:
            assert np.abs(got["sigre"] - want["sigre"]).max() <= 5e-5 * npar, variant


@pytest.mark.parametrize("nc", [3, 8])
def test_every_other_record_of_one_walk(nc):
    """tstep = 1 against tstep = 2: the same records fall in other batches.
    Eight compartments take the byte lattice and every count column."""
    rng = np.random.default_rng(nc)
    lab = rng.integers(1, nc, size=(16, 16, 16)).astype(np.uint8)
    D, T2 = [0.0] + [2.0] * (nc - 1), [80.0] * nc
    fine = make(50, 50, 4000, 40, lab, D, T2)[0].run(seed=3, precision="split").outputs()
    coarse = make(25, 50, 4000, 40, lab, D, T2)[0].run(seed=3, precision="split").outputs()
    assert np.array_equal(coarse["npar_count"], fine["npar_count"][::2])
    for k in ("sig0", "dx2", "dx4"):
        np.testing.assert_allclose(coarse[k], fine[k][::2], rtol=1e-12, atol=1e-18)


@pytest.mark.parametrize("npar", [1, 2, 1776, 1777, 3553, 20000])
def test_narrow_tiles_walk_the_same_walkers(npar):
    """Small launches walk fewer than 32 walkers a warp.  A launch's walkers are
    those of its shards, whose tiles have other widths and edges; the sums differ
    by their order alone."""
    sim = make(9, 20, npar, 3, T2=(80.0, 40.0))[0]
    whole = sim.run(seed=2, precision="split").outputs()
    parts = [make(9, 20, npar, 3, T2=(80.0, 40.0))[0].run(seed=2, precision="split", shard=(i, 3)).outputs()
             for i in range(3)]
    assert np.array_equal(sum(p["npar_count"] for p in parts), whole["npar_count"])
    assert np.array_equal(whole["npar_count"].sum(axis=1), np.full(9, float(npar)))
    for k in ("sig0", "dx2", "dx4", "sigre"):
        scale = np.abs(whole[k]).max()
        assert np.abs(sum(p[k] for p in parts) - whole[k]).max() <= 1e-12 * scale * max(1, npar ** 0.5), k
