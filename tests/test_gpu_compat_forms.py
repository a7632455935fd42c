"""The FP64 walk's launch forms: tiles of 1..32 walkers, record batches, and 4,
5 or 6 resident blocks per SM, against the oracle.

Walker by walker the walk is the oracle's (voxels, events and counts equal);
sums of FP64 products agree to 1e-9 of the row's scale, as everywhere in this
suite (last bits of sin, cos and exp, and the order of sums)."""
import numpy as np
import pytest

import pyoracle
from conftest import assert_fp64_close
from rms_b200 import engine, geometry

pytestmark = pytest.mark.gpu
D, T2 = [0.0, 2.0, 1.0], [80.0, 80.0, 40.0]


def lattice():
    lab = geometry.axon_lattice(16, 16, 24, 0.1, seed=4, exterior=2, r0=0.45)
    lab[:2] = 0
    return lab


def table(n, seed=0):
    rng = np.random.default_rng(seed)
    v = rng.normal(size=(n, 3))
    return rng.uniform(0.5, 2.0, n), v / np.linalg.norm(v, axis=1, keepdims=True)


@pytest.mark.parametrize("npar,T,tn,nb,boundary", [(1, 1, 1, 1, "mirror"), (33, 9, 20, 33, "periodic"),
                                                   (1777, 16, 50, 31, "mirror"), (6000, 7, 30, 90, "periodic")])
def test_sums_and_counts(npar, T, tn, nb, boundary):
    b, v = table(nb)
    lab = lattice()
    sim = engine.Sim(lab, dt=2e-4, tn=tn, npar=npar, res=0.1, diffusivity=D, t2=T2, bval=b, bvec=v, timepoints=T,
                     boundary=boundary)
    got = sim.run(seed=6, precision="compat").outputs()
    step, t2s, pij, td = pyoracle.reference_tables(2e-4, 0.1, D, T2, T, tn)
    job = pyoracle.Job(lab, dt=2e-4, tn=tn, npar=npar, res=0.1, step=step, t2_steps=t2s, pij=pij, seed=6,
                       timepoints=T, td=td, bval=b, bvec=v, boundary=1 if boundary == "periodic" else 0)
    want = pyoracle.run_oracle(job, nthreads=8)
    assert np.array_equal(got["npar_count"], want["npar_count"])
    for k in ("sig0", "dx2", "dx4", "sigre"):
        assert_fp64_close(got[k], want[k], 1e-9, k)


@pytest.mark.parametrize("npar", [77_000, 100_000, 230_000])
def test_launches_of_every_form(npar):
    """One round of 4 blocks, one of 6, and several rounds of 5 (a warp then adds
    its later tiles to its rows): the walkers of two halves and of the whole."""
    b, v = table(3)
    kw = dict(dt=2e-4, tn=12, npar=npar, res=0.1, diffusivity=D, t2=T2, bval=b, bvec=v, timepoints=5)
    lab = lattice()
    whole = engine.Sim(lab, **kw).run(seed=1, precision="compat").outputs()
    parts = [engine.Sim(lab, **kw).run(seed=1, precision="compat", shard=(i, 4)).outputs() for i in range(4)]
    assert np.array_equal(sum(p["npar_count"] for p in parts), whole["npar_count"])
    for k in ("sig0", "dx2", "dx4", "sigre"):
        scale = np.abs(whole[k]).max()
        assert np.abs(sum(p[k] for p in parts) - whole[k]).max() <= 1e-9 * scale, k


def test_infinite_t2_weighs_one():
    lab = lattice()
    o = engine.Sim(lab, dt=2e-4, tn=10, npar=100, res=0.1, diffusivity=D, t2=[np.inf] * 3, timepoints=10,
                   bval=[], bvec=np.zeros((0, 3))).run(seed=1, precision="compat").outputs()
    np.testing.assert_array_equal(o["sig0"], np.full(10, 100.0))


@pytest.mark.parametrize("ng", [1, 31, 33])
def test_pgse_gradients_per_lane(ng):
    rng = np.random.default_rng(ng)
    g = np.column_stack([rng.choice([0.004, 0.006], ng), rng.choice([0.002, 0.003], ng), rng.uniform(0.5, 40, ng),
                         rng.normal(size=(ng, 3))])
    g[:, 3:] /= np.linalg.norm(g[:, 3:], axis=1, keepdims=True)
    lab = lattice()
    sim = engine.Sim(lab, dt=2e-4, tn=50, npar=2500, res=0.1, diffusivity=D, t2=T2, grad=g, timepoints=10)
    got = sim.run(seed=8, precision="compat").outputs()
    step, t2s, pij, td = pyoracle.reference_tables(2e-4, 0.1, D, T2, 10, 50)
    job = pyoracle.Job(lab, dt=2e-4, tn=50, npar=2500, res=0.1, step=step, t2_steps=t2s, pij=pij, seed=8,
                       timepoints=10, td=td, grad=g)
    want = pyoracle.run_oracle(job, nthreads=8)
    assert_fp64_close(got["sig"], want["sig"], 1e-9, "sig")


@pytest.mark.parametrize("precision", ["compat", "split"])
@pytest.mark.parametrize("npar", [3, 5000, 100_000])
def test_b_values_shared_between_lanes(npar, precision):
    """Lanes beyond the b-values of a group share its walkers: each b-value's
    signal from tables of 1 to 49 of them, which split the lanes in every way,
    equals its signal from a table of its own (FP64 sums in another order)."""
    b, v = table(49, seed=1)
    lab = lattice()
    kw = dict(dt=2e-4, tn=9, npar=npar, res=0.1, diffusivity=D, t2=T2, timepoints=9)
    full = engine.Sim(lab, bval=b, bvec=v, **kw).run(seed=6, precision=precision).outputs()["sigre"]
    for n in (1, 2, 3, 8, 9, 16, 17, 33, 48):
        got = engine.Sim(lab, bval=b[:n], bvec=v[:n], **kw).run(seed=6, precision=precision).outputs()["sigre"]
        assert np.abs(got - full[:, :n]).max() <= 1e-12 * npar, n


@pytest.mark.parametrize("D0", [0.0, 5.0, 6.7, 20.0])
def test_table_that_lets_walkers_into_compartment_0(D0):
    """Only a permeation table opens compartment 0, whose step length is not held
    below a voxel (D0 = 20: 1.55 voxels): the same walk, or the same refusal of a
    segment that finds no face."""
    lab = lattice()
    dd, tn, npar = [D0, 2.0, 1.0], 12, 400
    pij = np.array([[1.0, 0.4, 0.4], [0.5, 1.0, 0.7], [0.5, 0.7, 1.0]])
    sim = engine.Sim(lab, dt=2e-4, tn=tn, npar=npar, res=0.1, diffusivity=dd, t2=T2, timepoints=tn,
                     permeation="table", pij=pij, bval=[], bvec=np.zeros((0, 3)))
    step, t2s, _, td = pyoracle.reference_tables(2e-4, 0.1, dd, T2, tn, tn)
    job = pyoracle.Job(lab, dt=2e-4, tn=tn, npar=npar, res=0.1, step=step, t2_steps=t2s, pij=pij.ravel(), seed=6,
                       timepoints=tn, td=td)
    try:
        got = sim.run(seed=6, precision="compat", trace_walkers=npar)
    except engine.RmsError as e:
        assert D0 == 20.0 and e.code == -4
        return
    want = pyoracle.run_oracle(job, trace_walkers=npar)
    tr = got.trace(npar)
    assert np.array_equal(tr["voxel"], want["trace"]["voxel"])
    assert np.array_equal(tr["events"], want["trace"]["events"])
