"""The FP64 walk in every launch form with warps that walk one tile and several:
a warp's first tile stores its rows, the later ones add to them.  Sums and counts
against the oracle (counts equal; FP64 sums to 1e-9 of the row's scale, as
everywhere in this suite).

The walker counts follow the launch's rule: a form of b = 4, 5 or 6 resident
blocks of four warps holds 4 b warps per SM, and the form whose rounds of tiles
end first is taken (a round of 5 weighs 1.16 rounds of 4, of 6 weighs 1.44)."""
import numpy as np
import pytest

import pyoracle
from conftest import assert_fp64_close
from rms_b200 import engine, geometry

pytestmark = pytest.mark.gpu
D, T2 = [0.0, 2.0, 1.0], [80.0, 80.0, 40.0]


def tiles(form, rounds, sms):
    """A number of full tiles for which the rule takes `form` with `rounds` rounds."""
    def rule(n):
        cost = {b: -(-n // (4 * b * sms)) * w for b, w in ((4, 1.0), (5, 1.16), (6, 1.44))}
        best = min(cost, key=lambda b: (cost[b], b))
        return best, -(-n // (4 * best * sms))
    hits = [n for n in range(12 * sms, 60 * sms, sms // 4) if rule(n) == (form, rounds)]
    return hits[len(hits) // 2]


@pytest.mark.parametrize("mode", ["narrow", "pgse"])
@pytest.mark.parametrize("form,rounds", [(4, 1), (4, 2), (5, 1), (5, 2), (6, 1), (6, 2)])
def test_rounds_of_every_form(form, rounds, mode):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    npar, tn, T = 32 * tiles(form, rounds, sms) - 5, 12, 5
    lab = geometry.axon_lattice(16, 16, 24, 0.1, seed=4, exterior=2, r0=0.45)
    lab[:2] = 0
    rng = np.random.default_rng(form * 10 + rounds)
    d = rng.normal(size=(17, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    if mode == "narrow":
        kw = dict(bval=rng.uniform(0.5, 2.0, 3), bvec=d[:3])
    else:
        kw = dict(grad=np.column_stack([rng.choice([0.0012, 0.0015], 17), np.full(17, 0.0006),
                                        rng.uniform(50, 4000, 17), d]))
    got = engine.Sim(lab, dt=2e-4, tn=tn, npar=npar, res=0.1, diffusivity=D, t2=T2, timepoints=T,
                     **kw).run(seed=6, precision="compat").outputs()
    step, t2s, pij, td = pyoracle.reference_tables(2e-4, 0.1, D, T2, T, tn)
    job = pyoracle.Job(lab, dt=2e-4, tn=tn, npar=npar, res=0.1, step=step, t2_steps=t2s, pij=pij, seed=6,
                       timepoints=T, td=td, **kw)
    want = pyoracle.run_oracle(job, nthreads=8)
    assert np.array_equal(got["npar_count"], want["npar_count"])
    for k in ("sig0", "dx2", "dx4", "sigre" if mode == "narrow" else "sig"):
        assert_fp64_close(got[k], want[k], 1e-9, k)


def open_compartment_0(D0, boundary, seed):
    """A job whose permeation table lets walkers into compartment 0, whose step
    length alone may be a voxel or more."""
    lab = geometry.axon_lattice(16, 16, 24, 0.1, seed=4, exterior=2, r0=0.45)
    lab[:2] = 0
    dd, tn, npar = [D0, 2.0, 1.0], 40, 600
    pij = np.array([[1.0, 0.4, 0.4], [0.5, 1.0, 0.7], [0.5, 0.7, 1.0]])
    sim = engine.Sim(lab, dt=2e-4, tn=tn, npar=npar, res=0.1, diffusivity=dd, t2=T2, timepoints=tn, boundary=boundary,
                     permeation="table", pij=pij, bval=[], bvec=np.zeros((0, 3)))
    step, t2s, _, td = pyoracle.reference_tables(2e-4, 0.1, dd, T2, tn, tn)
    job = pyoracle.Job(lab, dt=2e-4, tn=tn, npar=npar, res=0.1, step=step, t2_steps=t2s, pij=pij.ravel(), seed=seed,
                       timepoints=tn, td=td, boundary=1 if boundary == "periodic" else 0)
    return sim, job, step[0]


@pytest.mark.parametrize("boundary", ["mirror", "periodic"])
@pytest.mark.parametrize("D0", [8.3, 8.4, 12.0, 20.0, 33.0])
def test_steps_of_a_voxel_or_more_are_the_oracles(D0, boundary):
    """Steps of 0.998 to 1.990 voxels: the segment that finds no face ends inside a
    reach of two, so nothing is refused and every voxel and event is the oracle's."""
    for seed in (6, 7, 8):
        sim, job, step = open_compartment_0(D0, boundary, seed)
        assert 0.99 < step < 2.0
        got = sim.run(seed=seed, precision="compat", trace_walkers=600)
        want = pyoracle.run_oracle(job, trace_walkers=600)
        tr = got.trace(600)
        assert np.array_equal(tr["voxel"], want["trace"]["voxel"])
        assert np.array_equal(tr["events"], want["trace"]["events"])
        assert np.array_equal(got.get("npar_count").reshape(40, 3), want["npar_count"])


def test_a_step_that_finds_no_face_is_refused():
    """2.7 voxels: a direction with no face within the step has a reach beyond two."""
    sim, _, step = open_compartment_0(60.0, "mirror", 6)
    assert step > 2.0
    with pytest.raises(engine.RmsError) as e:
        sim.run(seed=6, precision="compat")
    assert e.value.code == -4
