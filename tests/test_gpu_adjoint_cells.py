"""The reverse pass on half-byte cells (lattices past the byte cells' limit): its
own walk's signal sums are the forward run's.  The reverse pass sums FP32 phases
(|phi| below 10 rad, 20 bins): 20 x 10 x 2^-24 ~ 1e-5 rad per walker."""
import numpy as np
import pytest

from rms_b200 import engine, geometry, waveforms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n3", [400, 470])
def test_signal_sums_of_a_large_lattice(n3):
    n, nb, nw = 3000, 20, 4
    w = waveforms.scale_to_b(waveforms.random_smooth(nw, nb, 1.0, seed=1), 0.01, np.linspace(0.2, 1.5, nw))
    with engine.Sim(dt=5e-4, tn=20 * nb, npar=n, res=0.1, diffusivity=[0, 2.0, 2.0], t2=[80, 80, 60],
                    shape=(396, 396, n3), wave=w, timepoints=20, boundary="periodic", permeation="kappa",
                    kappa=0.05) as sim:
        sim.set_tube_lattice(*geometry.axon_slices(396, 396, n3, 0.1, 1), inside=1, outside=2)
        fwd = sim.run(seed=3, precision="split").get("sigw").reshape(nw, 2)
        g = np.random.default_rng(0).normal(size=2 * nw) / n
        rev = sim.adjoint(g, seed=3)
        jac = sim.jacobian(seed=3)
    for got in (rev["sigw"], jac["sigw"]):
        assert np.abs(got - fwd).max() < 1e-4 * n
    assert np.isfinite(rev["d_wave"]).all() and np.abs(rev["d_wave"]).max() > 0
