"""The FP64 walk's T2 weight at the ends of the accepted range (T2 > 0): the
weight exp(-sum_c t_c / T2_c) of the division, whatever the T2 of a compartment."""
import numpy as np
import pytest

from rms_b200 import engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [1e-320, 1e-306, 1e-300, 1e-280, 1e-30, 1e30, 1e280, 1e307, np.inf])
def test_t2_of_any_size(far):
    """A compartment no walker enters adds t / T2 = 0 to the exponent; one whose T2
    is far below a step weighs nothing, one far above it everything."""
    def run(label, t2, nc):
        lab = np.full((8, 8, 8), label, np.uint8)
        with engine.Sim(lab, dt=2e-4, tn=16, npar=200, res=0.1, diffusivity=[0.0, 2.0, 2.0][:nc], t2=t2[:nc], nc=nc,
                        timepoints=16, bval=[], bvec=np.zeros((0, 3))) as sim:
            return sim.run(seed=3, precision="compat").outputs()["sig0"]

    usual = run(1, [80.0, 80.0], 2)
    assert 0.0 < usual[-1] < 200.0
    np.testing.assert_array_equal(run(1, [80.0, 80.0, far], 3), usual)
    np.testing.assert_array_equal(run(2, [80.0, 80.0, far], 3), np.full(16, 0.0 if far < 1 else 200.0))
