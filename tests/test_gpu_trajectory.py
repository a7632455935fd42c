"""The trajectory output's two store forms (eight bins in 16-byte stores, or bin
by bin) hold the same bytes, and the waveform phases do not depend on how many
waveforms a run has."""
import numpy as np
import pytest

from rms_b200 import engine, geometry, waveforms

pytestmark = pytest.mark.gpu


def sim(nb, npar, wave=None):
    lab = geometry.axon_lattice(20, 20, 40, 0.1, seed=3, exterior=2, r0=0.5)
    return engine.Sim(lab, dt=5e-4, tn=4 * nb, npar=npar, res=0.1, diffusivity=[0, 2.0, 2.0], t2=[1e6, 80, 60],
                      wave=np.zeros((1, nb, 3)) if wave is None else wave, timepoints=nb, boundary="periodic")


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("nb,npar", [(8, 1), (16, 33), (24, 2000), (4, 50), (12, 257), (15, 64)])
def test_store_forms_hold_the_same_bytes(nb, npar, split):
    """A buffer 4 bytes off a 16-byte boundary is written bin by bin."""
    import torch
    n = npar * nb * 3
    got = []
    for off in (0, 1):
        buf = torch.full((n + 8,), float("nan"), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        sim(nb, npar).run(seed=4, precision="split", traj_out=buf.data_ptr() + 4 * off, traj_split=split)
        raw = buf.view(torch.int32).cpu().numpy()
        got.append(raw[off:off + n])
        nan = np.float32("nan").view(np.int32)
        assert (np.delete(raw, np.s_[off:off + n]) == nan).all(), "written outside the buffer"
    np.testing.assert_array_equal(got[0], got[1])


@pytest.mark.parametrize("nw", [1, 3, 4, 5, 18])
def test_waveforms_four_at_a_time(nw):
    """Each waveform's sums from a run of all of them and of it alone: the same
    phases, sums over walkers in another order (FP64: 1e-12)."""
    nb, npar = 10, 500
    w = waveforms.scale_to_b(waveforms.random_smooth(nw, nb, 1.0, seed=2), 2e-3, np.linspace(0.2, 2.0, nw))
    both = sim(nb, npar, w).run(seed=4, precision="split").get("sigw").reshape(nw, 2)
    for j in range(nw):
        one = sim(nb, npar, w[j:j + 1]).run(seed=4, precision="split").get("sigw")
        np.testing.assert_allclose(both[j], one, rtol=0, atol=1e-12 * npar)
