"""Record totals of a launch over many axons: their memory is bounded over the
axons, and fewer row sets an axon add up to the same totals."""
import numpy as np
import pytest

from rms_b200 import engine, geometry

pytestmark = pytest.mark.gpu


def test_memory_of_many_axons():
    """40 axons with 20000 records and walkers for 16 row sets of 5 MB each: 3.3 GB
    of them without a bound over the axons; 1 GiB and the results (0.16 GB) with."""
    import torch
    n, T, npar = 40, 20_000, 33_000
    lab = geometry.axon_lattice(16, 16, 24, 0.1, seed=1, exterior=2, r0=0.5)
    kw = dict(dt=2e-4, tn=T, npar=npar, res=0.1, t2=[80.0, 80.0, 60.0], timepoints=T, bval=[], bvec=np.zeros((0, 3)))
    sims = [engine.Sim(lab, diffusivity=[0.0, 1.5 + 0.02 * k, 2.0], **kw) for k in range(n)]
    sims[0].run(seed=5, precision="split", walker_range=(0, 32))   # the context's own growth
    engine.trim_memory()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    engine.batch_run(sims, seed=5, precision="split")
    assert before - torch.cuda.mem_get_info()[0] < (1 << 30) + 8 * n * T * 25 + (128 << 20)
    for s in sims:
        np.testing.assert_array_equal(s.get("npar_count").reshape(T, 3).sum(1), npar)
    got = sims[0].outputs()
    want = sims[0].run(seed=5, precision="split").outputs()   # the batch's first member has the call's own seed
    np.testing.assert_array_equal(got["npar_count"], want["npar_count"])
    for k in ("sig0", "dx2", "dx4"):
        assert np.abs(got[k] - want[k]).max() <= 1e-11 * np.abs(want[k]).max(), k   # FP64 sums in another order
