"""Simulations are independent objects: one that grows its buffers, or is closed,
in one thread does not disturb a capture another thread has begun."""
import threading

import numpy as np
import pytest

from rms_b200 import engine, geometry

pytestmark = pytest.mark.gpu


def sim(npar, T):
    lab = geometry.axon_lattice(12, 12, 16, 0.1, seed=2, exterior=2, r0=0.4)
    return engine.Sim(lab, dt=2e-4, tn=40, npar=npar, res=0.1, diffusivity=[0, 2.0, 1.5], t2=[80, 80, 60],
                      timepoints=T, bval=[1.0], bvec=[[1.0, 0, 0]])


def test_closing_and_growing_leave_another_threads_capture_alone():
    import torch
    want = sim(64, 40).run(seed=1, precision="split").outputs()
    closed, grown = sim(64, 40), sim(40_000, 40)
    closed.run(seed=1, precision="split")
    grown.run(seed=1, precision="split", walker_range=(0, 32))
    x = torch.ones(1 << 20, device="cuda")
    y = torch.zeros_like(x)
    bad, got = [], []

    def other():
        try:
            closed.close()
            grown.run(seed=1, precision="compat")   # per-warp rows: buffers the small run did not have
            grown.close()
            with sim(64, 40) as s:                  # on the memory of the others
                got.append(s.run(seed=1, precision="split").outputs())
        except BaseException as e:   # noqa: BLE001
            bad.append(e)

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        torch.add(x, x, out=y)
        t = threading.Thread(target=other)
        t.start()
        t.join()
        torch.add(y, x, out=y)
    assert not bad, bad
    g.replay()
    torch.cuda.synchronize()
    assert bool((y == 3.0).all())
    np.testing.assert_array_equal(got[0]["npar_count"], want["npar_count"])
    for k in want:
        scale = np.abs(want[k]).max(initial=0.0)
        assert np.abs(got[0][k] - want[k]).max(initial=0.0) <= 1e-11 * scale, k
