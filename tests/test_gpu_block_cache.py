"""Device and pinned memory of closed simulations is kept for the next ones:
results do not depend on what a block held before, in one thread or several,
and what is kept is bounded."""
import threading

import numpy as np
import pytest

from rms_b200 import engine, geometry, waveforms

pytestmark = pytest.mark.gpu


def walk(k, precision):
    """A simulation of size k, made, run and closed."""
    side = 12 + 4 * (k % 5)
    lab = geometry.axon_lattice(side, side, 2 * side, 0.1, seed=k % 5, exterior=2, r0=0.5)
    kw = dict(dt=2e-4, tn=40, npar=300 + 400 * (k % 7), res=0.1, diffusivity=[0, 2.0, 1.5], t2=[80, 80, 60],
              timepoints=20 + 5 * (k % 3))
    if k % 3 == 0:
        kw.update(bval=np.linspace(1, 2, 1 + k % 40), bvec=np.tile([0.6, 0.0, 0.8], (1 + k % 40, 1)))
    elif k % 3 == 1:
        kw.update(grad=[[0.004, 0.002, 20.0, 1, 0, 0]])
    elif precision == "split":
        w = waveforms.random_smooth(1 + k % 6, 8, 1.0, seed=k)
        kw.update(wave=w)
    with engine.Sim(lab, **kw) as sim:
        return sim.run(seed=k, precision=precision).outputs()


def same(a, b):
    assert np.array_equal(a["npar_count"], b["npar_count"])
    for key in a:
        scale = np.abs(a[key]).max() if a[key].size else 0.0
        assert np.abs(a[key] - b[key]).max(initial=0.0) <= 1e-11 * scale, key


def test_results_do_not_depend_on_the_blocks():
    first = {(k, p): walk(k, p) for k in range(12) for p in ("split", "compat")}
    for k, p in list(first)[::-1]:
        same(first[k, p], walk(k, p))


def test_threads_share_the_cache():
    want = {k: walk(k, "split") for k in range(12)}
    bad = []

    def work(t):
        try:
            for r in range(3):
                for k in range(12):
                    same(want[(k + t) % 12], walk((k + t) % 12, "split"))
        except BaseException as e:   # noqa: BLE001
            bad.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


def test_what_is_kept_is_bounded():
    import torch
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for k in range(6):   # 1.1 GB of labels and 0.5 GB packed each, of another size every time
        n3 = 4200 + 300 * k
        with engine.Sim(dt=2e-4, tn=10, npar=64, res=0.1, diffusivity=[0, 2.0, 1.5], t2=[80, 80, 60],
                        shape=(512, 512, n3), timepoints=10, bval=[], bvec=np.zeros((0, 3))) as sim:
            sim.set_tube_lattice(*geometry.axon_slices(512, 512, n3), inside=1, outside=2)
            sim.run(seed=1, precision="split")
    torch.cuda.synchronize()
    # 4 GiB of blocks at most (and the context's own growth)
    assert free0 - torch.cuda.mem_get_info()[0] < (4 << 30) + (1 << 30)
