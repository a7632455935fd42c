"""Memory kept of closed simulations goes back: when requests pass it over, and
when a program asks."""
import numpy as np
import pytest

from rms_b200 import engine, geometry

pytestmark = pytest.mark.gpu
SIDE, LENGTH = 512, 2000          # 0.52 GB of labels and as much packed


def large():
    s = engine.Sim(dt=2e-4, tn=10, npar=64, res=0.1, diffusivity=[0, 2.0, 1.5], t2=[80, 80, 60],
                   shape=(SIDE, SIDE, LENGTH), timepoints=10, bval=[], bvec=np.zeros((0, 3)))
    s.set_tube_lattice(*geometry.axon_slices(SIDE, SIDE, LENGTH), inside=1, outside=2)
    return s.run(seed=1, precision="split")


def small(seed):
    lab = geometry.axon_lattice(8, 8, 8, 0.1, seed=1, exterior=2, r0=0.3)
    s = engine.Sim(lab, dt=2e-4, tn=10, npar=64, res=0.1, diffusivity=[0, 2.0, 1.5], t2=[80, 80, 60], timepoints=10,
                   bval=[], bvec=np.zeros((0, 3)))
    return s.run(seed=seed, precision="split")


def free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_blocks_passed_over_are_freed():
    """Simulations that are made and kept, none closed, ask for some 15 blocks each."""
    small(0)
    large().close()
    before = free()
    kept = [small(k) for k in range(30)]
    assert free() - before > SIDE * SIDE * LENGTH
    for s in kept:
        s.close()


def test_trim_gives_everything_back():
    engine.trim_memory()
    want = small(3).outputs()
    before = free()
    large().close()
    assert before - free() > SIDE * SIDE * LENGTH
    device, pinned = engine.trim_memory()
    assert device > SIDE * SIDE * LENGTH and pinned > 0
    assert before - free() < 64 << 20
    got = small(3).outputs()
    np.testing.assert_array_equal(got["npar_count"], want["npar_count"])


def test_contractions_leave_their_workspace_to_the_cache():
    import torch
    g = torch.Generator(device="cuda").manual_seed(0)
    pos = torch.randn((1000, 64, 3), generator=g, device="cuda")
    wave = 0.01 * torch.randn((300, 64, 3), generator=g, device="cuda")
    outs = []
    for trim in (False, True, False):
        if trim:
            assert engine.trim_memory()[0] >= 300 * 64 * 3 * 4
            assert engine.trim_memory() == (0, 0)
        out = torch.empty((300, 2), dtype=torch.float64, device="cuda")
        engine.contract_phases(pos.data_ptr(), 1000, 64, wave.data_ptr(), 300, out.data_ptr(),
                               stream=torch.cuda.current_stream().cuda_stream)
        outs.append(out.cpu().numpy())
    phase = pos.double().flatten(1) @ wave.double().flatten(1).T
    want = torch.stack([phase.cos().sum(0), phase.sin().sum(0)], 1).cpu().numpy()
    for out in outs:
        assert np.abs(out - want).max() <= 1e-4 * 1000


def test_reverse_pass_on_blocks_that_held_other_records():
    """Gradients on fresh memory and on blocks other walks have filled: the same
    walkers, FP32 sums by atomics in another order."""
    import torch
    from rms_b200 import adjoint, waveforms
    lab = geometry.axon_lattice(16, 16, 32, 0.1, seed=3, exterior=2, r0=0.5)

    def grads(seed, npar, bins, waves):
        setup = adjoint.WalkSetup(lab, dt=2e-4, tn=10 * bins, npar=npar, res=0.1, seed=seed, boundary="periodic")
        w = torch.tensor(0.5 * waveforms.random_smooth(waves, bins, 1.0, seed=seed), dtype=torch.float64,
                         requires_grad=True)
        leaves = [torch.tensor(x, dtype=torch.float64, requires_grad=True) for x in (2.0, 0.05, [80.0, 80.0, 60.0])]
        adjoint.waveform_signal(w, *leaves, setup).sum().backward()
        return [w.grad.numpy()] + [x.grad.numpy() for x in leaves]

    engine.trim_memory()
    want = grads(1, 3000, 40, 5)
    engine.trim_memory()
    for k, (npar, bins, waves) in enumerate([(4000, 30, 16), (2500, 60, 3), (3100, 40, 5)]):
        grads(k + 2, npar, bins, waves)
    for a, b in zip(grads(1, 3000, 40, 5), want):
        # 3000 walkers' FP32 terms, each rounded to 2^-24, some 100 partial sums of them
        assert np.abs(a - b).max() <= 1e-5 * np.abs(b).max()
