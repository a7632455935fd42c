"""The tensor-core contraction's tiles: 64, 128 or 256 walkers per unit by how
many units the SMs get, and a last pair of waveform tiles with one or two of
them in use.  Both tensor-core methods against FP64 on the same FP32 inputs
(1e-4 of the walker count, the hi/lo split's bound in this suite), every
waveform and no other written."""
import threading

import numpy as np
import pytest

import pyoracle
from rms_b200 import engine

pytestmark = pytest.mark.gpu


def inputs(nwalk, nbins, nwave, seed):
    rng = np.random.default_rng(seed)
    pos = np.cumsum(rng.normal(scale=0.5, size=(nwalk, nbins, 3)), axis=1).astype(np.float32)
    wave = (rng.normal(size=(nwave, nbins, 3)) * (2.0 / nbins)).astype(np.float32)
    return pos, wave


def split(pos):
    """BF16 hi parts then lo parts, as the walk writes them."""
    import torch
    x = torch.from_numpy(pos).cuda()
    hi = x.bfloat16()
    lo = (x - hi.float()).bfloat16()
    return torch.cat([hi.reshape(-1), lo.reshape(-1)]).view(torch.float32)


def run(pos, wave, method):
    import torch
    nwave = wave.shape[0]
    d_pos = split(pos) if method == "bf16x3_presplit" else torch.from_numpy(pos).cuda()
    d_wave = torch.from_numpy(wave).cuda()
    out = torch.full((nwave + 4, 2), -7.0, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    engine.contract_phases(d_pos.data_ptr(), pos.shape[0], pos.shape[1], d_wave.data_ptr(), nwave, out.data_ptr(),
                           method=method)
    out = out.cpu().numpy()
    assert (out[nwave:] == -7.0).all()
    return out[:nwave]


# units per SM on 148: 64 walkers a unit up to ~9472 walkers a pair, then 128 and 256
@pytest.mark.parametrize("method", ["bf16x3", "bf16x3_presplit"])
@pytest.mark.parametrize("nwalk,nwave", [(1, 1), (63, 128), (65, 129), (4763, 120), (9473, 128), (12000, 40),
                                         (19000, 257), (30000, 384), (40001, 385), (3000, 1000)])
def test_tiles(nwalk, nwave, method):
    pos, wave = inputs(nwalk, 24, nwave, nwalk + nwave)
    got = run(pos, wave, method)
    want = pyoracle.contract_phases_fp64(pos, wave)
    assert np.abs(got - want).max() < 1e-4 * nwalk


def test_threads_have_their_own_workspaces():
    cases = [inputs(500 + 700 * k, 16, 20 + 60 * k, k) for k in range(4)]
    want = [run(p, w, "bf16x3") for p, w in cases]
    bad = []

    def work(k):
        import torch
        try:
            p, w = cases[k]
            st = torch.cuda.Stream()
            d_pos, d_wave = torch.from_numpy(p).cuda(), torch.from_numpy(w).cuda()
            out = torch.zeros((w.shape[0], 2), dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
            for _ in range(30):
                engine.contract_phases(d_pos.data_ptr(), p.shape[0], p.shape[1], d_wave.data_ptr(), w.shape[0],
                                       out.data_ptr(), method="bf16x3", stream=st.cuda_stream)
                assert np.abs(out.cpu().numpy() - want[k]).max() <= 1e-9 * p.shape[0]
        except BaseException as e:   # noqa: BLE001
            bad.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
