"""A refused launch is the refused call's error alone: the calls after it, on the
same runner, on a new one, and through the other entry points, do what they do
without it.  (The launch, an RDS baseband of a rate whose tile does not fit in
shared memory, returns its error on the host; nothing of it runs.)"""
import ctypes as C

import numpy as np
import pytest

import gpudemod as G
from gpudemod._lib import lib

pytestmark = pytest.mark.gpu

FS, BLOCK = 10_000_000, 1 << 16


def _refuse(r, x):
    slot = r.admit(1000, 0.0, 200_000.0, 2_000_000, 101, G.MODE_WFM_STEREO, G.CH_RDS)
    with pytest.raises(G.GPUDError):
        r.process_block(x)
    r.retire(slot)


def _admit_48k(r, x):
    # rates that this process has not asked for: their resampler banks are made now
    slots = [r.admit(k + 1, 0.0, 5_000.0, rate, 65, G.MODE_NFM, G.CH_AUDIO48K)
             for k, rate in enumerate((20_000, 31_250))]
    r.process_block(x)
    assert all(r.result(s)["pcm_rate"] == 48_000 for s in slots)


def _spectrum(r, x):
    s = G.Spectrum()
    try:
        s.welch(x[:20_000], 1024)
    finally:
        s.close()


def _pilot(r, x):
    d = G.StereoPilotDetector(1, 20_000)
    try:
        d.run([x[:20_000]], [200_000])
    finally:
        d.close()


def _rds(r, x):
    d = G.RDSDecoder(1, 20_000)
    try:
        d.decode(x[:20_000], 19_000)
    finally:
        d.close()


def _launcher(r, x):
    import torch
    d = torch.from_numpy(x).cuda()
    out = torch.empty(x.size, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    assert lib.gpud_launch_am_envelope_cuda(d.data_ptr(), out.data_ptr(), x.size) == 0
    assert lib.gpud_stream_sync(None) == 0


def _segment(r, x):
    G.demod_audio_segment(G.MODE_NFM, x, 1_000_000, 10_000.0, 12_000.0)


@pytest.mark.parametrize("after", [_admit_48k, _spectrum, _pilot, _rds, _launcher, _segment])
@pytest.mark.parametrize("same", [True, False])
def test_calls_after_a_refused_launch(cuda, after, same):
    rng = np.random.default_rng(2)
    x = (rng.standard_normal(BLOCK) + 1j * rng.standard_normal(BLOCK)).astype(np.complex64)
    bad = G.ChannelRunner(FS, BLOCK, max_channels=4)
    good = bad if same else G.ChannelRunner(FS, BLOCK, max_channels=4)
    try:
        _refuse(bad, x)
        after(good, x)
    finally:
        bad.close()
        good.close()
