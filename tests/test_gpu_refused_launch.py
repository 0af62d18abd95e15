"""A block whose launches are refused half way (an RDS baseband of a rate whose
tile does not fit in shared memory: the launch returns an error on the host and
nothing of it runs) leaves no work behind: when the call returns its error, the
GPU is done with the caller's block and the frame's buffers.  The device is idle
when it takes less than a quarter of a whole block's time to synchronise with;
the block is sized to several milliseconds of extraction."""
import time

import numpy as np
import pytest

import gpudemod as G

pytestmark = pytest.mark.gpu

FS, BLOCK = 10_000_000, 1 << 21


def _runner():
    r = G.ChannelRunner(FS, BLOCK, max_channels=256, max_taps=4096)
    rng = np.random.default_rng(3)
    for k in range(250):  # another filter length each: nothing is grouped
        r.admit(k + 1, float(rng.uniform(-4e6, 4e6)), 100_000.0, 200_000, 2_500 + 6 * k, G.MODE_NFM, 0)
    r.set_host_outputs(False)
    return r


def test_nothing_is_left_running(cuda):
    import torch
    x = torch.randn(BLOCK, dtype=torch.complex64).pin_memory()
    r = _runner()
    try:
        for _ in range(5):  # the first on each frame allocate its buffers
            t = time.perf_counter()
            r.process_block(x)
            block = time.perf_counter() - t
        # its pilot loop forks the frame's streams, then its RDS launch is refused
        slot = r.admit(1000, 0.0, 200_000.0, 2_000_000, 101, G.MODE_WFM_STEREO, G.CH_RDS)
        for _ in range(2):
            torch.cuda.synchronize()
            with pytest.raises(G.GPUDError):
                r.process_block(x)
            t = time.perf_counter()
            torch.cuda.synchronize()
            left = time.perf_counter() - t
            assert left <= block / 4, (left, block)
        r.retire(slot)
        r.process_block(x)  # the runner goes on without the channel
    finally:
        r.close()
