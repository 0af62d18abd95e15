"""RDS windows too short to decode (fewer than 104 symbols) run the timing loop
only: no more than half of the time of a window of twice the length, whose 187
symbols also go through the Costas loop, the longer of the two chains.  Device
times from a profile, the shortest of 20 launches."""
import pytest

import gpudemod as G

pytestmark = pytest.mark.gpu


def _us(n):
    import torch
    from torch.profiler import ProfilerActivity, profile
    d = G.RDSDecoder(1, n)
    try:
        jobs = [(torch.randn(n, dtype=torch.complex64, device="cuda"), 19_000, 0)]
        torch.cuda.synchronize()
        for _ in range(3):
            d.run(jobs)
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            for _ in range(20):
                d.run(jobs)
            torch.cuda.synchronize()
    finally:
        d.close()
    times = [e.device_time for e in p.events() if "k_rds_decode" in e.name]
    assert len(times) >= 5  # a profile may miss launches at its start
    return min(times)


def test_short_windows_run_no_costas_loop(cuda):
    short, long = _us(1_500), _us(3_000)
    assert short <= 0.5 * long, (short, long)
