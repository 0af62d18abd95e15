"""Every ratio of the 48 kHz resampler finds its tile at once: an even one (240
kS/s: 1 to 5) takes no longer than twice an uneven one of the same size (250 kS/s:
24 to 125), where the arithmetic is the same.  Device times from a profile, the
shortest of 30 launches each."""
import pytest

import gpudemod as G

pytestmark = pytest.mark.gpu


def _us(rate):
    import torch
    from torch.profiler import ProfilerActivity, profile
    decim = 8
    n = rate * decim // 33  # 30 ms
    r = G.ChannelRunner(rate * decim, n, max_channels=4, max_taps=128)
    try:
        for k in range(4):
            r.admit(k + 1, 0.0, 0.4 * rate, rate, 65, G.MODE_NFM, G.CH_AUDIO48K)
        x = torch.randn(n, dtype=torch.complex64, device="cuda")
        torch.cuda.synchronize()
        for _ in range(4):
            r.process_block(x)
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            for _ in range(30):
                r.process_block(x)
            torch.cuda.synchronize()
    finally:
        r.close()
    times = [e.device_time for e in p.events() if "k_audio48_rs" in e.name]
    assert len(times) >= 5  # a profile may miss launches at its start
    return min(times)


@pytest.mark.parametrize("even,uneven", [(240_000, 250_000), (96_000, 97_500), (288_000, 292_500)])
def test_even_ratios_take_no_longer(cuda, even, uneven):
    a, b = _us(even), _us(uneven)
    assert a <= 2.0 * b, (a, b)
