"""Short windows of the pilot detector, whose few terms take a kernel of their own:
a station's decision is the same bits in a call of its own, among others of its
rate (which together take the other kernel) and among several rates; and a call of
three rates costs less than three calls."""
import numpy as np
import pytest

import gpudemod as G

pytestmark = pytest.mark.gpu


def _iq(fs, n, seed):
    rng = np.random.default_rng([fs, n, seed])
    t = np.arange(n) / fs
    m = 0.3 * np.sin(2 * np.pi * 400 * t) + 0.1 * np.sin(2 * np.pi * 19_000 * t)
    z = np.exp(1j * 2 * np.pi * 75_000 * np.cumsum(m) / fs)
    return (z + 0.1 * (rng.standard_normal(n) + 1j * rng.standard_normal(n))).astype(np.complex64)


# one term; fewer than a share; one and more shares per CTA; the rule's limit of
# 8192 terms and one more; windows of more than a period (40 kS/s: 4000 samples)
@pytest.mark.parametrize("fs,n", [(200_000, 2), (312_500, 31), (312_500, 558), (250_007, 2_000), (312_500, 8_193),
                                  (312_500, 8_194), (40_000, 4_001), (40_000, 9_001)])
def test_alone_and_among_others(cuda, fs, n):
    iq = [_iq(fs, n, k) for k in range(40)]
    other = [(rate, _iq(rate, 700, 1)) for rate in (48_000, 256_000)]
    det = G.StereoPilotDetector(64, max(n, 700))
    try:
        alone = [det.run([x], [fs])[0] for x in iq]
        assert det.run(iq, [fs] * 40) == alone
        mixed = det.run([other[0][1], iq[3], other[1][1], iq[7]], [other[0][0], fs, other[1][0], fs])
        assert [mixed[1], mixed[3]] == [alone[3], alone[7]]
    finally:
        det.close()


def test_several_rates_in_one_launch(cuda):
    """Device times from a profile, the least of 20 calls: the kernels of three
    short stations of three rates take less than twice those of one."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    jobs = [(torch.from_numpy(_iq(fs, 1_000, 0)).cuda(), fs) for fs in (200_000, 256_000, 312_500)]
    det = G.StereoPilotDetector(4, 1_000)

    def us(some):
        xs, rates = zip(*some)
        torch.cuda.synchronize()
        for _ in range(3):
            det.run(list(xs), list(rates))
        best = []
        for _ in range(20):
            with profile(activities=[ProfilerActivity.CUDA]) as p:
                det.run(list(xs), list(rates))
                torch.cuda.synchronize()
            best.append(sum(e.device_time for e in p.events() if "k_pilot" in e.name))
        return min(best)

    try:
        one, three = us(jobs[:1]), us(jobs)
    finally:
        det.close()
    assert 0 < three <= 2.0 * one, (one, three)
