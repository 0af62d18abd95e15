"""Short windows of the pilot detector, whose few terms take a kernel of their own:
a station's decision is the same bits in a call of its own, among others of its
rate (which together take the other kernel) and among several rates; and a call of
three rates takes no more launches than a call of one."""
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
    """A call of three rates launches what a call of one does: fold, bins, decision."""
    jobs = [(_iq(fs, 1_000, 0), fs) for fs in (200_000, 256_000, 312_500)]
    det = G.StereoPilotDetector(4, 1_000)
    try:
        for some in (jobs[:1], jobs):
            xs, rates = zip(*some)
            det.run(list(xs), list(rates))  # the table of a rate is made once
            before = G.kernel_launch_count()
            det.run(list(xs), list(rates))
            assert G.kernel_launch_count() - before == 3
    finally:
        det.close()
