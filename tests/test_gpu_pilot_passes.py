"""The pilot detector's batched bins at the edges of their layout: one station,
a full station group, a full pass of 40 and one more, several rates in one call
(one pass each), windows shorter than a period and than one staged chunk per
CTA.  Decisions and best bins equal the float64 oracle's; ratio and median
within 1e-6, as the detector's existing test has it (the oracle's Goertzel
recurrence itself loses digits in proportion to the window)."""
import numpy as np
import pytest

import gpudemod as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _iq(fs, n, pilot, seed):
    rng = np.random.default_rng(seed)
    t = np.arange(n) / fs
    ph = np.cumsum(2 * np.pi * 75000 / fs * (0.4 * np.sin(2 * np.pi * 900 * t) + pilot * np.sin(2 * np.pi * 19000 * t)))
    return (np.exp(1j * ph) + 0.1 * (rng.standard_normal(n) + 1j * rng.standard_normal(n))).astype(np.complex64)


@pytest.mark.parametrize("count", [1, 8, 9, 40, 41])
def test_station_counts(cuda, count):
    fs, n = 200_000, 21_000
    xs = [_iq(fs, n, 0.1 if k % 3 else 0.0, 50 + k) for k in range(count)]
    _check(xs, [fs] * count)


@pytest.mark.parametrize("n", [2, 3, 17, 500, 5_000, 40_001])
def test_window_lengths(cuda, n):
    _check([_iq(192_000, n, 0.1, n)], [192_000])


def test_mixed_rates(cuda):
    rates = [200_000, 312_501, 200_000, 250_003, 312_501, 48_000, 200_000]
    xs = [_iq(fs, 9_000 + 100 * k, 0.08 * (k % 2), 90 + k) for k, fs in enumerate(rates)]
    _check(xs, rates)


def _check(xs, rates):
    det = G.StereoPilotDetector(max_jobs=len(xs), max_samples=max(x.size for x in xs))
    try:
        got = det.run(xs, rates)
    finally:
        det.close()
    for x, fs, g in zip(xs, rates, got):
        lk, ratio, best, med, _ = O.stereo_pilot(x, fs, window=True)
        assert g["present"] == lk
        if x.size < 1000:
            continue  # a handful of samples: every bin is the same sum up to its last bits
        assert g["best_hz"] == best
        assert abs(g["ratio"] - ratio) <= 1e-6 * max(1.0, ratio)
        assert abs(g["median"] - med) <= 1e-6 * med
