"""The spectrum's transform at every way its stages group (three, two or one at
a time) and at the smallest sizes, against numpy's float64 FFT.  Tolerance: a
float64 FFT of n points is within log2(n) * 2^-52 of the largest bin, 1e-9 dB
for bins at most 120 dB below it (the noise here is 40 dB below)."""
import numpy as np
import pytest

import gpudemod as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 4, 8, 16, 32, 64, 128, 256, 512, 1024, 2048, 4096, 8192])
def test_sizes_against_numpy(cuda, n):
    rng = np.random.default_rng(n)
    x = (np.exp(0.37j * np.arange(n)) + 0.01 * (rng.standard_normal(n) + 1j * rng.standard_normal(n))).astype(np.complex64)
    sp = G.Spectrum(8192, 4)
    try:
        got = sp.single(x, hann=False)
        want = 20 * np.log10(np.abs(np.fft.fftshift(np.fft.fft(x.astype(np.complex128)))) / n + 1e-12)
        assert np.max(np.abs(got - want)) <= 1e-9
    finally:
        sp.close()
