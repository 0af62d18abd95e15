"""Tiles of the 48 kHz resampler: ratios with four outputs per thread (L from 1
to 124, last tile and last block of 4L ragged), with one, and with arms or a
window that stay in global memory.  The PCM of a channel that resamples against
the oracle's back end over the same channel's demodulator-rate audio, which a
second channel gives: the same float32 inputs through the same float64 sums in
the same order, so the s16le samples are equal."""
import numpy as np
import pytest

import gpudemod as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rate,decim,mode", [
    (24_000, 50, "NFM"),     # L 2, M 1
    (25_000, 40, "NFM"),     # L 48, M 25
    (12_500, 64, "USB"),     # L 96, M 25
    (5_000, 80, "CW"),       # L 48, M 5
    (96_000, 10, "AM"),      # L 1, M 2
    (16_000, 25, "NFM"),     # L 3, M 1
    (150_000, 16, "NFM"),    # L 8, M 25: four outputs, a window of 3.1 inputs per output
    (250_000, 8, "WFM"),     # L 24, M 125: one output per thread
    (312_500, 8, "WFM"),     # L 96, M 625
    (44_100, 40, "NFM"),     # L 160: arms in global memory
    (600_000, 4, "WFM"),     # L 2, M 25: window in global memory
])
def test_resampler_tiles_match_oracle(cuda, rate, decim, mode):
    fs = rate * decim
    m = {"NFM": G.MODE_NFM, "AM": G.MODE_AM, "USB": G.MODE_USB, "CW": G.MODE_CW, "WFM": G.MODE_WFM_STEREO}[mode]
    ch, bw = (2, 180_000.0) if mode == "WFM" else (1, 0.4 * rate)
    rng = np.random.default_rng(rate)
    lens = [int(decim * rate * t) + e for t, e in ((0.03, 0), (0.0213, 7), (0.001, 1), (0.025, decim // 2))]
    n = max(lens)
    t = np.arange(sum(lens)) / fs
    x = (np.exp(2j * np.pi * (0.05 * rate * t + 2.0 * np.sin(2 * np.pi * 700.0 * t)))
         + 0.05 * (rng.standard_normal(t.size) + 1j * rng.standard_normal(t.size))).astype(np.complex64)
    r = G.ChannelRunner(fs, n, max_channels=4, max_taps=256)
    back = O.Audio48(rate, ch, wfm=mode == "WFM", deemph_us=50.0)
    try:
        a = r.admit(1, 0.0, bw, rate, 65, m, 0)
        b = r.admit(2, 0.0, bw, rate, 65, m, G.CH_AUDIO48K)
        at = 0
        for k, c in enumerate(lens):
            r.process_block(x[at:at + c])
            at += c
            _, want = back.process(r.result(a)["audio"])
            got = r.result(b)["pcm"]
            assert got.size == want.size, k
            assert np.array_equal(np.asarray(got).reshape(-1), np.asarray(want).reshape(-1)), (
                k, int(np.abs(got.astype(int).reshape(-1) - want.astype(int).reshape(-1)).max()))
    finally:
        r.close()
