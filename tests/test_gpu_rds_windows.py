"""The RDS decoder's rounds at the edges of their windows (2048 samples, 256
symbols): lengths around one and two windows, a rate with more than one symbol
in every two samples (several rounds per window), many stations in one call,
and state carried from call to call.  Every call's groups, PI, PS and RT equal
the oracle's decoder exactly (both run the same float operations)."""
import numpy as np
import pytest

import gpudemod as G
from gpudemod import synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _baseband(fs, n, seed, snr_db=20.0):
    rng = np.random.default_rng(seed)
    pi, ps, rt = synth.random_station_text(rng)
    sym = synth.rds_symbols(synth.rds_bits(synth.rds_groups(pi, ps, rt), int(n * 1187.5 / fs) + 8))
    pos = np.arange(n) / fs * 1187.5 + rng.uniform(0, 1)
    k = pos.astype(np.int64)
    c = 0.5 * (1 + np.cos(np.pi * (pos - k)))
    z = (sym[k] * c + sym[k + 1] * (1 - c)) * np.exp(1j * rng.uniform(0, 2 * np.pi))
    noise = 10 ** (-snr_db / 20) * (rng.standard_normal(n) + 1j * rng.standard_normal(n))
    return (0.05 * (z + noise)).astype(np.complex64)


@pytest.mark.parametrize("fs,lengths", [
    (19_531, [2047, 2048, 2049, 2050, 4096, 4097, 30_001]),
    (2_375, [600, 2048, 5_000]),      # two samples a symbol: four rounds per window
    (19_000, [104, 1_700, 103, 40_000]),
])
def test_windows_and_rounds(cuda, fs, lengths):
    stations = 5
    dec = G.RDSDecoder(stations, max(lengths))
    refs = [O.RDSDecoder() for _ in range(stations)]
    try:
        for call, n in enumerate(lengths):
            xs = [_baseband(fs, n, 100 * call + st, 8.0 + 6.0 * st) for st in range(stations)]
            got = dec.run([(x, fs, st) for st, x in enumerate(xs)])
            for x, ref, g in zip(xs, refs, got):
                groups = ref.decode(x, fs)
                assert g["status"] == 0
                assert (g["groups"], g["pi"], g["ps"], g["rt"]) == (groups, *ref.result()), (call, n)
    finally:
        dec.close()
