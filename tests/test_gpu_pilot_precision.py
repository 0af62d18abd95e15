"""The pilot detector's float64 sums against 80-bit ones: ratio and median of a
station may be no further off than with the detector's plain order of sums (one
CTA's 256 threads, each a run of the folded samples, then a tree), here in
float64 on the CPU from the same 80-bit discriminator rounded once.  Both errors
are roundings that add up at random; over 36 stations their rms scatters by a
tenth, so a quarter more is allowed.  Windows shorter than a period (every
sample a term) and longer (folded in pairs), calls of few stations and of many."""
import math

import numpy as np
import pytest

import gpudemod as G

pytestmark = pytest.mark.gpu

LD = np.longdouble
STATIONS = 36


def _iq(fs, n, seed):
    rng = np.random.default_rng([fs, n, seed])
    t = np.arange(n) / fs
    m = (0.4 * np.sin(2 * np.pi * rng.uniform(300, 3000) * t) + 0.3 * np.sin(2 * np.pi * 400 * t)
         + 0.09 * np.sin(2 * np.pi * 19_000 * t + rng.uniform(0, 6)))
    z = np.exp(1j * 2 * np.pi * 75_000 * np.cumsum(m) / fs)
    noise = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    return (z + 10 ** (-rng.uniform(5, 35) / 20) * noise).astype(np.complex64)


def _ratio_median(mags):
    m = np.sort(mags)
    return m[-1] / m[100], m[100]


def _truth_and_plain(iq, fs):
    """(ratio, median) in 80 bits and in float64 with the plain order of sums."""
    x, y = iq.real.astype(LD), iq.imag.astype(LD)
    d = np.arctan2(x[:-1] * y[1:] - y[:-1] * x[1:], x[:-1] * x[1:] + y[:-1] * y[1:])
    P = fs // math.gcd(fs, 10)
    step = 10 // math.gcd(fs, 10)
    F = min(P, d.size)
    fold, fold64 = np.zeros(F, LD), np.zeros(F)
    for k in range(0, d.size, P):
        seg = d[k:k + P]
        fold[:seg.size] += seg
        fold64[:seg.size] += seg.astype(np.float64)
    a = np.arange(P).astype(LD) * (2 * LD("3.14159265358979323846264338327950288") / P)
    c, s = np.cos(a), np.sin(a)
    c64, s64 = c.astype(np.float64), s.astype(np.float64)
    per = -(-F // 256)
    pad = np.zeros(256 * per)
    pad[:F] = fold64
    m = np.arange(256 * per).reshape(256, per)
    mags, plain = [], []
    for b in range(201):
        w = ((1800 + b) * step * m[:, :]) % P
        i = ((1800 + b) * step * np.arange(F)) % P
        mags.append(np.hypot((fold * c[i]).sum(), (fold * s[i]).sum()))
        parts = []
        for tab in (c64, s64):
            run = np.cumsum(pad.reshape(256, per) * tab[w], axis=1)[:, -1]  # each thread's run, in order
            while run.size > 8:  # its warp's tree, then the warps in order
                run = run.reshape(-1, 2).sum(1)
            parts.append(float(np.cumsum(run)[-1]))
        plain.append(math.hypot(*parts))
    return _ratio_median(np.array(mags, LD)), _ratio_median(np.array(plain))


@pytest.mark.parametrize("fs,n", [(320_000, 30_000), (312_500, 156_250)])
def test_no_further_off_than_plain_sums(cuda, fs, n):
    iq = [_iq(fs, n, k) for k in range(STATIONS)]
    truth, plain = zip(*(_truth_and_plain(x, fs) for x in iq))
    det = G.StereoPilotDetector(STATIONS, n)
    try:
        many = det.run(iq, [fs] * STATIONS)
        few = [r for k in range(0, STATIONS, 12) for r in det.run(iq[k:k + 12], [fs] * 12)]
    finally:
        det.close()

    def rms(got):
        return math.sqrt(np.mean([float((LD(g) - t) / t) ** 2 for p, q in zip(got, truth) for g, t in zip(p, q)]))

    allowed = 1.25 * rms(plain)
    for got in (many, few):
        assert rms([(r["ratio"], r["median"]) for r in got]) <= allowed, (allowed,)
