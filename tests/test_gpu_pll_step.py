"""The pilot PLL's step and its arctangent against float64.

The step: on the same pilot samples a loop of it may be no further from the loop
in float64 than the plain form in the same types, which rounds the angle of every
step from the float64 phase and calls atan2f -- on a locked station, a station
acquired from a frequency error, and a band of noise, at each output rate.  The
two differ in where they round only, so their errors (over time, of the median
loop, which a slipped cycle does not move) are equal up to the scatter of 64
loops: 5 %.

The arctangent: 2 ulp, the bound of atan2f, at all quadrants, quotients and
magnitudes of the lowpass states, and the values it takes on the axes."""
import ctypes as C
import math
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "argus-sdr_b200")
N, LOOPS = 30_000, 64
D, P, I = C.c_double, C.c_void_p, C.c_int


@pytest.fixture(scope="module")
def check(cuda):
    lib = C.CDLL(os.path.join(PKG, "libgpudemod_check.so"))
    lib.gpud_check_pll_loop.argtypes = [P, I, I, D, D, D, D, D, D, I, P]
    lib.gpud_check_pll_atan2.argtypes = [P, P, I, I, P]
    return lib


def _pilots(kind, rate, rng):
    """Pilot band samples: a tone near 19 kHz and band-limited noise, 0.3 and +-pi before its band."""
    t = np.arange(N)
    k = np.arange(101) - 50
    band = 2 * 500 / rate * np.sinc(2 * 500 / rate * k) * np.hanning(101) * 2 * np.cos(2 * np.pi * 19_000 / rate * k)
    x = np.empty((LOOPS, N), np.float32)
    for c in range(LOOPS):
        noise = np.convolve(rng.uniform(-math.pi, math.pi, N + 100), band, "valid")
        if kind == "locked":
            f, phase, amp, level = 19_000 + rng.uniform(-2, 2), rng.uniform(-0.01, 0.01), 0.3, 0.02
        elif kind == "acquired":
            f, phase, amp, level = 19_000 + rng.uniform(-40, 40), rng.uniform(0, 2 * math.pi), 0.3, 0.1
        else:
            f, phase, amp, level = 19_000, 0.0, 0.0, 1.0
        x[c] = amp * np.cos(2 * math.pi * f / rate * t + phase) + level * noise
    return x


def _float64(x, alpha, beta, lpa, fmin, fmax, freq):
    loops = x.shape[0]
    dphi, df, li, lq = (np.zeros(loops) for _ in range(4))
    out = np.empty(x.shape)
    lpa = float(np.float32(lpa))
    for t in range(x.shape[1]):
        a = math.remainder(t * freq, 2 * math.pi) + dphi
        p = x[:, t].astype(np.float64)
        li += lpa * (p * np.cos(a) - li)
        lq += lpa * (-p * np.sin(a) - lq)
        e = np.arctan2(lq, li)
        df = np.clip(df + beta * e, fmin - freq, fmax - freq)
        dphi = dphi + df + alpha * e
        out[:, t] = dphi
    return out


@pytest.mark.parametrize("rate", [200_000, 300_000, 312_500])
@pytest.mark.parametrize("kind", ["locked", "acquired", "noise"])
def test_step_is_as_exact_as_the_plain_form(check, kind, rate):
    import torch
    x = _pilots(kind, rate, np.random.default_rng([rate, len(kind)]))
    wn = 2 * math.pi * 50 / rate
    par = (2 * 0.707 * wn, wn * wn, 1 - math.exp(-2 * math.pi * 200 / rate), 2 * math.pi * 17_000 / rate,
           2 * math.pi * 21_000 / rate, 2 * math.pi * 19_000 / rate)
    want = _float64(x, *par)
    d_x = torch.from_numpy(x).cuda()
    rms = []
    for plain in (0, 1):
        got = torch.zeros(LOOPS, N, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert check.gpud_check_pll_loop(d_x.data_ptr(), N, LOOPS, *par, plain, got.data_ptr()) == 0
        err = got.cpu().numpy() - want
        err -= 2 * math.pi * np.round(err / (2 * math.pi))
        rms.append(float(np.sqrt(np.mean(np.median(err * err, axis=0)))))
    assert rms[0] <= 1.05 * rms[1], rms


def test_atan2(check):
    import torch
    rng = np.random.default_rng(5)
    n = 4_000_000
    mag, ang = np.exp(rng.uniform(-60, 3, n)), rng.uniform(-math.pi, math.pi, n)
    y, x = (mag * np.sin(ang)).astype(np.float32), (mag * np.cos(ang)).astype(np.float32)
    y[: n // 4] = (x[: n // 4] * np.exp(rng.uniform(-12, 12, n // 4))).astype(np.float32)  # quotients far from one
    axes = [(0, 0), (0, 1), (0, -1), (1, 0), (-1, 0), (1, 1), (-1, 1), (1, -1), (-1, -1), (-0.0, 1), (-0.0, -1),
            (1e-30, 1e-30), (0, 1e-38), (1e-38, 0), (3e-39, -3e-39)]
    y[-len(axes):], x[-len(axes):] = np.array(axes, np.float32).T
    d_y, d_x = torch.from_numpy(y).cuda(), torch.from_numpy(x).cuda()
    got = torch.zeros(n, device="cuda")
    torch.cuda.synchronize()
    assert check.gpud_check_pll_atan2(d_y.data_ptr(), d_x.data_ptr(), n, 0, got.data_ptr()) == 0
    want = np.arctan2(y.astype(np.float64), x.astype(np.float64))
    ulp = np.spacing(np.abs(want).astype(np.float32)).astype(np.float64)
    err = np.abs(got.cpu().numpy().astype(np.float64) - want) / ulp
    assert err.max() <= 2.0, (err.max(), y[err.argmax()], x[err.argmax()])
