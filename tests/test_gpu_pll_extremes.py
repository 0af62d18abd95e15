"""The pilot loop where its numbers are extreme: an arctangent over all of
float32's magnitudes; composites at rates whose filters are designed beyond
Nyquist; a block with a non-finite sample in it.  The parallel solver stays with
the serial loop, which iterates the same step, and a loop that is not a number
(the recurrence's own end after such a sample) does not cost sweeps from then on."""
import ctypes as C
import os

import numpy as np
import pytest

import gpudemod as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "argus-sdr_b200")


def test_atan2_over_all_magnitudes(cuda):
    """2 ulp, as the step's own range (test_gpu_pll_step.py)."""
    import torch
    lib = C.CDLL(os.path.join(PKG, "libgpudemod_check.so"))
    lib.gpud_check_pll_atan2.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_void_p]
    rng = np.random.default_rng(8)
    n = 2_000_000
    mag, ang = np.exp(rng.uniform(np.log(1e-30), np.log(3e38), n)), rng.uniform(-np.pi, np.pi, n)
    y, x = (mag * np.sin(ang)).astype(np.float32), (mag * np.cos(ang)).astype(np.float32)
    d_y, d_x = torch.from_numpy(y).cuda(), torch.from_numpy(x).cuda()
    got = torch.zeros(n, device="cuda")
    torch.cuda.synchronize()
    assert lib.gpud_check_pll_atan2(d_y.data_ptr(), d_x.data_ptr(), n, 0, got.data_ptr()) == 0
    want = np.arctan2(y.astype(np.float64), x.astype(np.float64))
    ulp = np.spacing(np.abs(want).astype(np.float32)).astype(np.float64)
    err = np.abs(got.cpu().numpy().astype(np.float64) - want) / ulp
    assert err.max() <= 2.0, (err.max(), y[err.argmax()], x[err.argmax()])


def _pair(fs, block, rate, taps, decim):
    runners = [G.ChannelRunner(fs, block, max_channels=8, max_taps=1024) for _ in range(2)]
    runners[1].set_pll_solver(False)
    offs = (44_452.0, -310_000.0, 700_000.0)
    slots = [[r.admit(k + 1, o, 0.25 * rate, rate, taps, G.MODE_WFM_STEREO, 0, demod_decim=decim)
              for k, o in enumerate(offs)] for r in runners]
    return runners, slots


@pytest.mark.parametrize("rate,decim,steps", [
    (40_000, 2, 60), (40_000, 2, 3_000), (30_000, 1, 400), (40_000, 1, 40_000), (16_000, 1, 900), (48_000, 3, 5_000),
])
def test_filters_beyond_nyquist(cuda, rate, decim, steps):
    """Both solvers: finite, the same lock and stereo state, and the same floats
    (float32 values of order one: 1e-5; the frequency to its float32 ulp)."""
    fs = 3_840_000
    block = steps * decim * (fs // rate)
    (par, ser), (a, b) = _pair(fs, block, rate, 1000, decim)
    rng = np.random.default_rng(steps)
    try:
        for k in range(5):
            n = block - 77 * k
            t = np.arange(n) / fs
            x = 0.3 * np.exp(2j * np.pi * (0.11 * fs * t + 2.5 * np.sin(2 * np.pi * 900 * t)))
            x = (x + 0.2 * (rng.standard_normal(n) + 1j * rng.standard_normal(n))).astype(np.complex64)
            par.process_block(x)
            ser.process_block(x)
            for sa, sb in zip(a, b):
                p, q = par.result(sa), ser.result(sb)
                assert all(np.isfinite(p[f]) for f in ("coherence", "pilot_hz", "err_avg")), (k, p["pll_path"])
                assert (p["locked"], p["stereo"]) == (q["locked"], q["stereo"])
                assert abs(p["pilot_hz"] - q["pilot_hz"]) <= 2e-3
                assert abs(p["err_avg"] - q["err_avg"]) <= 1e-5
                assert abs(p["coherence"] - q["coherence"]) <= 1e-5 * max(1.0, abs(q["coherence"]))
    finally:
        par.close()
        ser.close()


@pytest.mark.parametrize("at,value", [(0, np.nan), (200_000, np.inf), (399_990, np.nan)])
def test_non_finite_sample(cuda, at, value):
    """The channel's composite is not a number around the sample (in the oracle
    too) and its loop from there on; later blocks take no sweeps over it."""
    fs, rate, block = 2_400_000, 300_000, 400_000
    (par, ser), (a, b) = _pair(fs, block, rate, 65, 1)
    rng = np.random.default_rng(4)
    try:
        for k in range(4):
            x = (0.5 * (rng.standard_normal(block) + 1j * rng.standard_normal(block))).astype(np.complex64)
            if k == 1:
                x[at] = value
            par.process_block(x)
            ser.process_block(x)
            for sa, sb in zip(a, b):
                p, q = par.result(sa), ser.result(sb)
                assert np.array_equal(np.isnan(p["audio"]), np.isnan(q["audio"]))
                assert np.isnan(p["err_avg"]) == np.isnan(q["err_avg"]) == (k >= 1)
                assert (p["locked"], p["stereo"]) == (q["locked"], q["stereo"])
                if k >= 2:
                    assert p["pll_iters"] <= 1, p["pll_iters"]
    finally:
        par.close()
        ser.close()
