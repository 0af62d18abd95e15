"""The streaming polyphase launcher's caller-owned buffers, step by step as its
contract has them: the block is read, shifted, before anything else is written,
so the history, the scratch, the shifted copy and the outputs may each lie in
the input block; afterwards the shifted buffer holds the rotated block and the
scratch the new history.  Against the oracle; 1e-5 max-abs, the reference
test's own (test_gpu_launcher_tiles.py)."""
import ctypes as C
import math

import numpy as np
import pytest

from gpudemod._lib import lib
from oracle import oracle as O
from signals import make_tone_noise_iq, max_abs

pytestmark = pytest.mark.gpu

FS, OFFSET, TAPS, DECIM = 4_096_000, 123_456.0, 257, 16
INC = -2 * math.pi * OFFSET / FS
CAP = TAPS - 1


def _call(d_in, n, d_sh, poly, d_hist, d_scr, hist_len, pc0, ph0, d_out):
    import torch
    d_taps = torch.from_numpy(poly).cuda()
    hl, pc, ph, nout = C.c_int(hist_len), C.c_int(pc0), C.c_double(ph0), C.c_int()
    torch.cuda.synchronize()
    rc = lib.gpud_launch_streaming_polyphase_stateful_cuda(
        d_in.data_ptr(), n, d_sh.data_ptr(), d_taps.data_ptr(), poly.size, DECIM, TAPS, d_hist.data_ptr(),
        d_scr.data_ptr(), CAP, C.byref(hl), C.byref(pc), C.byref(ph), INC, d_out.data_ptr(), d_out.numel(),
        C.byref(nout))
    assert rc == 0 and lib.gpud_stream_sync(None) == 0
    return nout.value, hl.value, pc.value, ph.value


# n below, at and above the history's length (a history that is partly kept is
# staged in the scratch); where the second buffer starts in the block
@pytest.mark.parametrize("n", [37, 255, 256, 257, 4099])
@pytest.mark.parametrize("where,at", [(None, 0), ("scratch", 0), ("scratch", 5), ("history", 0), ("history", 3),
                                      ("out", 0), ("shifted", 0)])
def test_buffers(cuda, n, where, at):
    import torch
    poly = O.build_polyphase_taps_phase_major(O.base_taps_f32(200_000, FS, TAPS), DECIM)
    x = make_tone_noise_iq(n + CAP, 0.021)
    ph0, pc0 = 0.7, 5
    # the block, with room behind it: a buffer of CAP samples may start inside it
    d_in = torch.zeros(n + 2 * CAP, dtype=torch.complex64, device="cuda")
    d_in[:n] = torch.from_numpy(x[:n])
    new = lambda m: torch.zeros(m, dtype=torch.complex64, device="cuda")
    d_hist = d_in[at:at + CAP] if where == "history" else new(CAP)
    d_scr = d_in[at:at + CAP] if where == "scratch" else new(CAP)
    d_sh = d_in if where == "shifted" else new(n)
    d_out = d_in[:n] if where == "out" else new(n // DECIM + 2)
    if where != "history":
        d_hist.copy_(torch.from_numpy(x[n:]))
    hist = d_hist.cpu().numpy().copy()
    want, o_ph, o_pc, o_hist = O.run_host_core(x[:n], FS, OFFSET, ph0, pc0, TAPS, DECIM, hist, poly)
    nout, hl, pc, ph = _call(d_in, n, d_sh, poly, d_hist, d_scr, CAP, pc0, ph0, d_out)
    assert (nout, pc, hl) == (want.size, o_pc, o_hist.size)
    assert max_abs(d_out[:nout].cpu().numpy(), want) <= 1e-5
    assert max_abs(d_hist.cpu().numpy(), o_hist) <= 1e-5
    assert abs(math.remainder(ph - o_ph, 2 * math.pi)) <= 1e-9
    if where in (None, "scratch", "history"):
        shifted = x[:n] * np.exp(1j * (ph0 + INC * np.arange(n)))
        assert max_abs(d_sh.cpu().numpy()[:n], shifted.astype(np.complex64)) <= 1e-5
    if where in (None, "out", "shifted"):
        assert max_abs(d_scr.cpu().numpy(), o_hist) <= 1e-5


@pytest.mark.parametrize("n", [0, 16, 1000])
def test_shifted_block_without_history(cuda, n):
    """One tap, no history to keep: the shifted copy is still written."""
    import torch
    x = make_tone_noise_iq(max(n, 1), 0.05)[:n]
    d_in = torch.from_numpy(np.append(x, np.complex64(0))).cuda()
    d_sh, d_hist, d_scr, d_out = (torch.zeros(n + 1, dtype=torch.complex64, device="cuda") for _ in range(4))
    taps = torch.ones(1, dtype=torch.float32, device="cuda")
    hl, pc, ph, nout = C.c_int(0), C.c_int(0), C.c_double(0.0), C.c_int()
    torch.cuda.synchronize()
    assert lib.gpud_launch_streaming_polyphase_stateful_cuda(
        d_in.data_ptr(), n, d_sh.data_ptr(), taps.data_ptr(), 1, 1, 1, d_hist.data_ptr(), d_scr.data_ptr(), 0,
        C.byref(hl), C.byref(pc), C.byref(ph), INC, d_out.data_ptr(), n, C.byref(nout)) == 0
    assert lib.gpud_stream_sync(None) == 0
    want = (x * np.exp(1j * INC * np.arange(n))).astype(np.complex64)
    assert nout.value == n and hl.value == 0
    assert max_abs(d_sh.cpu().numpy()[:n], want) <= 1e-5
    assert max_abs(d_out.cpu().numpy()[:n], want) <= 1e-5


@pytest.mark.parametrize("taps,decim,n", [
    (101, 4, 4_001), (512, 2, 160_003), (65, 64, 64 * 33 + 5), (300, 400, 12_345), (512, 500, 499), (1, 7, 700),
    (33, 200, 8_130), (512, 1000, 33_333),  # few taps far apart, rows too large: the gather kernel
])
def test_shifted_block_of_every_route(cuda, taps, decim, n):
    """Every sample of the shifted block: those an output's tile has in hand, the
    rest behind the newest output, and all of them where no tile runs."""
    import torch
    poly = O.build_polyphase_taps_phase_major(O.base_taps_f32(200_000, FS, max(taps, 2)), decim)
    cap = max(1, taps - 1)
    x = make_tone_noise_iq(n, 0.03)
    d_in, d_taps = torch.from_numpy(x).cuda(), torch.from_numpy(poly).cuda()
    d_sh, d_hist, d_scr = (torch.full((m,), float("nan"), dtype=torch.complex64, device="cuda") for m in (n, cap, cap))
    d_out = torch.zeros(n // decim + 2, dtype=torch.complex64, device="cuda")
    hl, pc, ph, nout = C.c_int(0), C.c_int(decim // 3), C.c_double(0.2), C.c_int()
    torch.cuda.synchronize()
    assert lib.gpud_launch_streaming_polyphase_stateful_cuda(
        d_in.data_ptr(), n, d_sh.data_ptr(), d_taps.data_ptr(), poly.size, decim, taps, d_hist.data_ptr(),
        d_scr.data_ptr(), cap, C.byref(hl), C.byref(pc), C.byref(ph), INC, d_out.data_ptr(), d_out.numel(),
        C.byref(nout)) == 0
    assert lib.gpud_stream_sync(None) == 0
    want = x * np.exp(1j * (0.2 + INC * np.arange(n)))
    assert max_abs(d_sh.cpu().numpy(), want.astype(np.complex64)) <= 1e-5
    assert max_abs(d_hist[:hl.value].cpu().numpy(), want[n - hl.value:].astype(np.complex64)) <= 1e-5
    assert max_abs(d_scr[:hl.value].cpu().numpy(), want[n - hl.value:].astype(np.complex64)) <= 1e-5
