"""The streaming polyphase launcher at the edges of its output tiles (32, 64 and
256 outputs) and of the rule that picks them (rows that fit in shared memory,
decimations far above the tap count), chunk by chunk against the oracle, and
with outputs or history that overlap the input block.  Tolerance 1e-5 max-abs:
the reference test's own (float32 sums of at most 512 taps of a low-pass of
gain one: 512 * 2^-24 * 0.3)."""
import ctypes as C
import math

import numpy as np
import pytest

from gpudemod._lib import lib
from oracle import oracle as O
from signals import make_tone_noise_iq, max_abs

pytestmark = pytest.mark.gpu

FS = 4_096_000


def _run(taps, decim, sizes, overlap=None, offset=123_456.0):
    import torch
    poly = O.build_polyphase_taps_phase_major(O.base_taps_f32(200_000, FS, taps), decim)
    inc = -2 * math.pi * offset / FS
    cap, top = taps - 1, max(sizes)
    d_taps = torch.from_numpy(poly).cuda()
    d_hist, d_scr = (torch.zeros(max(1, cap), dtype=torch.complex64, device="cuda") for _ in range(2))
    d_sh = torch.zeros(top, dtype=torch.complex64, device="cuda")
    hl, pc, ph, nout = C.c_int(0), C.c_int(0), C.c_double(0.0), C.c_int()
    o_hist, o_ph, o_pc = np.zeros(0, np.complex64), 0.0, 0
    x = make_tone_noise_iq(sum(sizes), 0.021)
    pos = 0
    for n in sizes:
        chunk = x[pos:pos + n]
        pos += n
        d_in = torch.from_numpy(chunk.copy()).cuda()
        n_max = n // decim + 2
        d_out = d_in if overlap == "out" else torch.zeros(n_max, dtype=torch.complex64, device="cuda")
        if overlap == "shifted":
            d_sh = d_in
        rc = lib.gpud_launch_streaming_polyphase_stateful_cuda(
            d_in.data_ptr(), n, d_sh.data_ptr(), d_taps.data_ptr(), poly.size, decim, taps, d_hist.data_ptr(),
            d_scr.data_ptr(), cap, C.byref(hl), C.byref(pc), C.byref(ph), inc, d_out.data_ptr(), min(n_max, d_out.numel()),
            C.byref(nout))
        assert rc == 0
        assert lib.gpud_stream_sync(None) == 0
        want, o_ph, o_pc, o_hist = O.run_host_core(chunk, FS, offset, o_ph, o_pc, taps, decim, o_hist, poly)
        assert (nout.value, pc.value, hl.value) == (want.size, o_pc, o_hist.size)
        assert max_abs(d_out.cpu().numpy()[: nout.value], want) <= 1e-5
        assert max_abs(d_hist.cpu().numpy()[: hl.value], o_hist) <= 1e-5
        assert abs(math.remainder(ph.value - o_ph, 2 * math.pi)) <= 1e-9


@pytest.mark.parametrize("taps,decim,outs", [
    (101, 4, [1, 63, 64, 65, 128]), (257, 20, [64, 1, 129]), (512, 2, [300, 76_000]), (65, 64, [31, 32, 33]),
    (300, 400, [64, 65, 7]), (512, 500, [33, 64]), (512, 1000, [5, 33]), (33, 200, [40, 64]),
])
def test_tile_edges(cuda, taps, decim, outs):
    _run(taps, decim, [decim * o + d for o, d in zip(outs, (3, 0, decim - 1, 1, 0))])


@pytest.mark.parametrize("overlap", ["out", "shifted"])
def test_overlapping_buffers(cuda, overlap):
    _run(129, 8, [4096, 1001, 8192], overlap)
