"""The parallel pilot-loop solver against the serial loop (the same recurrence)
at the edges of its segmentation: 16-step segments, 4096 steps per CTA, 32768
steps per chunk (longer blocks run chunk by chunk), on a station (acquisition,
then lock and stereo) and on noise (a loop that never locks).

Tolerances: both solvers round a step's angle to float32 (half an ulp of 2 pi:
2.4e-7 rad), which moves the L-R product by at most 5e-7 of its size, so the
audio agrees within 1e-6 rel-L2; the loop's frequency is an average of that
phase over >= 1 / beta steps (1e-7 of a step's angle: below 1e-4 Hz), its mean
error and coherence are float32 values of order one (1e-5)."""
import numpy as np
import pytest

import gpudemod as G
from gpudemod import synth
from signals import rel_l2

pytestmark = pytest.mark.gpu

FS, D = 2_400_000, 8


@pytest.mark.parametrize("steps", [1, 15, 16, 17, 255, 4095, 4096, 4097, 32767, 32768, 32769, 66_001])
def test_segment_and_chunk_edges(cuda, steps):
    import torch
    block = steps * D
    scene, _ = synth.plain_wfm_scene(device="cuda", block=block)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(steps)
    specs = [(1, 300_000.0, 250_000.0, FS // D, 128, G.MODE_WFM_STEREO, G.CH_RDS),
             (2, -500_000.0, 250_000.0, FS // D, 128, G.MODE_WFM_STEREO, 0)]
    par, ser = (G.ChannelRunner(FS, block, max_channels=2) for _ in range(2))
    ser.set_pll_solver(False)
    try:
        slots = [(par.admit(*s), ser.admit(*s)) for s in specs]
        for _ in range(6):
            x = scene.next_block()
            x = x + 0.1 * torch.view_as_complex(torch.randn(block, 2, generator=gen, device="cuda"))
            torch.cuda.synchronize()
            par.process_block(x)
            ser.process_block(x)
            for a_slot, b_slot in slots:
                a, b = par.result(a_slot), ser.result(b_slot)
                assert a["audio"].size == b["audio"].size
                if b["audio"].size:
                    assert rel_l2(a["audio"], b["audio"]) <= 1e-6, rel_l2(a["audio"], b["audio"])
                assert (a["locked"], a["stereo"]) == (b["locked"], b["stereo"])
                assert abs(a["pilot_hz"] - b["pilot_hz"]) <= 2e-3  # float32 ulp at 19 kHz
                assert abs(a["err_avg"] - b["err_avg"]) <= 1e-5
                assert abs(a["coherence"] - b["coherence"]) <= 1e-5
    finally:
        par.close()
        ser.close()
