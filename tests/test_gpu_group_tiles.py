"""Phase groups at their edges: arms of 1 to 16 taps, whose warps work alone on
chunks of 32 (16 above 8 taps) phases, and longer ones; odd and even
decimations (8- and 16-byte staging copies) with blocks that start on either
half of 16 bytes, groups that end inside a chunk, more taps than are held at a
time, float64 sums of rows (oversampled FM), several tiles per work item, and
blocks that end inside a tile, shorter than the filter's history.  IQ against
the oracle within the extraction's parity bound."""
import numpy as np
import pytest
import torch

import gpudemod as G
from oracle import oracle as O
from signals import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _run(chans, fs, lens, shift, group_phases=0):
    """chans: (offset, taps, decimation, oversampled)"""
    rng = np.random.default_rng(len(chans) * 1000 + lens[0])
    x = (rng.standard_normal(sum(lens)) + 1j * rng.standard_normal(sum(lens))).astype(np.complex64)
    r = G.ChannelRunner(fs, max(lens), max_channels=max(4, len(chans)), max_taps=4096)
    r.set_channel_groups(False)
    r.set_autotune_table([(t, d, G.FORM_GROUP, group_phases) for t, d in {c[1:3] for c in chans}])
    r.set_profiling(True)
    try:
        slots, refs = [], []
        for k, (off, taps, d, over) in enumerate(chans):
            rate = fs // d
            bw = rate / 5.0 if over else rate / 2.0
            slots.append(r.admit(k + 1, off, bw, rate, taps, G.MODE_NFM if over else G.MODE_IQ, G.CH_EMIT_IQ))
            assert r.channel_form(slots[-1])[0] == G.FORM_GROUP
            refs.append(O.OracleChannel(fs, off, bw, rate, taps, O.MODE_NFM, rds=False))
        at = 0
        dev = torch.empty(max(lens) + 1, dtype=torch.complex64, device="cuda")
        for b, n in enumerate(lens):
            blk = x[at:at + n]
            at += n
            view = dev[shift:shift + n]
            view.copy_(torch.from_numpy(blk))
            torch.cuda.synchronize()
            r.process_block(view)
            for k, (s, ref) in enumerate(zip(slots, refs)):
                g, w = r.result(s)["iq"], ref.process(blk)["iq"]
                assert g.size == w.size, (b, k)
                if g.size:
                    assert rel_l2(g, w) <= TOL, (b, k, rel_l2(g, w))
    finally:
        r.close()


@pytest.mark.parametrize("taps,decim,group_phases,over", [
    (64, 64, 0, False),      # L 1
    (130, 65, 0, False),     # L 2, odd D
    (260, 65, 65, False),    # L 4, groups of three chunks (32, 32, 1)
    (500, 100, 33, False),   # L 5, chunks of 32 and 1
    (255, 32, 32, False),    # L 8, one group
    (288, 32, 17, False),    # L 9: chunks of 16 and 1
    (300, 25, 25, False),    # L 12, odd D
    (512, 32, 0, False),     # L 16
    (2000, 160, 8, False),   # L 13, more taps than are held at a time
    (400, 50, 0, True),      # float64 row sums
    (350, 27, 0, True),
    (272, 16, 0, False),     # L 17: tiles of the whole CTA
    (513, 27, 17, False),    # L 19, odd D, two groups
    (640, 20, 20, False),    # L 32: no padding
    (1000, 25, 25, True),    # L 40, float64 row sums, odd D
    (4000, 10, 0, False),    # L 400
])
@pytest.mark.parametrize("shift", [0, 1])
def test_group_tiles_match_oracle(cuda, taps, decim, group_phases, over, shift):
    lens = [decim * 300 + 7, decim * 257, 31, decim * 33 + decim - 1, decim * 512 + 1]
    _run([(12_345.0, taps, decim, over)], decim * 50_000, lens, shift, group_phases)


def test_several_tiles_per_item_match_oracle(cuda):
    """Enough tiles that a work item takes several: few phases, two blocks."""
    fs = 1_600_000
    chans = [(1_000.0 * k - 40_000.0, t, 16, k == 1) for k, t in enumerate((80, 150, 96, 256, 300, 401))]
    _run(chans, fs, [16 * 256 * 1_250 + 5, 16 * 256 * 1_220], 0)
