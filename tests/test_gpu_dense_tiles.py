"""The dense form's classes that are too large or too misaligned for the
pipelined kernel: tiles whose warps work alone on chunks of 32 (16 above 8 taps
per arm) phases, odd and even decimations, blocks on either half of 16 bytes,
float64 sums of rows, and a block shorter than the filter's history.  IQ
against the oracle within the extraction's parity bound."""
import numpy as np
import pytest
import torch

import gpudemod as G
from oracle import oracle as O
from signals import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _run(chans, fs, lens, shift):
    """chans: (offset, taps, decimation, oversampled)"""
    rng = np.random.default_rng(len(chans) * 1000 + lens[0])
    x = (rng.standard_normal(sum(lens)) + 1j * rng.standard_normal(sum(lens))).astype(np.complex64)
    r = G.ChannelRunner(fs, max(lens), max_channels=max(4, len(chans)), max_taps=4096)
    r.set_channel_groups(False)
    r.set_autotune_table([(t, d, G.FORM_DENSE, 0) for t, d in {c[1:3] for c in chans}])
    r.set_profiling(True)
    try:
        slots, refs = [], []
        for k, (off, taps, d, over) in enumerate(chans):
            rate = fs // d
            bw = rate / 5.0 if over else rate / 2.0
            slots.append(r.admit(k + 1, off, bw, rate, taps, G.MODE_NFM if over else G.MODE_IQ, G.CH_EMIT_IQ))
            assert r.channel_form(slots[-1])[0] == G.FORM_DENSE
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


@pytest.mark.parametrize("geoms,over", [
    ([(33, 16), (50, 16), (80, 16)], False),              # L 3, 4, 5 together
    ([(90, 15), (160, 20), (200, 25)], False),            # L 6, 8, 8: odd and even D
    ([(144, 16), (250, 25), (256, 16)], False),           # L 9, 10, 16: chunks of 16 phases
    ([(330, 66), (600, 65)], False),                      # more than two chunks of 32, L 5 and 10
    ([(160, 20), (300, 20)], True),                       # float64 row sums
])
@pytest.mark.parametrize("shift", [0, 1])
def test_dense_tiles_match_oracle(cuda, geoms, over, shift):
    """Classes that share a launch of more than two tiles per SM, one channel each."""
    d_max = max(d for _, d in geoms)
    n = d_max * 256 * 300 // len(geoms) + 3
    chans = [(1_000.0 * k - 9_000.0, t, d, over) for k, (t, d) in enumerate(geoms)]
    _run(chans, 10_296_000, [n, 37, n - d_max * 100], shift)
