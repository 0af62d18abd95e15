"""Work items of the short-arm banks (bank_extract.cu) at their edges: tap
counts around the 64-tap chunks and odd ones, channel counts that leave 1 to
32 channels in the last chunk of 32 (one, two or four lane groups), and block
lengths that give 4, 2 or 1 outputs per lane, with a last item that is nearly
empty.  The IQ of channels at both ends of every chunk against the oracle;
the tolerance is the extraction's parity bound (float32 sums of at most 200
taps: 200 * 2^-24 * sqrt-law slack < 1e-5)."""
import numpy as np
import pytest

import gpudemod as G
from oracle import oracle as O
from signals import rel_l2

pytestmark = pytest.mark.gpu

FS, OUT, D = 2_400_000, 48_000, 50
TOL = 1e-5


@pytest.mark.parametrize("taps,nch,n_out", [
    (63, 4, 33), (64, 8, 65), (65, 9, 130),          # one output per lane
    (128, 16, 2375), (129, 17, 1250), (191, 33, 1300),  # two
    (200, 7, 4801), (127, 40, 2400), (193, 49, 2370),   # four: last chunks of 7, 8 and 17 channels
    (63, 32, 4737),
])
def test_bank_items_match_oracle(cuda, taps, nch, n_out):
    rng = np.random.default_rng(taps * 100 + nch)
    n = n_out * D + 13
    blocks = [(rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64) for _ in range(2)]
    offs = [-1_000_000.0 + 2_000_000.0 * i / nch + 37.0 * i for i in range(nch)]
    check = sorted({0, min(7, nch - 1), min(31, nch - 1), min(32, nch - 1), nch - 1})
    r = G.ChannelRunner(FS, n, max_channels=64, max_taps=256)
    r.set_profiling(True)
    try:
        slots = [r.admit(i + 1, o, 12_000.0, OUT, taps, G.MODE_IQ, G.CH_EMIT_IQ) for i, o in enumerate(offs)]
        refs = {i: O.OracleChannel(FS, offs[i], 12_000.0, OUT, taps, O.MODE_NFM, rds=False) for i in check}
        for x in blocks:
            r.process_block(x)
            assert "extract_bank" in {name for name, _ in r.stage_times()}
            for i, ref in refs.items():
                g, w = r.result(slots[i])["iq"], ref.process(x)["iq"]
                assert g.size == w.size
                assert rel_l2(g, w) <= TOL, (i, rel_l2(g, w))
    finally:
        r.close()
