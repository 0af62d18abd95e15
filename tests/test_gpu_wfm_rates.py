"""WFM channels of several demodulator rates in one runner: each rate has its own
set of filters.  Audio and RDS baseband of every channel against the oracle,
within the parity bound of the path (1e-5 rel-L2)."""
import numpy as np
import pytest

import gpudemod as G
from gpudemod import synth
from oracle import oracle as O
from signals import rel_l2

pytestmark = pytest.mark.gpu

FS, BLOCK = 2_400_000, 192_000


@pytest.mark.parametrize("rates", [(300_000, 240_000), (200_000, 300_000, 160_000, 240_000, 150_000)])
def test_every_rate_matches_the_oracle(cuda, rates):
    scene, _ = synth.plain_wfm_scene(block=BLOCK)
    r = G.ChannelRunner(FS, BLOCK, max_channels=8)
    specs = [(k + 1, 300_000.0, 140_000.0, rate, 101) for k, rate in enumerate(rates)]
    slots = [r.admit(*s, G.MODE_WFM_STEREO, G.CH_RDS) for s in specs]
    refs = [O.OracleChannel(FS, *s[1:4], s[4], O.MODE_WFM_STEREO, rds=True) for s in specs]
    try:
        for _ in range(6):  # stereo from the fourth locked block on
            x = scene.next_block().numpy()
            r.process_block(x)
            for s, slot, ref in zip(specs, slots, refs):
                g, w = r.result(slot), ref.process(x)
                assert (g["locked"], g["stereo"]) == (w["locked"], w["stereo"]), s
                for key in ("audio", "rds"):
                    assert g[key].size == w[key].size
                    assert rel_l2(g[key], w[key]) <= 1e-5, (s, key, rel_l2(g[key], w[key]))
    finally:
        r.close()
