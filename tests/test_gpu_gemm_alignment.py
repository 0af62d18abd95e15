"""Channel groups of the tensor-core extraction on device blocks at both halves of
16 bytes: their spans come in by bulk copies, which start on 16 bytes.  The IQ of
every channel is the same bits wherever the block lies, for odd and even starts of
a tile's span (block lengths that move the phase) and a block end just behind it;
and the oracle's within the extraction's parity bound."""
import numpy as np
import pytest

import gpudemod as G
from oracle import oracle as O
from signals import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5
FS = 10_000_000


def _run(lens, at, taps, decim, offs, x):
    import torch
    r = G.ChannelRunner(FS, max(lens), max_channels=8, max_taps=1024)
    r.set_profiling(True)
    out = []
    try:
        slots = [r.admit(k + 1, o, 0.5 * FS / decim, FS // decim, taps, G.MODE_IQ, G.CH_EMIT_IQ)
                 for k, o in enumerate(offs)]
        dev = torch.empty(max(lens) + 2, dtype=torch.complex64, device="cuda")
        pos = 0
        for n in lens:
            view = dev[at:at + n]
            assert view.data_ptr() % 16 == 8 * at
            view.copy_(torch.from_numpy(x[pos:pos + n]))
            pos += n
            torch.cuda.synchronize()
            r.process_block(view)
            out.append(([r.result(s)["iq"] for s in slots], "extract_gemm" in {k for k, _ in r.stage_times()}))
    finally:
        r.close()
    return out


@pytest.mark.parametrize("taps,decim", [(256, 32), (400, 80), (700, 64), (300, 40)])
def test_blocks_on_either_half_of_16_bytes(cuda, taps, decim):
    rng = np.random.default_rng(taps)
    lens = [decim * 900 + k for k in (0, 1, decim // 2, 7, 0)]
    x = (rng.standard_normal(sum(lens)) + 1j * rng.standard_normal(sum(lens))).astype(np.complex64)
    offs = [-3.1e6, -0.7e6, 0.2e6, 1.9e6, 3.3e6]
    even, odd = (_run(lens, at, taps, decim, offs, x) for at in (0, 1))
    refs = [O.OracleChannel(FS, o, 0.5 * FS / decim, FS // decim, taps, O.MODE_NFM, rds=False) for o in offs]
    pos = 0
    for n, (a, grouped), (b, too) in zip(lens, even, odd):
        assert grouped and too
        for k, ref in enumerate(refs):
            w = ref.process(x[pos:pos + n])["iq"]
            assert a[k].size == b[k].size == w.size
            assert np.array_equal(a[k].view(np.uint64), b[k].view(np.uint64)), k
            assert rel_l2(b[k], w) <= TOL, (k, rel_l2(b[k], w))
        pos += n
