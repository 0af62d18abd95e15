"""Which kernel a dense class of a misaligned block takes: one tile per CTA below
two tiles per SM of this GPU, warps that work alone from there on.  Read from a
profile of the launches, at the rule's two sides; a channel's IQ is the same bits
on both, and the oracle's within the extraction's parity bound."""
import numpy as np
import pytest

import gpudemod as G
from oracle import oracle as O
from signals import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-5
D, TAPS, FS = 16, 144, 9_600_000  # arms of 9 taps


def _iq(x):
    """(kernel names, IQ) of one block that starts on an odd multiple of 8 bytes."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    r = G.ChannelRunner(FS, x.size, max_channels=2, max_taps=256)
    r.set_channel_groups(False)
    r.set_autotune_table([(TAPS, D, G.FORM_DENSE, 0)])
    try:
        slot = r.admit(1, 310_000.0, 200_000.0, FS // D, TAPS, G.MODE_IQ, G.CH_EMIT_IQ)
        dev = torch.empty(x.size + 1, dtype=torch.complex64, device="cuda")
        view = dev[1:]
        view.copy_(torch.from_numpy(x))
        torch.cuda.synchronize()
        r.process_block(view)
        iq = r.result(slot)["iq"]
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            for _ in range(10):  # a profile may miss launches at its start
                r.process_block(view)
            torch.cuda.synchronize()
        return [e.name for e in p.events() if "k_extract" in e.name], iq
    finally:
        r.close()


def test_both_sides_of_the_rule(cuda):
    import torch
    tiles = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(11)
    n = tiles * 256 * D
    x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
    names, alone = _iq(x[:(tiles - 1) * 256 * D + D])  # one output in the last tile: as many tiles
    assert any("k_extract_rot<true>" in k for k in names), names
    names, small = _iq(x[:(tiles - 1) * 256 * D])
    assert any("k_extract_dense<9>" in k for k in names) and not any("k_extract_rot" in k for k in names), names
    assert alone.size == small.size + 1
    assert np.array_equal(alone[:-1].view(np.uint64), small.view(np.uint64))
    want = O.OracleChannel(FS, 310_000.0, 200_000.0, FS // D, TAPS, O.MODE_NFM, rds=False).process(x)["iq"]
    assert rel_l2(alone, want[:alone.size]) <= TOL
