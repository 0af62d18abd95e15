"""The pilot detector's workspace: what a detector for thousands of stations
takes from the device, and calls whose passes take turns in it."""
import gc

import numpy as np
import pytest

import gpudemod as G

pytestmark = pytest.mark.gpu


def _baseband(fs, n, seed):
    rng = np.random.default_rng(seed)
    t = np.arange(n) / fs
    m = 0.3 * np.sin(2 * np.pi * (300 + 11 * seed) * t) + (0.1 if seed % 2 else 0.0) * np.sin(2 * np.pi * 19_000 * t)
    z = np.exp(1j * 2 * np.pi * 75_000 * np.cumsum(m) / fs)
    return (z + 0.05 * (rng.standard_normal(n) + 1j * rng.standard_normal(n))).astype(np.complex64)


@pytest.mark.parametrize("stations,samples", [(4096, 2048), (1, 2048), (2000, 20_000)])
def test_workspace_of_many_stations(cuda, stations, samples):
    """Per station its folded window and decision (8 bytes a sample, under 1 KB);
    on top the roots table (16 MiB) and the partial sums of one pass (40 stations
    x 201 bins x at most four shares per SM: 77 MB), with 8 MB for the
    allocator's rounding."""
    import torch
    gc.collect()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    det = G.StereoPilotDetector(stations, samples)
    try:
        used = before - torch.cuda.mem_get_info()[0]
    finally:
        det.close()
    assert used <= stations * (8 * samples + 1024) + (16 << 20) + 77_000_000 + (8 << 20)


def test_passes_take_turns(cuda):
    """133 stations at three rates, in an order that mixes them: full passes and
    rests, more than the workspace holds at once.  Every decision is the one of
    the station alone, bit for bit."""
    import torch
    plan = [(312_500, 40_000), (256_000, 20_000), (250_007, 30_000)]
    jobs = [plan[(3 * i + i // 7) % 3 if i < 100 else 0] for i in range(133)]
    iq = [torch.from_numpy(_baseband(fs, n, i)).cuda() for i, (fs, n) in enumerate(jobs)]
    det = G.StereoPilotDetector(133, 40_000)
    one = G.StereoPilotDetector(1, 40_000)
    try:
        torch.cuda.synchronize()
        got = det.run(iq, [fs for fs, _ in jobs])
        for i, (fs, _) in enumerate(jobs):
            assert got[i] == one.run([iq[i]], [fs])[0], i
        assert 0 < sum(g["present"] for g in got) < 133
    finally:
        det.close()
        one.close()
